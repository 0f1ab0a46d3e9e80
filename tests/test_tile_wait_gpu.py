"""The persistent TMA-fed tile factor (9 to 16 columns, several tiles per
resident CTA): a wait that runs out ends the CTA with its copy landed and the
status word set, and the next call with the default limit succeeds and clears
the word.  The limit of 0 polls makes the first wait of each CTA give up."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(700000, 16), (700001 + 3, 9)])
def test_persistent_tile_wait_that_runs_out_is_reported(cuda, tg, m, n):
    import torch
    L = tg.lib()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(19)
    a0 = tg.empty_colmajor(m, n, torch.float32, "cuda")
    a0.t().uniform_(-1.0, 1.0, generator=gen)
    w = torch.full((tg.workspace_bytes(m, n, torch.float32),), 0xFF, dtype=torch.uint8, device="cuda")
    q = a0.t().clone().t()
    try:
        assert L.tsqr_debug_set_wait_limit(0) == 0
        tg.tsqr_(q, work=w)
        torch.cuda.synchronize()
        assert L.tsqr_workspace_check(w.data_ptr()) == 4  # TSQR_ERR_CUDA
    finally:
        L.tsqr_debug_set_wait_limit(-1)
    q = a0.t().clone().t()
    r = tg.tsqr_(q, work=w)
    torch.cuda.synchronize()
    assert L.tsqr_workspace_check(w.data_ptr()) == 0
    a64, q64, r64 = a0.double(), q.double(), r.double()
    bar = 10 * n * 2.0 ** -24
    assert float((a64 - q64 @ r64).norm() / a64.norm()) <= bar
    assert float((q64.t() @ q64 - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) <= bar
