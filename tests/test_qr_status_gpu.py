"""GPU test that a bounded wait which gives up inside a panel of a blocked QR is
reported in the call's own status word: shapes and leading dimensions whose
only kernels with bounded waits are the panels' (the TMA-fed tile factor of a
single panel; the tcgen05 Q assembly where an odd leading dimension keeps
every product off TMA).  The wait runs out by a limit of 0 polls
(tsqr_debug_set_wait_limit); with the default limit the same call succeeds and
the word reads clear.

Bars of the second call: 10 n u for the plain form, 1e-5 for the precision
form's panels (its 64-column products here are FP32)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,precision,algorithm", [(400000, 32, "plain", "block_gs"),
                                                     (400000, 32, "plain", "householder"),
                                                     (70001, 32, "tf32x3", "block_gs"),
                                                     (70001, 64, "tf32x3", "block_gs"),
                                                     (70001, 64, "tf32x3", "householder")])
def test_panel_wait_that_runs_out_is_reported(cuda, tg, m, n, precision, algorithm):
    import torch
    L = tg.lib()
    kw = {"precision": precision, "algorithm": algorithm}
    gen = torch.Generator(device="cuda")
    gen.manual_seed(7)
    a0 = tg.empty_colmajor(m, n, torch.float32, "cuda")
    a0.t().uniform_(-1.0, 1.0, generator=gen)
    w = torch.full((tg.qr_workspace_bytes(m, n, torch.float32, **kw),), 0xFF, dtype=torch.uint8, device="cuda")
    q = a0.t().clone().t()
    try:
        assert L.tsqr_debug_set_wait_limit(0) == 0
        tg.qr_(q, work=w, **kw)
        torch.cuda.synchronize()
        assert L.tsqr_workspace_check(w.data_ptr()) == 4  # TSQR_ERR_CUDA
    finally:
        L.tsqr_debug_set_wait_limit(-1)
    torch.cuda.synchronize()
    q = a0.t().clone().t()
    r = tg.qr_(q, work=w, **kw)
    torch.cuda.synchronize()
    assert L.tsqr_workspace_check(w.data_ptr()) == 0
    bar = 10 * n * 2.0 ** -24 if precision == "plain" else 1e-5
    a64, q64, r64 = a0.double(), q.double(), r.double()
    assert float((a64 - q64 @ r64).norm() / a64.norm()) <= bar
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert float((q64.t() @ q64 - eye).norm()) <= max(bar, 10 * n * 2.0 ** -24)
