"""GPU test of the Householder path with a workspace of exactly the size that
the query gives, for panels narrower than 32 columns: what a leaf writes
(U^-1 of the reconstruction among it) stays inside its block, so the results
hold and the bytes after the workspace keep their value.  A single leaf
(n <= panel) has no product buffers between U^-1 and T, and 17 columns in
panels of 16 only 512 bytes of them.

Bars: backward error and orthogonality <= 10 n u, as for the path's other
tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 8192


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("m,n,panel", [(70, 1, 1), (300, 5, 5), (300, 8, 8), (500, 16, 8), (300, 16, 16),
                                       (300, 17, 16), (1000, 24, 24), (1000, 25, 24), (700, 31, 31), (2000, 40, 8),
                                       (600, 32, 32)])
def test_workspace_of_the_queried_size_is_enough(orc, cuda, tg, m, n, panel, dtype):
    import torch
    dt = torch.float32 if dtype == np.float32 else torch.float64
    A = orc.fill_uniform(m, n, dtype, seed=73)
    q = tg.empty_colmajor(m, n, dt, "cuda")
    q.copy_(torch.from_numpy(np.ascontiguousarray(A)))
    size = tg.qr_workspace_bytes(m, n, dt, algorithm="householder", panel=panel)
    buf = torch.full((size + GUARD,), 0x5A, dtype=torch.uint8, device="cuda")
    r = tg.qr_(q, algorithm="householder", panel=panel, work=buf[:size])
    torch.cuda.synchronize()
    assert bool((buf[size:] == 0x5A).all())
    met = orc.metrics(A, q.t().contiguous().cpu().numpy().T, r.t().contiguous().cpu().numpy().T)
    u = orc.unit_roundoff(dtype)
    assert met["backward"] <= 10 * n * u and met["orth"] <= 10 * n * u, met
