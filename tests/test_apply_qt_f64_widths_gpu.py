"""Q^T c in FP64 with one or two columns at widths around the 8-term steps in
which its triangular products leave past n.  Bar as for the other tests of the
kernel: |D - Q^T C| <= 10 n u |c|, column by column."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32])
def test_fp64_apply_qt_widths(cuda, tg, n):
    import torch
    m, k, u = 1301, 2, 2.0 ** -53
    gen = torch.Generator(device="cuda")
    gen.manual_seed(15)
    a = tg.empty_colmajor(m, n, torch.float64, "cuda")
    a.t().uniform_(-1.0, 1.0, generator=gen)
    c = tg.empty_colmajor(m, k, torch.float64, "cuda")
    c.t().uniform_(-1.0, 1.0, generator=gen)
    f = tg.factor_(a)
    d = tg.apply_qt_(f, c)
    q = tg.form_q_(f)
    err = (d - q.t() @ c).abs().amax(0)
    assert bool((err <= 10 * n * u * c.norm(dim=0)).all()), err
