"""The precision form from host memory takes the same Q assembly, level by
level, as from device memory: bit for bit the same Q and R where level 0 is one
chunk (below 32 MB) and the device matrix is aligned as the library's own copy
is.  On both sides of the lines of the rule (padded and full widths, up to and
above 128 and 512 tiles), and an odd leading dimension against the form's bar."""
import pytest

pytestmark = pytest.mark.gpu


def device_matrix(tg, m, n, seed, ld=None):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    a = tg.empty_colmajor(m, n, torch.float32, "cuda", ld=ld)
    a.copy_(torch.rand((n, m), generator=gen, device="cuda").mul_(2).sub_(1).t())
    return a


@pytest.mark.parametrize("m,n", [(512, 32), (27648, 32), (128 * 512, 32), (129 * 512, 32), (40000, 20), (300000, 16),
                                 (300000, 5), (60000, 64), (513 * 512, 24), (100000, 40)])
def test_host_and_device_precision_forms_agree(cuda, tg, m, n):
    import torch
    a = device_matrix(tg, m, n, 11)
    h = a.t().cpu().pin_memory().t()
    r = tg.tsqr_(a, precision="tf32x3")
    hq, hr = tg.tsqr_host_(h, precision="tf32x3")
    torch.cuda.synchronize()
    assert torch.equal(hq, a.cpu()) and torch.equal(hr, r.cpu())


@pytest.mark.parametrize("m,n", [(128 * 512, 16), (129 * 512, 16), (1000003, 16), (128 * 512, 32), (129 * 512, 32),
                                 (300001, 9), (384 * 512, 31), (385 * 512, 31), (300001, 12), (300001, 50), (513 * 512, 64), (5000, 64)])
def test_odd_leading_dimension(cuda, tg, m, n):
    import torch
    a = device_matrix(tg, m, n, 12, ld=m + 1 + m % 2)
    a0 = a.double()
    r = tg.tsqr_(a, precision="tf32x3")
    q, r64 = a.double(), r.double()
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    assert float((a0 - q @ r64).norm() / a0.norm()) <= 1e-5
    assert float((q.t() @ q - eye).norm()) <= 1e-5
