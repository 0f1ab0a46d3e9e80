"""FP64 qr with less workspace than the query now asks for: the sizes that the
query gave when partial sums were cut into chunks of 256 rows stay enough (a
caller may keep such a buffer), one byte less is refused, and
nothing is written past the end.  Results within 10 n u for the Householder
path, and for block Gram-Schmidt on these well-conditioned inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U64 = 2.0 ** -53
GUARD = 65536

# (m, n, algorithm, reorth, panel, bytes)
SIZES = [(100, 16, "block_gs", False, 8, 4864), (1000, 33, "block_gs", False, 32, 38144),
         (4096, 64, "block_gs", True, 32, 291072), (20000, 64, "block_gs", False, 32, 1396992),
         (27648, 96, "block_gs", False, 32, 2789632), (2000, 160, "block_gs", True, 32, 512256),
         (27648, 128, "block_gs", False, 32, 4559104), (100, 32, "householder", False, 8, 20224),
         (4096, 64, "householder", False, 32, 356608), (1500, 60, "householder", False, 24, 133120)]


@pytest.mark.parametrize("m,n,algorithm,reorth,panel,size", SIZES)
def test_fp64_qr_takes_the_earlier_sizes(orc, cuda, tg, m, n, algorithm, reorth, panel, size):
    import torch
    kw = {"algorithm": algorithm, "reorth": reorth, "panel": panel}
    A = orc.fill_uniform(m, n, np.float64, seed=81)
    q = tg.empty_colmajor(m, n, torch.float64, "cuda")
    q.copy_(torch.from_numpy(np.ascontiguousarray(A)))
    buf = torch.full((size + GUARD,), 0x5A, dtype=torch.uint8, device="cuda")
    r = tg.qr_(q, work=buf[:size], **kw)
    torch.cuda.synchronize()
    assert bool((buf[size:] == 0x5A).all())
    met = orc.metrics(A, q.t().contiguous().cpu().numpy().T, r.t().contiguous().cpu().numpy().T)
    assert met["backward"] <= 10 * n * U64 and met["orth"] <= 10 * n * U64, met


def test_fp64_qr_refuses_less(cuda, tg):
    import torch
    q = tg.empty_colmajor(4096, 64, torch.float64, "cuda").normal_()
    with pytest.raises(tg.TsqrError) as e:
        tg.qr_(q, work=torch.empty(291072 - 1, dtype=torch.uint8, device="cuda"), reorth=True)
    assert e.value.status == 3
