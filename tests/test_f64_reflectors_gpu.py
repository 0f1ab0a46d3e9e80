"""How orthogonal the FP64 reflectors above level 0 are: H = I - tau v v^T is
orthogonal where tau v^T v = 2, so the relative error of tau v^T v / 2 is
taken for every column of a level-1 tile (tau is T's diagonal, v_j = 1) and
its root mean square over all of them.

Bar.  A value formed with correctly rounded operations carries six independent
roundings that reach tau v^T v at full size or less: alpha - beta, its
reciprocal, (alpha - beta) / beta, beta itself, the squared norm under its
root, and v's own (which average out).  The relative error of rounding a value
with a logarithmically distributed mantissa has the root mean square
u sqrt((1 / 3) (3 / 8) / ln 2) = 0.425 u, so 0.425 sqrt(6) u = 1.04 u in all.
Every further rounding of tau (a product with a scale and back, an unrounded
reciprocal) adds to it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U64 = 2.0 ** -53


@pytest.mark.parametrize("n", [8, 16, 32])
def test_fp64_reflectors_above_level_0_are_orthogonal(orc, cuda, tg, n):
    import torch
    rows = 512 if n <= 16 else 256
    tiles = 8
    err = []
    for seed in range(40):
        a = tg.empty_colmajor(rows * tiles, n, torch.float64, "cuda")
        a.copy_(torch.from_numpy(np.ascontiguousarray(orc.fill_uniform(rows * tiles, n, np.float64, seed=200 + seed))))
        fac = tg.factor_(a)
        torch.cuda.synchronize()
        h = tiles * n  # one tile of the level above; behind the 256-byte status header
        ld = (h + 31) // 32 * 32
        t = fac.work.cpu().numpy()[256:256 + 8 * ld * n].view(np.float64).reshape(n, ld)[:, :h]
        for j in range(n):
            v = t[j, j + 1:].astype(np.longdouble)
            err.append(float(np.longdouble(t[j, j]) * (1 + v @ v) / 2 - 1))
    rms = np.sqrt(np.mean(np.square(err)))
    assert rms <= 0.425 * np.sqrt(6.0) * U64, rms / U64
