"""The rounding error of an FP64 projection R12 = Q1^T A2 over many rows at a
width where each output tile has one chunk: entries of R12 against sums of the
same products in extended precision.

Bar.  A running sum of independent terms of variance s^2 has, after i terms, a
rounding error of root mean square 0.425 u s sqrt(i) (0.425 u: the relative error
of rounding a value with a logarithmically distributed mantissa); over blocks of
256 rows that is 0.425 u s 256 / sqrt(2) each, and sqrt(K / 256) times that for
the K rows together.  Twice that is allowed; one running sum over K rows has
sqrt(K / 256) times more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_fp64_projection_sums_in_blocks(cuda, tg):
    import torch
    K, n, n1, cols = 16384, 1024, 512, 24
    gen = torch.Generator(device="cuda")
    gen.manual_seed(23)
    a = tg.empty_colmajor(K, n, torch.float64, "cuda")
    a.t().normal_(generator=gen)
    a2 = a[:, n1:n1 + cols].cpu().numpy()
    r = tg.qr_(a)
    q1 = a[:, :cols].cpu().numpy()
    r12 = r[:cols, n1:n1 + cols].cpu().numpy()
    exact = q1.T.astype(np.longdouble) @ a2.astype(np.longdouble)
    err = (r12 - exact).astype(np.float64)
    s = np.sqrt(np.mean(np.square(q1)) * np.mean(np.square(a2)))
    bar = 2 * 0.425 * 2.0 ** -53 * s * 256 / np.sqrt(2.0) * np.sqrt(K / 256)
    assert np.sqrt(np.mean(np.square(err))) <= bar, (np.sqrt(np.mean(np.square(err))), bar)
