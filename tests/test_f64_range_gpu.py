"""FP64 trees of columns whose squared norms are small, subnormal or large, and
of columns of very different norms in one matrix, against an FP64 tree of the
same matrix scaled to order 1 (columns times powers of two: the same Q, the
same R with its columns scaled).  Several tiles, so that the levels above the
first take part, at each tile width.

Bars.  A squared norm of entries near 2^e sums products near 2^2e; where those
are subnormal each is rounded by up to 2^-1075 in place of u times itself, so
the relative error of a norm and of a dot product grows by up to
d(e) = 3 2^(-1075 - 2 e) (uniform entries: mean square 1/3).  Every bar is the
one of the ordinary tests with u + d in place of u."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U64 = 2.0 ** -53


def run(tg, A):
    import torch
    m, n = A.shape
    d = tg.empty_colmajor(m, n, torch.float64, "cuda")
    d.copy_(torch.from_numpy(np.ascontiguousarray(A)))
    R = tg.tsqr_(d)
    torch.cuda.synchronize()
    return d.t().contiguous().cpu().numpy().T, R.t().contiguous().cpu().numpy().T


def rounding(exponents):
    return U64 + max(3.0 * 2.0 ** (-1075.0 - 2.0 * e) for e in exponents)


def check(orc, tg, m, n, exponents, seed):
    """Columns times 2^exponents[c]; metrics on the columns scaled back."""
    e = np.asarray(exponents)
    A = orc.fill_uniform(m, n, np.float64, seed=seed)
    Q, R = run(tg, np.asfortranarray(np.ldexp(A, e[None, :])))
    Rs = np.asfortranarray(np.ldexp(R, -e[None, :]))
    assert np.isfinite(Q).all() and np.isfinite(Rs).all()
    met = orc.metrics(A, Q, Rs)
    bar = 10 * n * rounding(exponents)
    assert met["backward"] <= bar and met["orth"] <= bar, (met, bar)
    return Q, Rs


@pytest.mark.parametrize("n", [8, 16, 24, 32])
@pytest.mark.parametrize("exponent", [-495, -505, -515, -517, -520, 495, 504])
def test_fp64_extreme_scales(orc, cuda, tg, exponent, n):
    """-495: the general reciprocals with every product normal; from -515 on
    subnormal squared norms (2^-520: norms below 1e-155); 495 and 504: squares
    up to 1e306."""
    m = 5000
    Q, R = check(orc, tg, m, n, [exponent] * n, 8)
    if abs(exponent) <= 505:
        Q1, R1 = run(tg, orc.fill_uniform(m, n, np.float64, seed=8))
        assert np.abs(Q - Q1).max() <= 100 * n * U64
        assert np.abs(R - R1).max() <= 100 * n * U64 * np.abs(R1).max()


@pytest.mark.parametrize("n", [8, 16, 24, 32])
@pytest.mark.parametrize("small,large", [(-518, 0), (0, -518), (-518, 500), (500, -518), (-495, 500)])
def test_fp64_columns_of_very_different_norms(orc, cuda, tg, small, large, n):
    """One column at 2^small and a later one at 2^large, the others of order 1."""
    e = [0] * n
    e[n // 4], e[n // 2 + 1] = small, large
    check(orc, tg, 3000, n, e, 9)


@pytest.mark.parametrize("n", [8, 16, 24, 32])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 1e200])
def test_fp64_a_bad_last_column_leaves_the_others_of_r(orc, cuda, tg, bad, n):
    """An element that makes the last column's norm infinite or NaN: the columns
    of R before it are formed without it and keep every bit."""
    m = 5000
    A = orc.fill_uniform(m, n, np.float64, seed=10)
    _, R0 = run(tg, A)
    A[m - 1, n - 1] = bad
    _, R = run(tg, A)
    assert np.array_equal(R[:, :n - 1], R0[:, :n - 1])
    assert not np.isfinite(R[:, n - 1]).all()
