"""GPU test of tc_nn_kernel's bounded waits, with a status word of its own.

A whole qr call cannot show them: its other TMA-fed kernels set the same word.
So the launch function is called through its C++ symbol.  With the limit at 0
polls (tsqr_debug_set_wait_limit) every role gives up at its first wait: the
word is set, C is not touched, the copies in flight land, TMEM is freed.  With
the default limit the next call gives C + alpha A B and leaves the word alone.

Bar of the product, element by element: TF32x3 keeps each product to 2^-20
and each of the 3 K accumulated terms adds one FP32 rounding, both relative to
|A| |B|; the sum with C one more."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

SYMBOL = "_ZN4tsqr14tc_nn_residentEliifPKflS1_lPflPiP11CUstream_st"


@pytest.mark.parametrize("m,n,k", [(4096, 128, 128), (1000, 200, 64), (3333, 40, 300), (100, 17, 500),
                                   (60000, 256, 256)])
def test_wait_that_runs_out_is_reported_by_the_kernel_itself(cuda, tg, m, n, k):
    import torch
    L = tg.lib()
    fn = getattr(L, SYMBOL)
    fn.restype = ctypes.c_bool
    i64, p = ctypes.c_int64, ctypes.c_void_p
    fn.argtypes = [i64, ctypes.c_int, ctypes.c_int, ctypes.c_float, p, i64, p, i64, p, i64, p, p]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    ld = (m + 3) // 4 * 4  # TMA takes leading dimensions of whole 16 bytes
    a, b, c = (tg.empty_colmajor(r, q, torch.float32, "cuda", ld=l) for r, q, l in ((m, k, ld), (k, n, k), (m, n, m)))
    for x in (a, b, c):
        x.copy_(torch.rand(x.shape, generator=gen, device="cuda") * 2 - 1)
    c0 = c.clone()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def call():
        s = torch.cuda.current_stream().cuda_stream
        assert fn(m, n, k, -0.5, a.data_ptr(), ld, b.data_ptr(), k, c.data_ptr(), m, status.data_ptr(), s)
        torch.cuda.synchronize()

    try:
        assert L.tsqr_debug_set_wait_limit(0) == 0
        call()
    finally:
        L.tsqr_debug_set_wait_limit(-1)
    assert int(status) == 1
    assert torch.equal(c, c0)
    status.zero_()
    call()
    assert int(status) == 0
    a64, b64, c64 = a.double(), b.double(), c0.double()
    bar = 0.5 * (2.0 ** -20 + 3 * k * 2.0 ** -24) * (a64.abs() @ b64.abs()) + 2.0 ** -23 * c64.abs()
    err = (c.double() - (c64 - 0.5 * a64 @ b64)).abs()
    assert bool((err <= bar).all()), float((err / bar).max())
