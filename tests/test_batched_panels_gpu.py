"""Batches of small problems, 17 to 32 columns wide, with more tiles in all than
the column split runs at once (2 per SM): the launch then factors them as two
panels of 16 columns, while each problem alone takes the column split.  Tree
and signs are the same, the rounding is not: R and Q agree with the
single-problem call to the sum of both errors, 10 n u each, and every problem
meets the parity bar itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24


@pytest.mark.parametrize("shapes", [[(3000, 32)] * 40 + [(2700, 24)] * 50,
                                    [(300, 20)] * 310,
                                    [(512, 17), (513, 31), (40, 32)] * 120])
def test_batch_of_small_problems_in_panels(cuda, tg, shapes):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(17)
    assert sum(-(-m // 512) for m, _ in shapes) > 2 * torch.cuda.get_device_properties(0).multi_processor_count
    As = [tg.empty_colmajor(m, n, torch.float32, "cuda") for m, n in shapes]
    for a in As:
        a.t().uniform_(-1.0, 1.0, generator=gen)
    A0 = [a.clone() for a in As]
    Rs = tg.tsqr_batched_(As)
    torch.cuda.synchronize()
    for (m, n), a0, q, r in zip(shapes, A0, As, Rs):
        q1 = a0.t().clone().t()
        r1 = tg.tsqr_(q1)
        bar = 10 * n * U32
        a64, q64, r64 = a0.double(), q.double(), r.double()
        assert float((a64 - q64 @ r64).norm() / a64.norm()) <= bar
        assert float((q64.t() @ q64 - torch.eye(n, dtype=torch.float64, device="cuda")).norm()) <= bar
        assert float((r1.double() - r64).abs().max()) <= 2 * bar * float(r64.abs().max())
        if m >= 2 * n:  # a nearly square problem is not well conditioned: Q may turn with its rounding
            assert float((q1.double() - q64).abs().max()) <= 2 * bar
