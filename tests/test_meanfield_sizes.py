"""GPU: the mean-field kernels at the sizes where their launch form changes -- every number of 256-column chunks from one to
eight (J in tensor memory; 16, 32 and 64 replicas per group), nine to twelve (two row blocks per CTA), launch sequences
beyond -- and at the checkpoint edges (a last segment of one step), against the FP64 recurrence.

The schedule keeps the map a contraction, so that rounding is not amplified with the steps: T >= 2 sqrt(n) and
||J|| <= 2 sqrt(0.6 n) give beta ||J|| <= 0.39, and beta gamma <= 0.07 with the counted correction. The error of one step
is at most 1e-6 (test_meanfield.py), so that of any number of steps is at most 1e-6 / (1 - 0.46) in the norm of the
contraction, 1e-5 per element with a factor 5 in hand; the five derivatives, sums of S n f32 products, 1e-3 relative."""
import math

import pytest
import torch

from anechoic_b200 import instances as I
from anechoic_b200.meanfield import MeanField, SoftSchedule, initial_magnetisations, relax
from tests.test_meanfield import _case, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,S", [(256, 17), (257, 33), (700, 18), (1000, 16), (1281, 1), (1500, 33), (1600, 5), (2048, 18),
                                 (2049, 17), (2800, 33), (3072, 2), (3073, 17)])
def test_forms_vs_fp64(cuda, n, S):
    inst = I.random_kbit(n, 2, 900 + n, pzero=0.4, bmax=3)
    theta = (4.0 * math.sqrt(n), math.log(2.0), 1.0, 0.5, 1.05)
    mr = torch.rand(64, n, generator=torch.Generator().manual_seed(3)) * 2 - 1
    r = _case(inst, S, 64, "counted", theta, m0=mr)
    assert (r["mS"] - r["m64"]).abs().max().item() <= 1e-5
    assert _rel(r["g"], r["g64"]) <= 1e-3, (r["g"].tolist(), r["g64"].tolist())


def test_calls_on_one_context_repeat_bit_for_bit(cuda):
    """Lengths in turn on one context (its buffers grow and hold the previous call's values), and a call that gives up."""
    inst = I.complete_pm1(900, 4)
    mf, m0 = MeanField(inst), None
    m0 = mf.pad(initial_magnetisations(900, 64, 1))
    g = mf.pad(torch.randn((64, 900), generator=torch.Generator().manual_seed(2)) / 900)

    def call(S, ctx):
        v = [x.detach().cuda().requires_grad_() for x in SoftSchedule(S=S).vectors(
            torch.tensor([20.0, math.log(6.0), 3.0, 0.0, 1.05], dtype=torch.float64))]
        m = relax(ctx, *v, m0)
        return [m.detach()] + list(torch.autograd.grad(m, v, g))

    want = {S: call(S, MeanField(inst)) for S in (5, 33)}
    for S in (5, 33, 5, 33):
        assert all(torch.equal(a, b) for a, b in zip(call(S, mf), want[S]))
    mf.set_wait_ns(0)
    with pytest.raises(Exception, match="wait expired"):
        call(33, mf)
    mf.set_wait_ns(2_000_000_000)
    assert all(torch.equal(a, b) for a, b in zip(call(33, mf), want[33]))
