"""GPU: the streaming kernel with more replicas than the 256 it advances at once. The pairs of replica groups follow one another
in the same exchange buffers, and a CTA may enter the next pair while another still loads the last step's updates of this one:
each pair's buffers must not be the ones that the last step of the pair before it filled, for even and odd step counts. Every
output of a run of several pairs equals that of one run per pair, the fields equal J s + b, and sampled anneals the restatement.
Integers: bit-exact."""
import numpy as np
import pytest
import torch

import anechoic_b200 as A
from anechoic_b200 import instances as I
from tests.test_parity_plain import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,chains,S", [(6200, 1, 600, 20), (8300, 1, 300, 40), (8300, 2, 520, 41), (12300, 1, 260, 10)])
def test_pairs_in_turn(cuda, oracle, n, K, chains, S):
    g = torch.Generator("cuda").manual_seed(n)
    r = torch.randint(0, 4, (n, n), generator=g, dtype=torch.int8, device="cuda")
    J = torch.triu((r & 1) * 2 - 1 if K == 1 else (r & 1) - (r >> 1), 1)
    J = J + J.T
    inst = A.Instance(n=n, dense=J.cpu().numpy())
    sc = dict(S=S, t0=30.0, t1=5.0, q=4.0, lam=1.05, ramp=True)
    dev, tb = A.DeviceInstance(inst), A.Tables.from_schedule(A.Schedule(**sc))
    opts = dict(trace=True, fields=True, **({"engine": "tensor"} if n > 8192 else {"flip_fraction": 0.4}))
    got = A.run(dev, tb, 5, 40, chains, **opts)
    assert got.kernel == "tensor-int8"
    for a in range(0, chains, 256):
        b = min(chains, a + 256)
        one = A.run(dev, tb, 5, 40 + a, b - a, **opts)
        for name in ("spins", "flips", "sum_bs", "trace", "sum_sh", "fields"):
            assert np.array_equal(getattr(got, name)[a:b], getattr(one, name)), (name, a)
    bits = np.unpackbits(got.spins.view(np.uint8), axis=1, bitorder="little")[:, :n]
    s = torch.as_tensor(bits, device="cuda").float() * 2 - 1
    assert torch.equal((s @ J.float()).int().cpu(), torch.as_tensor(got.fields))
    for c in (0, 255, 256, chains - 1):
        ref = oracle.run_batch(n, oracle.tables(**sc), 5, 40 + c, 1, dense=inst.dense)
        assert_same(got, {k: v[0] for k, v in ref.items()}, c, f"n={n} chain {c}")
