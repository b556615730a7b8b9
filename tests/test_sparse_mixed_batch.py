"""GPU: anc_run_batch calls whose jobs differ in what the sparse launches have to keep apart -- the clamped decision, the
length of the schedule, the size of the results -- against the golden-model restatement (integers: bit-exact)."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import instances as I
from tests.test_parity_plain import assert_same

pytestmark = pytest.mark.gpu

SCHED = dict(S=7, t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True)


def _needs_clamp(inst):
    """The instance with one bias at the accepted bound: (max row sum + bias) 2^16 leaves no room in 32 bits."""
    bias = np.zeros(inst.n, np.int32)
    bias[inst.n // 2] = 32767
    return A.Instance(n=inst.n, row_ptr=inst.row_ptr, col=inst.col, val=inst.val, bias=bias)


@pytest.mark.parametrize("clamped", ["sparse group", "sparse weighted", "dense"])
def test_clamped_job_beside_unclamped_groups(cuda, oracle, clamped):
    """More than eight sparse anneals per SM; one job needs the clamped decision, the others do not."""
    insts = [I.random_graph(500, 3000, True, 1, bmax=2), I.torus(45, 46, 5, bmax=2), I.random_graph(3000, 15000, True, 2)]
    counts = [500, 401, 300]
    if clamped == "sparse group":
        insts.append(_needs_clamp(I.random_graph(700, 4200, True, 3)))
    elif clamped == "sparse weighted":
        g = I.random_graph(700, 4200, True, 3)
        w = (g.val.astype(np.int16) * (1 + (g.col + np.repeat(np.arange(700), np.diff(g.row_ptr))) % 3)).astype(np.int8)
        insts.append(_needs_clamp(A.Instance(n=700, row_ptr=g.row_ptr, col=g.col, val=w)))
    else:
        d = I.complete_pm1(300, 4)
        bias = np.zeros(300, np.int32)
        bias[7] = -32767
        insts.append(A.Instance(n=300, dense=d.dense, bias=bias))
    counts.append(9)
    tb = A.Tables.from_schedule(A.Schedule(**SCHED))
    devs = [A.DeviceInstance(i) for i in insts]
    assert [d.range_plan(tb)["plain_ok"] for d in devs] == [True, True, True, False]
    outs = A.run_batch([dict(dev=d, tb=tb, seed=5, trial_offset=1000 * k, nchains=c, trace=True)
                        for k, (d, c) in enumerate(zip(devs, counts))])
    for k, (i, c, r) in enumerate(zip(insts, counts, outs)):
        for ch in (0, 1, 7, 8, c // 2, c - 1):
            J = dict(csr=i.to_csr()) if i.is_sparse else dict(dense=i.dense)
            ref = oracle.run_batch(i.n, oracle.tables(**SCHED), 5, 1000 * k + ch, 1, bias=i.bias, **J)
            assert_same(r, {kk: v[0] for kk, v in ref.items()}, ch, f"job {k} chain {ch}")
