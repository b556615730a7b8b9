"""GPU: the rule that picks the form of a sparse launch (sparse_engine.cu): parity with the golden-model restatement on both sides
of its lines, and no number of anneals slower than waves of one anneal per SM, which every size can run as."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import instances as I
from tests.test_parity_plain import assert_same

pytestmark = pytest.mark.gpu

SCHED = dict(t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True)


def _graph(n, degree, unit):
    g = I.random_graph(n, n * degree // 2, True, 7, bmax=2)
    if unit:
        return g
    v = g.val.astype(np.int16) * (1 + (g.col + np.repeat(np.arange(n), np.diff(g.row_ptr))) % 5)     # symmetric
    return A.Instance(n=n, row_ptr=g.row_ptr, col=g.col, val=v.astype(np.int8), bias=g.bias)


# n, degree, +-1 weights, anneals (148 SMs): 2 / 3 / 4 / 5 per SM, one past each, and the sizes where fewer CTAs fit
CASES = [(700, 70, False, 370), (700, 70, False, 371), (900, 33, True, 739), (900, 33, True, 740), (2000, 50, True, 887),
         (2000, 50, True, 888), (5000, 50, True, 445), (7900, 10, True, 1185), (8449, 16, True, 445), (8500, 15, False, 445),
         (10880, 9, True, 296), (10881, 9, True, 296), (10900, 13, False, 444), (10900, 12, True, 445), (10900, 11, True, 445),
         (10900, 20, False, 741), (13000, 4, True, 300), (20000, 4, False, 149)]


@pytest.mark.parametrize("n,degree,unit,chains", CASES)
def test_forms_at_the_lines(cuda, oracle, n, degree, unit, chains):
    inst = _graph(n, degree, unit)
    sc = dict(SCHED, S=5)
    r = A.run(A.DeviceInstance(inst), A.Tables.from_schedule(A.Schedule(**sc)), 11, 40, chains, trace=True, fields=True)
    for c in (0, 7, chains // 2, chains - 1):
        ref = oracle.run_batch(n, oracle.tables(**sc), 11, 40 + c, 1, csr=inst.to_csr(), bias=inst.bias)
        assert_same(r, {k: v[0] for k, v in ref.items()}, c, f"n={n} chain {c}")
    assert np.array_equal(r.fields[chains - 1], inst.fields(r.spins[chains - 1]))


@pytest.mark.parametrize("n,degree,unit,chains", [(2000, 40, True, 310), (4000, 80, True, 310), (7900, 20, True, 1200),
                                                  (16000, 20, True, 444), (10000, 48, True, 592), (800, 80, False, 310)])
def test_not_slower_than_waves_of_one_per_sm(cuda, n, degree, unit, chains):
    inst = _graph(n, degree, unit)
    dev, tb = A.DeviceInstance(inst), A.Tables.from_schedule(A.Schedule(**SCHED, S=150))
    one, many = (min(A.run(dev, tb, 3, 0, c).device_ms for _ in range(4)) for c in (148, chains))
    assert many <= 1.1 * -(-chains // 148) * one, (many, one)
