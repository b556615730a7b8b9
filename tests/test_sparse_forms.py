"""GPU parity of the sparse launch's forms (sparse_engine.cu) with the golden-model restatement, at the sizes where one gives
way to another: one CTA per anneal (up to one anneal per SM), the wide forms (NP > 4096; two anneals per SM), four anneals per
SM, and groups of eight replicas (unit weights, rows of at most 120 edges, NP <= 7936), with bias, the clamped decision, rows
of no edges, and batches that mix the forms. Integer results: bit-exact."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import instances as I
from tests.test_parity_plain import assert_same

pytestmark = pytest.mark.gpu

SCHED = dict(S=7, t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True)
COUNTED = dict(S=7, t0=6.0, t1=0.5, q=1.5, lam=0.8, ramp=True)


def _hub(n, degree):
    """A graph whose vertex 0 has `degree` edges of mixed sign; the last vertex has none."""
    j = np.arange(1, degree + 1)
    return I._from_edges(n, np.zeros(degree, np.int64), j, np.where(j % 3 == 0, -1, 1), None, "hub")


def _weighted(n, seed):
    g = I.random_graph(n, 3 * n, True, seed, bmax=4)
    v = g.val.astype(np.int16) * (1 + (g.col + np.repeat(np.arange(n), np.diff(g.row_ptr))) % 5)     # symmetric
    return A.Instance(n=n, row_ptr=g.row_ptr, col=g.col, val=v.astype(np.int8), bias=g.bias)


CASES = [
    ("one per SM", lambda: I.random_graph(900, 9000, True, 1, bmax=3), 5),
    ("two per SM", lambda: I.random_graph(2048, 4096, True, 2, bmax=3), 200),
    ("wide", lambda: I.torus(60, 70, 3, bmax=2), 3),
    ("wide, many", lambda: I.torus(100, 200, 4, bmax=2), 151),
    ("four per SM", lambda: I.torus(45, 46, 5, bmax=2), 301),
    ("groups", lambda: I.random_graph(1000, 10000, True, 6, bmax=5), 1187),
    ("groups, + edges", lambda: I.random_graph(801, 19176, False, 7), 304),
    ("groups, largest", lambda: I.random_graph(7936, 7936 * 5, True, 8, bmax=1), 1184),
    ("past the groups", lambda: I.random_graph(7937, 7937 * 5, True, 9), 300),
    ("longest row", lambda: _hub(300, 120), 1190),
    ("row too long", lambda: _hub(300, 121), 1190),
    ("weights", lambda: _weighted(700, 10), 1185),
]


def _check(r, inst, sched, seed, off, oracle, chains):
    """chains of the result against the restatement (all of them where few)."""
    for c in chains:
        ref = oracle.run_batch(inst.n, oracle.tables(**sched), seed, off + c, 1, csr=inst.to_csr(), bias=inst.bias)
        assert_same(r, {k: v[0] for k, v in ref.items()}, c, f"n={inst.n} chain {c}")


@pytest.mark.parametrize("name,build,chains", CASES, ids=[c[0] for c in CASES])
@pytest.mark.parametrize("sched,wide", [(SCHED, "auto"), (COUNTED, 1)], ids=["tecT", "counted clamped"])
def test_forms_vs_oracle(cuda, oracle, name, build, chains, sched, wide):
    inst = build()
    dev = A.DeviceInstance(inst)
    r = A.run(dev, A.Tables.from_schedule(A.Schedule(**sched)), 11, 40, chains, trace=True, fields=True, wide=wide)
    assert r.kernel == "plain"
    picks = sorted({0, 1, 7, 8, chains // 2, chains - 2, chains - 1} & set(range(chains)))
    _check(r, inst, sched, 11, 40, oracle, picks)
    assert np.array_equal(r.fields[chains - 1], inst.fields(r.spins[chains - 1]))


def test_batch_mixes_forms(cuda, oracle):
    """More anneals than eight per SM: groups of two sizes, weighted rows, long rows and a 20000-spin torus in one call."""
    insts = [I.random_graph(500, 3000, True, 1, bmax=2), I.random_graph(3000, 9000, False, 2), _weighted(600, 3),
             _hub(400, 150), I.torus(100, 200, 4), I.torus(20, 40, 5, bmax=1)]
    counts = [333, 200, 150, 130, 3, 401]
    tb = A.Tables.from_schedule(A.Schedule(**SCHED))
    outs = A.run_batch([dict(dev=A.DeviceInstance(i), tb=tb, seed=5, trial_offset=1000 * k, nchains=c, trace=True)
                        for k, (i, c) in enumerate(zip(insts, counts))])
    for k, (i, c, r) in enumerate(zip(insts, counts, outs)):
        _check(r, i, SCHED, 5, 1000 * k, oracle, [0, 1, c // 2, c - 1])
