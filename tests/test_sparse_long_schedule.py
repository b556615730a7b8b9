"""GPU: an anneal's flip total needs 64 bits on a long schedule, in every form of the sparse launch. With a self-coupling far
below zero every spin flips at every step (z = s h + q is below -2T whatever the draw), so the totals and the spins are known
without a reference run: n S flips, and after an even number of steps the initial spins, which a two-step run returns."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import instances as I

pytestmark = pytest.mark.gpu


def _tables(S):
    return A.Tables.from_schedule(A.Schedule(S=S, t0=1.0, t1=1.0, q=-200.0))


def test_flip_total_of_a_long_schedule_in_groups(cuda):
    """7936 spins x 280000 steps = 2.2e9 flips, above 2^31. The short jobs put the call above eight anneals per SM."""
    one_edge = I._from_edges(7936, np.array([3]), np.array([5000]), np.array([1]), None, "edge")
    filler = I.torus(10, 20, 3)
    dev, other = A.DeviceInstance(one_edge), A.DeviceInstance(filler)
    S = 280000
    outs = A.run_batch([dict(dev=dev, tb=_tables(S), seed=9, trial_offset=0, nchains=8),
                        dict(dev=other, tb=_tables(2), seed=9, trial_offset=50, nchains=1300)])
    short = A.run(dev, _tables(2), 9, 0, 8)
    assert np.array_equal(short.flips, np.full(8, 2 * 7936))
    assert np.array_equal(outs[0].flips, np.full(8, S * 7936, np.int64))
    assert np.array_equal(outs[1].flips, np.full(1300, 2 * 200))
    assert np.array_equal(outs[0].spins, short.spins)
