"""GPU: the CSR-pass tuner keeps its choice per form of the sparse launch. The forms are different kernels and a variant
means something else in each, so a run in a form that has not been tuned yet probes that form, whatever ran before."""
import ctypes as C

import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import _lib, instances as I

pytestmark = pytest.mark.gpu


def _tuning(dev):
    v, us = C.c_int(-7), (C.c_double * 4)()
    _lib.check(_lib.load().anc_sparse_tuning(dev._h, C.byref(v), us))
    return v.value, list(us)


def test_each_form_is_tuned_on_its_first_run(cuda):
    inst = I.random_graph(2000, 20000, True, 5, bmax=2)
    tb = A.Tables.from_schedule(A.Schedule(S=64, t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True))
    dev = A.DeviceInstance(inst)
    ref = A.run(A.DeviceInstance(inst), tb, 3, 0, 2400)
    seen = []
    for chains in (16, 290, 600, 2400):       # one anneal per SM, two, four or more, groups
        r = A.run(dev, tb, 3, 0, chains)
        assert np.array_equal(r.spins, ref.spins[:chains]) and np.array_equal(r.flips, ref.flips[:chains])
        v, us = _tuning(dev)
        assert us[v] == min(us) > 0
        seen.append(us)
    assert all(a != b for k, a in enumerate(seen) for b in seen[:k])        # four probes
    # a step takes longer the more anneals share an SM: 4, 6, 14 and 23 us here
    assert min(seen[0]) < min(seen[2]) < min(seen[3])
    for chains in (16, 600, 2400, 290):       # tuned forms are not probed again
        A.run(dev, tb, 3, 0, chains)
        assert _tuning(dev)[1] == seen[3]
