"""GPU: waits that give up in the streaming kernel. The wait limit holds for it as for the other tensor kernels: zero expires at the
first wait that is not satisfied at once, 3 us somewhere in the run, with copies and MMAs on their way. The call reports the timeout
(or, with the longer limit, may get through, exactly), and the handle then runs the same anneals exactly."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import _lib, instances as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,chains", [(8300, 1, 300), (8300, 2, 100)])
def test_expiry_and_recovery(cuda, n, K, chains):
    inst = I.complete_pm1(n, 6) if K == 1 else I.random_kbit(n, K, 6, pzero=0.4, bmax=3)
    dev = A.DeviceInstance(inst)
    tb = A.Tables.from_schedule(A.Schedule(S=20, t0=30.0, lam=1.05, ramp=True))
    run = lambda: A.run(dev, tb, 1, 0, chains, trace=True, engine="tensor")
    want = run()
    assert want.kernel == "tensor-int8"
    L = _lib.load()
    old = L.anc_get_wait_ns()

    def same(r):
        return all(np.array_equal(getattr(r, k), getattr(want, k)) for k in ("spins", "flips", "sum_sh", "trace"))

    for ns in (0, 3000, 0):
        L.anc_set_wait_ns(ns)
        try:
            r = run()
            assert ns and same(r)
        except A.AncError as e:
            assert e.code == -3
        finally:
            L.anc_set_wait_ns(old)
        assert same(run())
