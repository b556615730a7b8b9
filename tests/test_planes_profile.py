"""GPU: the planes kernel's phase profile at sizes that no other tensor kernel takes, and the anneals it leaves unchanged."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import instances as I

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chains,ctas", [(2501, 100, 64), (5000, 130, 128), (2000, 9, 64)])
def test_profiled_run(cuda, n, chains, ctas):
    dev = A.DeviceInstance(I.complete_pm1(n, 3))
    S = 500
    tb = A.Tables.from_schedule(A.Schedule(S=S, lam=1.05, ramp=True))
    plain = A.run(dev, tb, 5, 0, chains, engine="tensor", tensor_kind="planes")
    r = A.run(dev, tb, 5, 0, chains, engine="tensor", tensor_kind="planes", profile=True)
    assert r.kernel == "tensor-planes" and np.array_equal(r.spins, plain.spins) and np.array_equal(r.flips, plain.flips)
    p = r.profile
    assert p["ctas"] == ctas and p["cluster"] == 1
    # the phases are parts of a step, and the steps' cycles over the launch's time are the SM clock, as a mean over the CTAs
    assert 0 < p["decide"] < p["step"] and 0 < p["exchange"] < p["step"]
    assert 1.0e9 < p["step"] * S / (r.device_ms * 1e-3) < 2.1e9
