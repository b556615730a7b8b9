"""GPU: calls under AUTO with little device memory left. An engine that needs operands and workspaces gives way to one that
needs none."""
import contextlib
import ctypes as C

import numpy as np
import pytest
import torch

import anechoic_b200 as A
from anechoic_b200 import instances as I

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def _free_left(target):
    """Holds device memory, straight from the driver, so that between `target` and `target` + 2 MB are free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cuda = C.CDLL("libcuda.so.1")
    held = []
    try:
        for step in (4096 * MB, 256 * MB, 16 * MB, 2 * MB):
            while torch.cuda.mem_get_info()[0] - step >= target:
                p = C.c_uint64()
                assert cuda.cuMemAlloc_v2(C.byref(p), C.c_size_t(step)) == 0
                held.append(p)
        yield
    finally:
        for p in held:
            cuda.cuMemFree_v2(p)


@pytest.mark.parametrize("n,K,chains", [(5000, 1, 128), (5000, 4, 130)])
def test_auto_without_room_for_operands(cuda, n, K, chains):
    """The planes kernel's and the streaming kernel's copies of J (13 and 27 MB) do not fit: the plain engine runs."""
    inst = I.complete_pm1(n, 5) if K == 1 else I.random_kbit(n, K, 5, pzero=0.3, bmax=2)
    tb = A.Tables.from_schedule(A.Schedule(S=6, t0=30.0 if K == 1 else 500.0, lam=1.05, ramp=True))
    want = A.run(A.DeviceInstance(inst), tb, 3, 0, chains)
    assert want.kernel != "plain"
    plain = A.run(A.DeviceInstance(inst), tb, 3, 0, chains, engine="plain")     # its kernels are loaded
    dev = A.DeviceInstance(inst)
    with _free_left(9 * MB):
        r = A.run(dev, tb, 3, 0, chains)
    assert r.kernel == "plain"
    assert np.array_equal(r.spins, want.spins) and np.array_equal(r.spins, plain.spins)
    assert A.run(dev, tb, 3, 0, chains).kernel == want.kernel         # with room again, the quicker kernel
