"""GPU: calls under AUTO and sparse batches with little device memory left, and a batch whose results are large. An engine that
needs operands and workspaces gives way to one that needs none, and memory that the library keeps between batches is given back
before a call is refused for want of it."""
import contextlib
import ctypes as C
import gc

import numpy as np
import pytest
import torch

import anechoic_b200 as A
from anechoic_b200 import instances as I

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def _free_left(target):
    """Takes device memory straight from the driver until none is left (freed pieces that it holds back included), then gives
    `target` bytes back."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cuda = C.CDLL("libcuda.so.1")
    held = []
    try:
        for step in (4096 * MB, 256 * MB, 16 * MB, 2 * MB):
            p = C.c_uint64()
            while cuda.cuMemAlloc_v2(C.byref(p), C.c_size_t(step)) == 0:
                held.append((step, p))
                p = C.c_uint64()
        given = 0
        while held and given < target:
            step, p = held.pop()
            cuda.cuMemFree_v2(p)
            given += step
            while given > target:                    # the part of a large block that is too much
                p = C.c_uint64()
                assert cuda.cuMemAlloc_v2(C.byref(p), C.c_size_t(2 * MB)) == 0
                held.append((2 * MB, p))
                given -= 2 * MB
        yield
    finally:
        for _, p in held:
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
    with _free_left(8 * MB):
        r = A.run(dev, tb, 3, 0, chains)
    assert r.kernel == "plain"
    assert np.array_equal(r.spins, want.spins) and np.array_equal(r.spins, plain.spins)
    assert A.run(dev, tb, 3, 0, chains).kernel == want.kernel         # with room again, the quicker kernel


def test_kept_batch_memory_is_given_back(cuda):
    """A batch leaves a block of 160 MB for the next; a larger one fits only where that block was."""
    dev = A.DeviceInstance(I.torus(10, 20, 3))
    tb = A.Tables.from_schedule(A.Schedule(S=2000, t0=6.0, t1=0.5, q=1.5, kappa=2.0))
    small = dict(dev=dev, tb=tb, seed=1, trial_offset=0, nchains=20000, trace=True)       # 8 KB of trace an anneal
    large = dict(small, nchains=30000)
    gc.collect()                             # no block is kept but this one's
    first = A.run_batch([small])[0]
    with _free_left(150 * MB):
        r = A.run_batch([large])[0]
    want = A.run_batch([large])[0]
    assert np.array_equal(r.trace, want.trace) and np.array_equal(r.spins, want.spins)
    assert np.array_equal(first.trace, want.trace[:20000])


def test_batch_without_room_for_groups(cuda):
    """Groups of replicas keep their fields in device memory (two classes here, 29 and 38 MB); without room none are formed."""
    gc.collect()                             # the last instance takes the block kept for batches with it
    insts = [I.random_graph(3000, 15000, True, 1), I.random_graph(7900, 40000, True, 2)]
    tb = A.Tables.from_schedule(A.Schedule(S=20, t0=6.0, t1=0.5, q=1.5, kappa=2.0))
    want = [A.run(A.DeviceInstance(i), tb, 4, 5000 * k, 1300) for k, i in enumerate(insts)]
    jobs = [dict(dev=A.DeviceInstance(i), tb=tb, seed=4, trial_offset=5000 * k, nchains=1300) for k, i in enumerate(insts)]
    with _free_left(24 * MB):
        outs = [A.run_batch(jobs) for _ in range(2)]
    for got in outs:
        for a, b in zip(got, want):
            assert np.array_equal(a.spins, b.spins) and np.array_equal(a.flips, b.flips) and np.array_equal(a.sum_sh, b.sum_sh)


def test_results_above_the_staged_size(cuda):
    """27000 anneals of 20000 spins return 69 MB, which go straight to the caller's arrays; their halves are staged."""
    dev = A.DeviceInstance(I.torus(100, 200, 4, bmax=2))
    tb = A.Tables.from_schedule(A.Schedule(S=2, t0=6.0, t1=0.5, q=1.5, kappa=2.0))
    job = dict(dev=dev, tb=tb, seed=1, trial_offset=0, nchains=27000, trace=True)
    whole = A.run_batch([job])[0]
    for a in (0, 13500):
        half = A.run_batch([dict(job, trial_offset=a, nchains=13500)])[0]
        for name in ("spins", "sum_sh", "sum_bs", "flips", "trace"):
            assert np.array_equal(getattr(whole, name)[a:a + 13500], getattr(half, name)), name
