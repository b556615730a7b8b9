"""GPU parity of the planes kernel (J as one or two e2m1 planes, NP = 2048 .. 6144) with the golden-model restatement: at
the edges of every compiled geometry (rounds per lane 8, 9 .. 12, 13 .. 16, 17 .. 20, 21 .. 24), with one and two planes,
bias, the clamped decision, partial and several replica groups, and after a wait that gave up. Integer results: bit-exact."""
import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import _lib
from anechoic_b200 import instances as I
from tests.test_parity_plain import assert_same

pytestmark = pytest.mark.gpu

# n, K, bias bound, anneals, steps. The geometry follows from the rounds (RP), the planes and the replica groups: fewer
# groups take fewer lanes per thread (LT).
CASES = [(17, 4, 3, 1, 40), (2048, 4, 7, 130, 12), (2000, 4, 0, 260, 8),      # RP 8, two planes: LT 2, 2 and 4
         (1000, 3, 2, 9, 12), (1, 3, 1, 400, 6), (2048, 3, 0, 530, 6),          # RP 8, one plane: LT 2, 4 and 8
         (2049, 1, 0, 33, 10), (2501, 2, 2, 100, 12), (2500, 1, 0, 300, 6),     # RP 12 (R 9, 10), one plane: LT 2, 2, 4
         (3072, 4, 40, 260, 6), (3000, 3, 0, 5, 12), (3072, 1, 0, 700, 4),      # RP 12 (R 12): two planes; LT 2; two waves
         (3073, 1, 0, 300, 6), (4096, 4, 0, 129, 5), (4096, 2, 3, 64, 5),       # RP 16 (R 13, 16): LT 2, two planes, LT 1
         (4097, 2, 9, 130, 5), (5120, 1, 0, 31, 6),                             # RP 20 (R 17, 20)
         (5121, 1, 0, 17, 5), (6144, 2, 0, 129, 4)]                             # RP 24 (R 21, 24)


def _instance(n, K, bmax):
    return I.complete_pm1(n, 50 + n) if K == 1 else I.random_kbit(n, K, 50 + n, pzero=0.2, bmax=bmax)


def _same(r, ref, what):
    for c in range(len(r.spins)):
        assert_same(r, {k: v[c] for k, v in ref.items()}, c, f"{what} chain {c}")


@pytest.mark.parametrize("n,K,bmax,chains,S", CASES)
def test_planes_vs_oracle(cuda, oracle, n, K, bmax, chains, S):
    inst = _instance(n, K, bmax)
    dev = A.DeviceInstance(inst)
    sc = dict(S=S, t0=float(1.0 + 0.5 * np.sqrt(n) * (1 << (K - 1))), t1=1.0, q=2.0, lam=0.7, ramp=True)
    tb = A.Tables.from_schedule(A.Schedule(**sc))
    r = A.run(dev, tb, 5, 40, chains, trace=True, fields=True, engine="tensor", tensor_kind="planes")
    assert r.kernel == "tensor-planes"
    _same(r, oracle.run_batch(n, oracle.tables(**sc), 5, 40, chains, dense=inst.dense, bias=inst.bias), f"n={n} K={K}")
    assert np.array_equal(r.fields[-1], inst.fields(r.spins[-1]))


def test_planes_clamped_decision(cuda, oracle):
    """Row sums above 2^15: the range plan needs the clamp, and wide=1 forces it where it does not."""
    k4 = I.random_kbit(2500, 4, 5, pzero=0.0, bmax=30000)
    sc = dict(S=10, t0=900.0, t1=40.0, q=2000.0, lam=0.3, ramp=True)
    dev, tb = A.DeviceInstance(k4), A.Tables.from_schedule(A.Schedule(**sc))
    assert not dev.range_plan(tb)["plain_ok"]
    ref = oracle.run_batch(2500, oracle.tables(**sc), 1, 0, 9, dense=k4.dense, bias=k4.bias)
    _same(A.run(dev, tb, 1, 0, 9, trace=True, engine="tensor", tensor_kind="planes"), ref, "clamp")
    pm1 = I.complete_pm1(2500, 6)
    dev = A.DeviceInstance(pm1)
    sc = dict(S=12, t0=30.0, t1=5.0, q=4.0, lam=1.05, ramp=True)
    tb = A.Tables.from_schedule(A.Schedule(**sc))
    ref = oracle.run_batch(2500, oracle.tables(**sc), 1, 0, 9, dense=pm1.dense)
    _same(A.run(dev, tb, 1, 0, 9, trace=True, engine="tensor", tensor_kind="planes", wide=1), ref, "wide")


def test_planes_limits_and_expiry(cuda, oracle):
    """Refused outside its range (two planes above n = 4096, one above 6144, wide fields); a wait limit of 0 reports the
    timeout and the handle then runs exactly."""
    tb = A.Tables.from_schedule(A.Schedule(S=5, t0=900.0, t1=40.0, q=4.0))
    for inst in (I.random_kbit(4097, 4, 1), I.complete_pm1(6145, 1), I.random_kbit(4096, 4, 2, pzero=0.0, bmax=32767)):
        bound = inst.stats()["hmax"] + inst.stats()["bmax"]
        if inst.n == 4096 and bound < 1 << 16:
            continue
        with pytest.raises(A.AncError) as e:
            A.run(A.DeviceInstance(inst), tb, 1, 0, 2, engine="tensor", tensor_kind="planes")
        assert e.value.code == -1
    inst = I.complete_pm1(2500, 6)
    dev = A.DeviceInstance(inst)
    sc = dict(S=8, t0=30.0, t1=5.0, q=4.0, lam=1.05, ramp=True)
    tb = A.Tables.from_schedule(A.Schedule(**sc))
    L = _lib.load()
    old = L.anc_get_wait_ns()
    L.anc_set_wait_ns(0)
    try:
        with pytest.raises(A.AncError) as e:
            A.run(dev, tb, 3, 0, 130, engine="tensor", tensor_kind="planes")
        assert e.value.code == -3
    finally:
        L.anc_set_wait_ns(old)
    _same(A.run(dev, tb, 3, 0, 130, trace=True, engine="tensor", tensor_kind="planes"),
          oracle.run_batch(2500, oracle.tables(**sc), 3, 0, 130, dense=inst.dense), "after expiry")


@pytest.mark.parametrize("n,K,chains", [(4100, 4, 130), (8192, 4, 3), (7000, 1, 300)])
def test_auto_streams_between_the_other_kernels(cuda, oracle, n, K, chains):
    """Sizes above the planes kernel's (two planes n > 4096, one plane n > 6144) up to 8192: AUTO runs the streaming kernel
    (32 columns per lane, 17 to 32 rounds); ANC_ENGINE_TENSOR still refuses them."""
    inst = _instance(n, K, 5)
    dev = A.DeviceInstance(inst)
    sc = dict(S=4, t0=float(1.0 + 0.5 * np.sqrt(n) * (1 << (K - 1))), t1=1.0, q=2.0, lam=0.7, ramp=True)
    tb = A.Tables.from_schedule(A.Schedule(**sc))
    r = A.run(dev, tb, 5, 40, chains, trace=True, fields=True, flip_fraction=0.5)
    assert r.kernel == "tensor-int8"
    _same(r, oracle.run_batch(n, oracle.tables(**sc), 5, 40, chains, dense=inst.dense, bias=inst.bias), f"n={n} K={K}")
    assert np.array_equal(r.fields[-1], inst.fields(r.spins[-1]))
    with pytest.raises(A.AncError):
        A.run(dev, tb, 5, 40, 2, engine="tensor")
