"""GPU: captured anc_run_device calls and the workspaces of their handles. A larger run of the same handle after the capture
leaves the captured call's workspaces in place, so that replays stay exact; and a handle whose workspaces do not exist yet (no
eager call, or one with fewer anneals) can be captured under AUTO, as the engines that need none always could."""
import numpy as np
import pytest
import torch

import anechoic_b200 as A
from anechoic_b200 import _lib, instances as I

pytestmark = pytest.mark.gpu

SCHED = dict(S=9, lam=1.05, ramp=True)
SPARSE = dict(S=9, t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True)

# name, instance, schedule, engine and operand format, anneals captured, anneals of the larger run
CASES = {
    "sparse groups": (lambda: I.random_graph(1000, 10000, True, 6, bmax=2), SPARSE, "auto", "auto", 1187, 2400),
    "planes": (lambda: I.complete_pm1(2501, 4), SCHED, "auto", "auto", 100, 1300),
    "fp4": (lambda: I.complete_pm1(2000, 4), SCHED, "tensor", "fp4", 130, 2100),
    "int8": (lambda: I.random_kbit(2000, 4, 5, pzero=0.2, bmax=3), dict(SCHED, t0=300.0), "tensor", "int8", 130, 1100),
    "streaming": (lambda: I.complete_pm1(6200, 4), SCHED, "auto", "auto", 130, 900),
}


class _Out:
    def __init__(self, n, chains):
        W = A.spin_words(n)
        z = lambda *s: torch.zeros(s, dtype=torch.int64, device="cuda")
        self.t = (z(chains, W), z(chains), z(chains), z(chains))

    def launch(self, dev, tb, o, off, stream):
        _lib.check(_lib.load().anc_run_device(dev._h, tb._h, 11, off, len(self.t[1]), o, *(x.data_ptr() for x in self.t),
                                              None, stream.cuda_stream))

    def same(self, r):
        sp, sh, bs, fl = (x.cpu().numpy() for x in self.t)
        return (np.array_equal(sp.view(np.uint64), r.spins) and np.array_equal(sh, r.sum_sh) and
                np.array_equal(bs, r.sum_bs) and np.array_equal(fl, r.flips))


def _eager(out, *args):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        out.launch(*args, side)
    torch.cuda.synchronize()


def _capture(out, *args):
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        out.launch(*args, torch.cuda.current_stream())
    return g


@pytest.mark.parametrize("case", CASES)
def test_replay_after_a_larger_run(cuda, case):
    build, sched, engine, kind, few, many = CASES[case]
    inst = build()
    dev, tb = A.DeviceInstance(inst), A.Tables.from_schedule(A.Schedule(**sched))
    o = _lib.opts(engine, tensor_kind=kind)
    ref = A.run(dev, tb, 11, 40, few, engine=engine, tensor_kind=kind)
    out = _Out(inst.n, few)
    _eager(out, dev, tb, o, 40)
    g = _capture(out, dev, tb, o, 40)
    big = A.run(dev, tb, 11, 0, many, engine=engine, tensor_kind=kind)
    assert np.array_equal(big.spins[40:40 + few], ref.spins)
    fill = [torch.full((1 << 18,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]   # freed blocks find new owners
    for _ in range(2):
        for x in out.t:
            x.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert out.same(ref)
    assert all(int((f != -1).sum()) == 0 for f in fill)


@pytest.mark.parametrize("case", ["sparse groups", "planes", "streaming"])
@pytest.mark.parametrize("before", ["nothing", "fewer anneals"])
def test_capture_without_workspaces(cuda, case, before):
    build, sched, engine, kind, few, many = CASES[case]
    inst = build()
    tb = A.Tables.from_schedule(A.Schedule(**sched))
    o = _lib.opts(engine, tensor_kind=kind)
    ref = A.run(A.DeviceInstance(inst), tb, 11, 0, many)       # another handle: loads the kernels
    A.run(A.DeviceInstance(inst), tb, 11, 0, many, engine="plain")
    dev = A.DeviceInstance(inst)
    out = _Out(inst.n, many)
    if before == "fewer anneals":
        _eager(_Out(inst.n, 5), dev, tb, o, 0)
    g = _capture(out, dev, tb, o, 0)
    for _ in range(2):
        for x in out.t:
            x.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert out.same(ref)


def test_meanfield_replay_after_more_steps(cuda):
    """The relaxation's kernels of up to 3072 spins can be captured after an eager call; a longer call in between moves nothing."""
    import math
    from anechoic_b200.meanfield import CHECKPOINT, MeanField, SoftSchedule, initial_magnetisations
    mf, S = MeanField(I.complete_pm1(900, 4)), 20
    theta = torch.tensor([20.0, math.log(6.0), 3.0, 0.0, 1.05], dtype=torch.float64)
    sched = lambda S: torch.stack(list(SoftSchedule(S=S).vectors(theta))).detach().to("cuda", torch.float32).contiguous()
    s20, s300 = sched(S), sched(300)
    m0 = mf.pad(initial_magnetisations(900, 64, 1))
    g = mf.pad(torch.randn((64, 900), generator=torch.Generator().manual_seed(2)))
    prev = torch.ones_like(m0)
    want, ck = mf.forward_raw(s20, m0, prev)
    wg = mf.backward_raw(s20, ck, g)
    out, gs, ck2 = torch.empty_like(want), torch.empty_like(wg), torch.empty_like(ck)
    L = _lib.load()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(L.anc_mf_forward(mf._h, S, s20.data_ptr(), m0.data_ptr(), prev.data_ptr(), ck2.data_ptr(), out.data_ptr(), st))
        _lib.check(L.anc_mf_backward(mf._h, S, s20.data_ptr(), ck2.data_ptr(), g.data_ptr(), gs.data_ptr(), st))
    long_m, long_ck = mf.forward_raw(s300, m0, prev)
    mf.backward_raw(s300, long_ck, g)
    assert long_ck.shape[0] == math.ceil(300 / CHECKPOINT)
    fill = [torch.full((1 << 18,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]
    for _ in range(2):
        for x in (out, gs, ck2):
            x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(gs, wg) and torch.equal(ck2, ck)
    assert all(int((f != -1).sum()) == 0 for f in fill)
