"""What this framework is timed on: its annealing engines and the mean-field relaxation, each called the way a user's
program calls it (anechoic_b200.run, run_batch, and meanfield.relax under torch autograd), from one short anneal to
the benchmark's largest batches.

A case is a dict of plain values; "kind" names its family:

  dense    anneals of one dense instance (run, engine "auto"): K = 1 is a +-1 complete graph, K = 2 / 4 are iid
           couplings in [-1, 1] (half of them zero) / [-7, 7]
  sparse   anneals of one sparse instance (run): a toroidal grid or a uniform random graph
  batch    anneals of many sparse instances of uneven size in one launch (run_batch)
  relax    the differentiable relaxation, forward and adjoint (meanfield.relax + torch.autograd.grad)

The anneals' results are integers (bit-exact by contract), so exact() has values for the relaxation only.
"""
import math

import numpy as np
import torch

import anechoic_b200 as A
from anechoic_b200 import instances as I
from anechoic_b200 import meanfield as M

# Schedules: the reference's default with the counted Onsager correction (the headline benchmark), the
# temperature-scaled correction of its published headline, a cold start (few flips), the large-instance schedule whose
# start temperature follows the field's size, and the sparse instances' schedule. "flips" is the fraction of spins that
# flip per step, about, for the operation counts of work().
SCHEDULES = {
    "counted": (dict(t0=30.0, t1=5.0, q=4.0, lam=1.05, ramp=True), 0.33),
    "tecT": (dict(t0=15.0, t1=5.0, q=8.0, kappa=2.0, ramp=True), 0.11),
    "plain": (dict(t0=30.0, t1=5.0, q=4.0), 0.33),
    "cold": (dict(t0=4.0, t1=1.0, q=4.0, lam=1.05, ramp=True), 0.05),
    "large": (dict(t1=2.0, q=4.0, lam=1.05, ramp=True), 0.35),
    "sparse": (dict(t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True), 0.25),
}


def listed():
    return [
        # the smallest call: one short anneal of a small graph with its n_lin trace (the golden model's run_trial)
        dict(name="one small anneal", kind="dense", n=500, K=1, bias=False, sched="counted", S=100, chains=1, trace=True),
        # one anneal of the benchmark's instance: the reference's single-chain latency
        dict(name="one anneal", kind="dense", n=2000, K=1, bias=False, sched="counted", S=1000, chains=1, trace=False),
        # the reference's published headline: 120 short anneals with the temperature-scaled correction
        dict(name="tecT batch", kind="dense", n=2000, K=1, bias=False, sched="tecT", S=120, chains=120, trace=False),
        # the benchmark's headline batch
        dict(name="batch 1024", kind="dense", n=2000, K=1, bias=False, sched="counted", S=1000, chains=1024, trace=False),
        # multi-bit couplings with bias at the headline's size: a batch of replicas
        dict(name="k4 bias batch", kind="dense", n=2000, K=4, bias=True, sched="large", S=500, chains=256, trace=False),
        # ternary couplings at an odd size above the reference's 2048, without a correction
        dict(name="k2 ragged batch", kind="dense", n=2501, K=2, bias=False, sched="plain", S=300, chains=100, trace=False),
        # a larger complete graph
        dict(name="pm1 n 5000", kind="dense", n=5000, K=1, bias=False, sched="counted", S=200, chains=128, trace=False),
        # the large dense stress: 4-bit couplings with bias, 256 anneals, J too large to stay on chip
        dict(name="large k4 bias", kind="dense", n=10000, K=4, bias=True, sched="large", S=200, chains=256, trace=False),
        # a few anneals of the largest sparse class (toroidal grid, 20000 vertices)
        dict(name="torus 20000", kind="sparse", n=20000, degree=4, signed=True, S=300, chains=16, trace=False),
        # the 51 uneven sparse instances of the benchmark, 64 anneals each, in one launch
        dict(name="51 instances", kind="batch", count=51, S=1000, chains=64, trace=False),
        # schedule tuning's inner step: 64 replicas, 200 unrolled steps, forward and adjoint
        dict(name="relax 200", kind="relax", n=2000, R=64, S=200, mode="counted", bias=False),
        # a short relaxation of a small biased instance, few replicas
        dict(name="relax 37 small", kind="relax", n=700, R=16, S=37, mode="tecT", bias=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["dense", "sparse", "batch", "relax"], weights=[5, 2, 2, 3])[0]
    if kind == "relax":
        return dict(kind=kind, n=_log(rng, 300, 4000), R=rng.choice([1, 8, 16, 33, 64]), S=_log(rng, 16, 200),
                    mode=rng.choice(["counted", "tecT", "none"]), bias=rng.random() < 0.5)
    if kind == "sparse":
        return dict(kind=kind, n=_log(rng, 800, 20000), degree=rng.choice([4, 6, 12, 20, 48]), signed=rng.random() < 0.5,
                    S=_log(rng, 50, 500), chains=_log(rng, 1, 300), trace=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(4, 51), S=_log(rng, 50, 600), chains=_log(rng, 4, 64),
                    trace=rng.random() < 0.3)
    n = _log(rng, 200, 10000)
    K = rng.choice([1, 1, 2, 4])
    chains, S = _log(rng, 1, 1024), _log(rng, 50, 1000)
    # no drawn case costs more than the largest listed ones: 148 anneals advance at once on the slowest path, and a
    # step of theirs costs about n^2 times the bits of a coupling
    room = 3.0e10 / (max(n, 2000) ** 2 * K)
    while S * -(-chains // 148) > room and (S > 20 or chains > 1):
        S, chains = max(20, S // 2), max(1, chains * 3 // 4)
    sched = "large" if K == 4 else rng.choice(["counted", "counted", "tecT", "plain", "cold"])
    return dict(kind=kind, n=n, K=K, bias=K > 1 and rng.random() < 0.5, sched=sched, S=S, chains=chains,
                trace=rng.random() < 0.3)


# ---------------------------------------------------------------------------------------------------------- inputs
def _bias(n, rng, top):
    return rng.integers(-top, top + 1, size=n).astype(np.int32)


def _dense(n, K, seed, bias):
    """Symmetric couplings, zero diagonal: +-1 (K = 1), -1, 0, 0, 1 (K = 2), [-7, 7] (K = 4)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(dev).manual_seed(seed)
    r = torch.randint(0, 4 if K < 4 else 15, (n, n), generator=g, dtype=torch.int8, device=dev)
    J = (r & 1) * 2 - 1 if K == 1 else (r & 1) - (r >> 1) if K == 2 else r - 7
    J = torch.triu(J, 1)
    J = (J + J.T).cpu().numpy()
    return A.Instance(n=n, dense=J, bias=_bias(n, np.random.default_rng(seed), 7 if K == 4 else 2) if bias else None)


def _sparse(case, seed):
    n, d = case["n"], case["degree"]
    if d == 4:
        side = max(3, math.isqrt(n // 2))
        return I.torus(side, max(3, n // side), seed, signed=case["signed"], bmax=2)
    return I.random_graph(n, min(n * d // 2, n * (n - 1) // 2), case["signed"], seed, bmax=2)


def _schedule(case):
    sched = "sparse" if case["kind"] in ("sparse", "batch") else case["sched"]
    f = dict(SCHEDULES[sched][0])
    if sched == "large":
        f["t0"] = 8.0 * math.sqrt(case["n"])
    return A.Tables.from_schedule(A.Schedule(S=case["S"], **f))


def _relax_inputs(case, seed):
    inst = _dense(case["n"], 1 if not case["bias"] else 2, seed, case["bias"])
    n, R, S = case["n"], case["R"], case["S"]
    # the reference's default schedule, its temperatures scaled to the size of this instance's fields
    scale = math.sqrt(n / 2000.0) * (1.0 if not case["bias"] else math.sqrt(0.5))
    gain = 0.1 if case["mode"] == "tecT" else 1.05
    theta = torch.tensor([30.0 * scale, math.log(6.0), 4.0 * scale, 0.0, gain], dtype=torch.float64)
    vectors = [v.detach().clone() for v in M.SoftSchedule(S=S, mode=case["mode"]).vectors(theta)]
    m0 = M.initial_magnetisations(n, R, seed)
    g = torch.randn((R, n), generator=torch.Generator().manual_seed(seed + 1), dtype=torch.float32) / n
    return inst, vectors, m0, g


def prepare(case, seed):
    state = dict(case=case, seed=seed)
    if case["kind"] == "relax":
        inst, vectors, m0, g = _relax_inputs(case, seed)
        mf = M.MeanField(inst)
        state.update(mf=mf, vectors=[v.cuda().requires_grad_() for v in vectors], m0=mf.pad(m0), g=mf.pad(g))
        return state
    if case["kind"] == "batch":
        instances = [build() for _, build in _spread(I.sparse_classes_manifest(seed), case["count"])]
    elif case["kind"] == "sparse":
        instances = [_sparse(case, seed)]
    else:
        instances = [_dense(case["n"], case["K"], seed, case["bias"])]
    state.update(devices=[A.DeviceInstance(i) for i in instances], tables=_schedule(case))
    return state


def _spread(items, count):
    """count of the items, evenly over the list (its classes follow one another)."""
    return [items[k * len(items) // count] for k in range(count)]


# ------------------------------------------------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    if case["kind"] == "relax":
        mS = M.relax(state["mf"], *state["vectors"], state["m0"])
        grads = torch.autograd.grad(mS, state["vectors"], state["g"])
        return dict(m=mS.detach(), grads=list(grads))
    if case["kind"] == "batch":
        out = A.run_batch([dict(dev=d, tb=state["tables"], seed=state["seed"], trial_offset=64 * k,
                                nchains=case["chains"], trace=case["trace"]) for k, d in enumerate(state["devices"])])
        return [np.concatenate([x.reshape(-1) for x in xs]) for xs in zip(*(_results(r) for r in out))]
    return _results(A.run(state["devices"][0], state["tables"], state["seed"], 0, case["chains"], trace=case["trace"]))


def _results(r):
    out = [r.spins.view(np.int64), r.sum_sh, r.sum_bs, r.flips]
    return out if r.trace is None else out + [r.trace]


# ------------------------------------------------------------------------------------------------------------ work
def _dense_work(n, K, phi, S, chains, trace):
    """Every flip changes n fields by one coupling each (two operations), every spin is decided once a step (about
    ten); the couplings are read once, the results written once."""
    flops = float(chains) * S * (2.0 * phi * n * n + 10.0 * n)
    nbytes = K * n * n / 8.0 + chains * (n / 8.0 + 24.0 + (4.0 * S if trace else 0.0))
    return nbytes, flops


def _sparse_work(n, nnz, phi, S, chains, trace):
    flops = float(chains) * S * (2.0 * phi * nnz + 10.0 * n)
    nbytes = 4.0 * nnz + 4.0 * n + chains * (n / 8.0 + 24.0 + (4.0 * S if trace else 0.0))
    return nbytes, flops


def work(case):
    if case["kind"] == "relax":
        n, R, S = case["n"], case["R"], case["S"]
        # J m in every forward step, J p in every adjoint step; J as 2-byte words, m_0 and g in, m_S and the gradients out
        return dict(bytes=2.0 * n * n + 4.0 * (3 * R * n + 8 * S), flops=4.0 * n * n * R * S)
    if case["kind"] == "dense":
        b, f = _dense_work(case["n"], case["K"], SCHEDULES[case["sched"]][1], case["S"], case["chains"], case["trace"])
        return dict(bytes=b, flops=f)
    phi = SCHEDULES["sparse"][1]
    if case["kind"] == "sparse":
        b, f = _sparse_work(case["n"], case["n"] * case["degree"], phi, case["S"], case["chains"], case["trace"])
        return dict(bytes=b, flops=f)
    # the batch's classes: about 2000 vertices of degree 20 on the whole
    b, f = _sparse_work(2000, 2000 * 20, phi, case["S"], case["chains"], case["trace"])
    return dict(bytes=case["count"] * b, flops=case["count"] * f)


# ----------------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    """The relaxation in float64 on the float32 inputs the kernels take: m_S and its derivatives by torch autograd."""
    if case["kind"] != "relax":
        return None
    inst, vectors, m0, g = _relax_inputs(case, seed)
    n, R, S = case["n"], case["R"], case["S"]
    npad = -(-n // 256) * 256
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    J = torch.as_tensor(inst.dense, device=dev).double()
    b = torch.zeros(n, device=dev, dtype=torch.float64)
    if inst.bias is not None:
        b += torch.as_tensor(inst.bias, device=dev).double()
    beta, q, u, w = (v.float().double().to(dev).requires_grad_() for v in vectors)
    # the padded replica rows start at zero magnetisation and belong to the result: all 64 rows are computed
    m = torch.zeros((64, n), device=dev, dtype=torch.float64)
    m[:R] = m0.to(dev).double()
    prev = torch.ones_like(m)
    for t in range(S):
        gamma = u[t] * (1.0 - m * m).sum(dim=1, keepdim=True) + w[t]
        m, prev = torch.tanh(beta[t] * (m @ J + b + q[t] * m - gamma * prev)), m
    gm = torch.zeros_like(m)
    gm[:R] = g.to(dev).double()
    grads = torch.autograd.grad(m, (beta, q, u, w), gm, allow_unused=True)
    grads = [torch.zeros(S, device=dev, dtype=torch.float64) if x is None else x for x in grads]
    out = torch.zeros((64, npad), device=dev, dtype=torch.float64)
    out[:, :n] = m.detach()
    return dict(m=out, grads=grads)
