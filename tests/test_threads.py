"""GPU: calls from several threads, each on handles of its own. The kernels' attributes and the device are shared, the results are
those of the same calls one after another."""
import threading

import numpy as np
import pytest

import anechoic_b200 as A
from anechoic_b200 import instances as I

pytestmark = pytest.mark.gpu

COUNTED = dict(S=20, lam=1.05, ramp=True)
SPARSE = dict(S=20, t0=6.0, t1=0.5, q=1.5, kappa=2.0, ramp=True)
# sizes whose launches of one kernel differ in their shared memory, and kernels whose CTAs wait for one another
CASES = [(lambda: I.complete_pm1(2000, 1), COUNTED, 256), (lambda: I.complete_pm1(500, 3), COUNTED, 1),
         (lambda: I.complete_pm1(2501, 2), COUNTED, 60), (lambda: I.random_kbit(5000, 2, 4, pzero=0.5), COUNTED, 3),
         (lambda: I.random_graph(1500, 15000, True, 4, bmax=2), SPARSE, 1200), (lambda: I.random_graph(3900, 15000, True, 5), SPARSE, 60),
         (lambda: I.torus(30, 30, 3), SPARSE, 60), (lambda: I.torus(60, 70, 3), SPARSE, 500), (lambda: I.torus(20, 30, 3), SPARSE, 500)]


def _handles():
    return [(A.DeviceInstance(build()), A.Tables.from_schedule(A.Schedule(**sc)), c) for build, sc, c in CASES]


def _run(h):
    r = A.run(h[0], h[1], 7, 3, h[2])
    return r.spins, r.flips, r.sum_sh


def test_threads_on_their_own_handles(cuda):
    want = [_run(h) for h in _handles()]
    bad = []

    def work(k):
        try:
            handles = _handles()
            for i in np.random.default_rng(k).integers(0, len(CASES), 300):
                if not all(np.array_equal(a, b) for a, b in zip(_run(handles[i]), want[i])):
                    bad.append((k, int(i)))
        except Exception as e:      # noqa: BLE001 -- reported by the main thread
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:5]
