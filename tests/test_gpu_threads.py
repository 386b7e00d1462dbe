"""Two and more host threads, each with its own case (or batch), at the same
time in one process: the fields of the same runs one after another, bit for
bit.  The threads go first, so that they meet what the process makes on first
use (kernel figures, pinned buffers, graphs) together."""
import threading

import numpy as np
import pytest

from mahyco_b200.cases import MINMOD, SUPERBEE, VANLEER, bar_impact, sedov, seeded_two_state, sod

FIELDS = ("Density", "Pressure", "InternalEnergy", "Velocity", "NodeMass")


def _sod(n, remap=True, **kw):
    return sod(**dict(dict(dim=len(n), n=n, L=tuple(0.01 * m for m in n), bi=remap, remap=remap, deltat_init=1e-3), **kw))


# case, graph replay or launches
RUNS = [
    (lambda: _sod((65, 33, 17), limiter=SUPERBEE), True),
    (lambda: _sod((211, 57), limiter=VANLEER), False),
    (lambda: _sod((43, 21), remap=False), True),
    (lambda: sedov(dim=2, n=(60, 60), deltat_init=1e-4), False),
    (lambda: bar_impact(n=(20, 60), L=(0.01, 0.03)), True),
    (lambda: _sod((31, 29, 27), limiter=MINMOD), False),
]


def _solo(make, graph):
    from mahyco_b200 import Hydro
    with Hydro(make()) as h:
        h.hydroStartInit()
        for n in (3, 8, 5):
            h.cycle(n, graph=graph)
        assert h.synchronize() == 0
        return {f: h.field(f) for f in FIELDS}, h.scalars()


def _batch(seed):
    from mahyco_b200 import Batch
    with Batch() as b:
        idx = [b.add(seeded_two_state(seed + q, 40 + 7 * q)) for q in range(4)]
        b.init()
        b.cycle(12, graph=seed % 2 == 0)
        return [(b.field(i, "Density"), b.scalars(i)) for i in idx]


@pytest.mark.gpu
def test_threads_with_their_own_cases():
    jobs = [lambda r=r: _solo(*r) for r in RUNS] + [lambda s=s: _batch(s) for s in (10, 21)]
    repeats = 4
    got, errors = [[] for _ in jobs], []
    start = threading.Barrier(len(jobs))

    def work(q):
        try:
            start.wait(60)
            for _ in range(repeats):
                got[q].append(jobs[q]())
        except Exception as e:  # reported below, in the test's own thread
            errors.append((q, repr(e)))

    threads = [threading.Thread(target=work, args=(q,), daemon=True) for q in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    assert not errors and not any(t.is_alive() for t in threads), errors
    for q, (make, graph) in enumerate(RUNS):
        fields, scalars = _solo(make, graph)
        for f, s in got[q]:
            assert s == scalars, q
            for k in FIELDS:
                assert np.array_equal(f[k], fields[k]), (q, k)
    for q, seed in enumerate((10, 21)):
        want = _batch(seed)
        for run in got[len(RUNS) + q]:
            for (f, s), (fw, sw) in zip(run, want):
                assert s == sw and np.array_equal(f, fw), (seed, s, sw)
