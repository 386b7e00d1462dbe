"""Cases of a batch that fail in the middle of an iteration leave the others
alone, with persistent grids too: blocks that go on from an item of a failing
case to one of a healthy case.  The failing cases meet a NaN in the first
iterations (the finalize pass of the cells raises it beside the node sweeps,
or the time step does), set up on the host: a negative initial pressure has
no sound speed.  The healthy cases equal their solo runs bit for bit."""
import numpy as np
import pytest

from mahyco_b200.cases import SUPERBEE, VANLEER, bar_impact, seeded_two_state, sod

FIELDS = ("Density", "Pressure", "InternalEnergy", "SoundSpeed", "CellMass", "Velocity", "NodeMass")


def _bisod(n, **kw):
    return sod(**dict(dict(dim=3, n=n, L=tuple(0.01 * m for m in n), bi=True, limiter=SUPERBEE, deltat_init=1e-3), **kw))


def _sod2d(n, limiter=VANLEER):
    return sod(dim=2, n=n, L=tuple(0.01 * m for m in n), bi=True, limiter=limiter, deltat_init=1e-3)


def _failing(p, env=0):
    p.env[env].pression_initiale = -1.0
    return p


MIXES = {
    # more items than resident blocks, of several cases each
    "3d": lambda: [(_bisod((96, 40, 33)), True), (_failing(_bisod((96, 40, 33))), False),
                   (_bisod((64, 33, 50)), True), (_failing(_bisod((80, 48, 31)), 1), False),
                   (_bisod((50, 60, 40)), True)],
    "2d": lambda: [(_sod2d((301, 257)), True), (_failing(_sod2d((300, 255))), False), (_sod2d((97, 411)), True),
                   (_failing(_sod2d((128, 300)), 1), False), (seeded_two_state(7, 150), True)],
    "lagrangian": lambda: [(sod(dim=2, n=(200, 100), L=(2., 1.), bi=False, remap=False, deltat_init=1e-3), True),
                           (_failing(sod(dim=2, n=(200, 100), L=(2., 1.), bi=False, remap=False, deltat_init=1e-3)), False),
                           (sod(dim=2, n=(150, 90), L=(2., 1.), bi=False, remap=False, deltat_init=1e-3), True)],
}


def _solo(p, n):
    from mahyco_b200 import Hydro
    with Hydro(p) as h:
        h.hydroStartInit()
        h.cycle(n)
        assert h.synchronize() == 0
        return {f: h.field(f) for f in FIELDS}


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0, 1])
@pytest.mark.parametrize("mix", MIXES)
def test_failing_cases_leave_neighbours_intact(mix, scale):
    from mahyco_b200 import Batch
    n = 8
    cases = MIXES[mix]()
    want = [_solo(p, n) if good else None for p, good in cases]
    for _ in range(3):
        with Batch() as b:
            b.set_grid_scale(scale)
            idx = [b.add(p) for p, _ in cases]
            b.init()
            b.cycle(n)
            for i, (p, good), ref in zip(idx, cases, want):
                s = b.scalars(i)
                if not good:
                    assert s["status"] != 0 and s["iteration"] < n, s
                    continue
                assert s["status"] == 0 and s["iteration"] == n, s
                for f in FIELDS:
                    assert np.array_equal(b.field(i, f), ref[f]), (i, f)


@pytest.mark.gpu
@pytest.mark.parametrize("n,deltat", [((16, 8), 1e-4), ((9, 31), 1e-5), ((80, 40), 1e-5)])
def test_negative_volume_of_the_cell_pass_is_the_status(n, deltat):
    """An elasto-plastic case whose first time step turns cells over: the same
    status, iteration and time through the entry points (the geometry raises
    the flag) and whole iterations (the last block of the pass does), at one
    block and several, and again after a restart."""
    from mahyco_b200 import Hydro, ST_NEG_VOLUME
    for how in ("entry points", "cycle", "graph"):
        with Hydro(bar_impact(n=n, L=(0.01, 0.03), deltat_init=deltat)) as h:
            for _ in range(2):
                h.hydroStartInit()
                if how == "entry points":
                    for _ in range(4):
                        h.iterate()
                else:
                    h.cycle(4, graph=how == "graph")
                s = h.scalars()
                assert s["status"] == ST_NEG_VOLUME and s["iteration"] == 0, (how, s)
