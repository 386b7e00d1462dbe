"""A case that starts again (HydroStartInit) replays the CUDA graph of its
first run when nothing about its launches changed, and captures a new one when
something did: the fields and scalars of every run equal those of a fresh
case, bit for bit, in 2D, 3D and Lagrangian runs, with the grid or the sweep
layout changed between runs, after a checkpoint at an iteration that is not a
multiple of the sweep rotation, and for run lengths around the graph's own."""
import numpy as np
import pytest

from mahyco_b200.cases import sod, two_state

FIELDS = ("Density", "Pressure", "InternalEnergy", "Velocity", "NodeMass")
CASES = {
    "remap2d": lambda: two_state(dim=2, n=(31, 18), left=(1.7, 1.3), right=(0.2, 0.07), deltat_init=1e-3),
    "remap3d": lambda: sod(dim=3, n=(17, 6, 5), L=(1.0, 0.3, 0.25), deltat_init=1e-3),
    "lagrange": lambda: sod(dim=2, n=(31, 5), L=(1.0, 0.15), remap=False, deltat_init=1e-3),
}


def _out(h):
    h.synchronize()
    return h.scalars(), [h.field(f) for f in FIELDS]


def _fresh(p, n):
    from mahyco_b200 import Hydro
    h = Hydro(p)
    h.hydroStartInit()
    h.cycle(n)
    out = _out(h)
    h.close()
    return out


def _same(a, b):
    return a[0] == b[0] and all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_restart_keeps_or_renews_the_graph(name):
    from mahyco_b200 import Hydro
    p = CASES[name]()
    h = Hydro(p)
    for n in (6, 13, 1, 2, 3, 7, 12):
        h.hydroStartInit()
        h.cycle(n, graph=True)
        assert _same(_out(h), _fresh(p, n)), n
    want = _fresh(p, 14)
    for change in (lambda: h.set_stage_grid_scale("lagrange_nodes", 1), lambda: h.set_sweep_layout(1, 1),
                   lambda: h.set_sweep_layout(3, 3), lambda: h.set_grid_scale(0), lambda: h.set_sweep_layout(0, 0)):
        h.hydroStartInit()
        h.cycle(6, graph=True)
        change()
        h.hydroStartInit()
        h.cycle(14, graph=True)
        assert _same(_out(h), want)
    h.hydroStartInit()
    h.cycle(5, graph=True)
    saved = h.checkpoint()
    h.cycle(9, graph=True)
    assert _same(_out(h), want)
    h.restore(saved)
    h.cycle(9, graph=True)
    assert _same(_out(h), want)
    h.hydroStartInit()
    h.cycle(14, graph=True)
    assert _same(_out(h), want)
    h.close()
