"""A small case's cell sweeps split their variables between up to three blocks
an item; a batch's blocks take them all.  The same case alone and in a batch
of two gives the same fields bit for bit, on meshes on both sides of the sizes
where three, two and one blocks an item fit a B200 at once, for one, two and
three environments, in 2D and 3D."""
import numpy as np
import pytest

from mahyco_b200.case import MINMOD, SUPERBEE, VANLEER
from mahyco_b200.cases import sod, triple_point, two_state

FIELDS = ("Density", "Pressure", "InternalEnergy", "PseudoViscosity", "Velocity", "NodeMass")


def _two(n, env, limiter):
    return two_state(dim=2, n=n, L=(0.01 * n[0], 0.01 * n[1]), interface=0.004 * n[0], nb_env=env, limiter=limiter,
                     deltat_init=1e-3)


CASES = {
    "one_env_tiny": lambda: _two((7, 5), 1, MINMOD),
    "one_env_211x201": lambda: _two((211, 201), 1, SUPERBEE),
    "two_env_213x201": lambda: _two((213, 201), 2, VANLEER),
    "two_env_319x200": lambda: _two((319, 200), 2, MINMOD),
    "two_env_321x200": lambda: _two((321, 200), 2, SUPERBEE),
    "three_env_130x61": lambda: triple_point(n=(130, 61, 1), limiter=MINMOD, deltat_init=1e-5),
    "two_env_3d_41x33x29": lambda: sod(dim=3, n=(41, 33, 29), L=(1.0, 0.8, 0.7), limiter=VANLEER, deltat_init=2e-3),
    "two_env_3d_51x37x35": lambda: sod(dim=3, n=(51, 37, 35), L=(1.0, 0.8, 0.7), limiter=SUPERBEE, deltat_init=2e-3),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_split_variables_change_nothing(name):
    from mahyco_b200 import Batch, Hydro
    h = Hydro(CASES[name]())
    h.hydroStartInit()
    h.cycle(9)
    assert h.synchronize() == 0
    with Batch() as b:
        idx = [b.add(CASES[name]()) for _ in range(2)]
        b.init()
        b.cycle(9)
        for f in FIELDS:
            want = h.field(f)
            for i in idx:
                assert np.array_equal(b.field(i, f), want), f
    h.close()
