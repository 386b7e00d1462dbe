"""The end of an iteration -- time step, stop test, error flags -- is the same
through the entry points one by one (the time step in a pass of its own),
whole iterations (a Lagrangian case's in its cell pass), their CUDA graph,
and a batch of two cases (the minimum, then the scalars): status, iteration
count, time, time step and fields, bit for bit.  Meshes of one block, of a
block more and a block less one cell, and of many blocks; runs that reach
their final time, underflow their time step, meet a NaN or a negative
volume."""
import numpy as np
import pytest

from mahyco_b200.cases import bar_impact, sod

FIELDS = ("Density", "Pressure", "InternalEnergy", "SoundSpeed", "CellVolume", "Velocity")


def _sod(n, remap, **kw):
    opts = dict(dim=len(n), n=n, L=tuple(0.01 * m for m in n), bi=False, remap=remap, deltat_init=1e-3)
    opts.update(kw)
    return sod(**opts)


def _nan(p):
    p.env[0].pression_initiale = -1.0  # the sound speed of the first time step is a NaN
    return p


def _underflow(p):
    p.deltat_min = 1.01e-3  # the first steps grow past it, the shock's bound falls below
    p.deltat_init = 1.1e-3
    p.deltat_max = 1.0e-3
    return p


CASES = {
    "lag_one_block": lambda: _sod((16, 8), False),
    "lag_block_less_one": lambda: _sod((127, 1), False),
    "lag_block_and_one": lambda: _sod((43, 3), False),
    "lag_3d": lambda: _sod((33, 7, 5), False),
    "lag_many_blocks": lambda: _sod((400, 120), False),
    "lag_elasto": lambda: bar_impact(n=(9, 31), L=(0.01, 0.03)),
    "lag_final_time": lambda: _sod((43, 3), False, final_time=6.5e-3),
    "lag_underflow": lambda: _underflow(_sod((43, 3), False)),
    "lag_nan": lambda: _nan(_sod((43, 3), False)),
    "lag_negative_volume": lambda: _sod((43, 3), False, deltat_init=0.2),
    "remap_one_block": lambda: _sod((16, 8), True),
    "remap_block_and_one": lambda: _sod((43, 3), True),
    "remap_3d": lambda: _sod((33, 7, 5), True),
    "remap_final_time": lambda: _sod((43, 3), True, final_time=6.5e-3),
    "remap_nan": lambda: _nan(_sod((43, 3), True)),
    "remap_many_blocks": lambda: _sod((700, 600), True),
}


def _state(p, how, n=12):
    from mahyco_b200 import Hydro
    h = Hydro(p)
    h.hydroStartInit()
    if how == "entry points":
        for _ in range(n):
            h.iterate()
    else:
        h.cycle(n, graph=how == "graph")
    h.synchronize()
    out = h.scalars(), {f: h.field(f) for f in FIELDS}
    h.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_step_end(name):
    from mahyco_b200 import Batch
    p = CASES[name]()
    want, fields = _state(p, "entry points")
    for how in ("cycle", "graph"):
        got, f = _state(p, how)
        assert got == want or (str(got) == str(want)), (how, got, want)
        for k in FIELDS:
            assert np.array_equal(f[k], fields[k], equal_nan=True), (how, k)
    with Batch() as b:
        idx = [b.add(CASES[name]()) for _ in range(2)]
        b.init()
        b.cycle(12)
        for i in idx:
            got = b.scalars(i)
            assert str(got) == str(want), (got, want)
            for k in FIELDS:
                assert np.array_equal(b.field(i, k), fields[k], equal_nan=True), k
