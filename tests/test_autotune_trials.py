"""What the tuner tries: each kernel layout once (3 launches the kernels of 2,
so it is no trial of its own), every grid scale once; a cached decision that
still names layout 3 is installed as it is.  A stand-in for the case, no GPU."""
import json
import os

from mahyco_b200 import autotune
from mahyco_b200.cases import sod


class Target:
    def __init__(self):
        self.layouts, self.scales, self.stages, self.trials, self.cycles = [], [], {}, 0, 0

    def set_sweep_layout(self, cells, nodes):
        self.layouts.append((cells, nodes))

    def set_grid_scale(self, scale):
        self.scales.append(scale)

    def set_stage_grid_scale(self, stage, scale):
        self.stages[stage] = scale

    def cycle_timed(self, n):
        self.trials += 1
        self.cycles += n
        return {s: (float(self.trials), 1) for s in ("sweep_cells", "sweep_nodes", "delta_t")}


def test_each_layout_and_scale_is_tried_once():
    t = Target()
    d = autotune.tune(t, cycles_per_trial=1)
    assert t.layouts == [(1, 1), (2, 2), (1, 1)]  # the trials, then the fastest
    assert t.scales == list(autotune.CANDIDATES) + [0]
    assert t.trials == 2 + len(autotune.CANDIDATES)
    assert (d["cell_layout"], d["node_layout"]) == (1, 1)


def test_cached_layout_3_is_installed(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("MHC_TUNE_CACHE", str(path))
    p = sod(dim=2, n=(20, 10), L=(1.0, 0.5), bi=True, deltat_init=1e-3)
    path.write_text(json.dumps({autotune.bucket(p): {"cell_layout": 3, "node_layout": 2, "grid": {"delta_t": 4}}}))
    t = Target()
    d = autotune.tune(t, params_list=p)
    assert d["cached"] and t.trials == 0 and t.layouts == [(3, 2)] and t.stages == {"delta_t": 4}


def test_trial_cycles_are_what_a_tuning_runs():
    """Callers that compare a tuned run with another one count them (bench.py)."""
    for n, candidates in ((1, autotune.CANDIDATES), (2, autotune.CANDIDATES), (3, (0, 2))):
        t = Target()
        autotune.tune(t, cycles_per_trial=n, candidates=candidates)
        assert t.cycles == autotune.trial_cycles(n, candidates)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with open(os.path.join(root, "bench.py")) as f:
        text = f.read()
    assert "tune_cycles = trial_cycles(2)" in text and "len(CANDIDATES)" not in text
