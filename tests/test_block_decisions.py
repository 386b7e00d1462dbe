"""A case that fails while a kernel runs must not tear a block (or a warp)
apart: the kernels whose passes hold block barriers take an item by one
decision of the block, those that exchange values by shuffles by one of the
warp.  Read from the kernels' source, since what a torn block does is not to
be shown on a GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mahyco_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _functions(text, prefix):
    """name -> text of every function whose name starts with `prefix` (signature and body)."""
    out = {}
    for m in re.finditer(r"\b(%s\w+)\(" % prefix, text):
        depth, i = 0, m.end() - 1
        while i < len(text):  # the parameter list
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        body = re.match(r"\s*\{", text[i:])
        if not body:
            continue  # a call
        j = i + body.end()
        depth = 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        out[m.group(1)] = text[i:j]
    return out


def _text():
    return _source("mhc_kernels.cuh") + _source("mhc_sweep.cuh") + _source("mhc_launch.cuh")


def _kernels():
    """kernel -> (its text with that of the passes it calls, its own text)"""
    text = _text()
    passes = {**_functions(text, "body_"), **_functions(text, "delta_t_"), **_functions(text, "lane_")}
    # the lanes' exchanges of values are methods of their own
    passes = {k: v + (" __shfl_sync" if re.search(r"\b(CellLane|NodeLane)<", v) else "") for k, v in passes.items()}
    out = {}
    for name, own in _functions(text, "kb_").items():
        called = {f for f in re.findall(r"\b\w+", own) if f in passes}
        called |= {g for f in called for g in re.findall(r"\b\w+", passes[f]) if g in passes}
        out[name] = (own + "".join(passes[f] for f in called), own)
    return out


# threads that leave an item by their own reading of the case's state
ALONE = r"\bcase_active\(\w+\)\)\s*(continue|return)"
# the kernels that they may in, since nothing raises a flag while they run: the
# cell pass (below) and the cell sweeps, beside which only node sweeps run
QUIET = {"kb_lagrange_cells", "kb_sweep_cells_tile"}


def test_barriers_follow_a_decision_of_the_block():
    kernels = _kernels()
    barred = {k for k, (full, _) in kernels.items() if "__syncthreads" in full}
    assert {"kb_sweep_cells_tile", "kb_sweep_nodes_tile", "kb_delta_t", "kb_lagrange_cells"} <= barred
    for k in barred - QUIET:
        own = kernels[k][1]
        assert "block_active(" in own and not re.search(ALONE, own), k


def test_shuffles_follow_a_decision_of_the_warp_or_block():
    kernels = _kernels()
    shuffled = {k for k, (full, _) in kernels.items() if "__shfl" in full}
    assert {"kb_sweep_cells", "kb_sweep_nodes", "kb_sweep_nodes_tile"} <= shuffled
    for k in shuffled - QUIET:
        own = kernels[k][1]
        assert re.search(r"\b(warp|block)_active\(", own) and not re.search(ALONE, own), k


def test_cell_pass_raises_no_flag_before_its_time_step_ends():
    """With the time step in it (DT) the pass notes its negative volumes beside the block count."""
    body = _functions(_text(), "body_lagrange_")["body_lagrange_cells"]
    assert body.count("status") == 1
    assert re.search(r"if constexpr \(DT\)[^;]*dt_blocks[^;]*;\s*else atomicOr\(&F\.s->status", body)
    assert "body_lagrange_cells<DIM, NE, EULER, EL, CSTS, DT>" in _kernels()["kb_lagrange_cells"][1]


def test_sweeps_raise_no_flag():
    bodies = _functions(_text(), "body_sweep_")
    assert len(bodies) >= 5
    for k, body in bodies.items():
        assert "status" not in body, k
