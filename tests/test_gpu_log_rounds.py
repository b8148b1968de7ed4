"""Which rounds of MAP and sampling run grid-wide (csrc/runtime.cc, SetLogRounds
and LogTail): a large tree among many small ones keeps its own rounds, and trees
that fill the chip more than once have no tail. The per-tree engines' bits
either way."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


def outputs(ws, model, uniforms):
    view = ws.maximum_a_posteriori_prepared(model)
    out = [np.array(view.log_weights), np.array(view.states)]
    return out + [np.array(ws.posterior_sample_prepared(model, uniforms).states)]


def check(ws, model, uniforms):
    """The number of launches of the sampling call."""
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    got = outputs(ws, model, uniforms)
    launches = ws.launches
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES, stripes=2)
    for a, b in zip(got, outputs(ws, model, uniforms)):
        assert np.array_equal(a, b)
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs(ws, model, uniforms)):
        assert np.array_equal(a, b)
    return launches


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states,large,small", [(4, 30000, 100), (8, 5000, 300), (8, 5000, 1500),
                                                (20, 2000, 400)])
def test_one_large_tree_among_small_ones(gpu, states, large, small, scalar):
    rng = np.random.default_rng(states + small)
    plans = gpu.Plan.many([synthetic.random_recursive(rng, n)
                           for n in [7] * (small // 2) + [large] + [7] * (small // 2)])
    nodes = sum(p.num_nodes for p in plans)
    edges = sum(p.num_edges for p in plans)
    ws = gpu.Workspace()
    ws.reserve_forest(plans, states, kind="maximum,sampling", scalar=scalar)
    launches = check(ws, gpu.BatchedModelView(
        None, states, len(plans), (rng.random(nodes * states) + 0.05).astype(scalar),
        (rng.random(edges * states ** 2) + 0.01).astype(scalar)), rng.random(nodes).astype(scalar))
    # Two rounds at least: gathers and compressions, the tail or the roots, and
    # their states.
    assert launches >= 9


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states", [1, 4, 8, 20])
def test_items_beyond_the_chip(gpu, states, scalar):
    rng = np.random.default_rng(states)
    plan = gpu.Plan(synthetic.random_recursive(rng, 15))
    capacity = 3000  # more tail blocks than any kernel has on the chip
    ws = gpu.Workspace()
    ws._reserve("maximum,sampling", plan, states, capacity, 0, scalar, None)
    edges = (rng.random(plan.num_edges * states ** 2) + 0.01).astype(scalar)
    for items, tail in ((capacity, False), (30, True)):
        nodes = items * plan.num_nodes
        launches = check(ws, gpu.BatchedModelView(
            plan, states, items, (rng.random(nodes * states) + 0.05).astype(scalar), edges),
            rng.random(nodes).astype(scalar))
        assert (launches == 1) == tail
        ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES)
