"""MAP and sampling of nodes with many children: a gather of more than 16 rakes
in a grid-wide round has a block of its own, in a tail its block forms the
messages a rake per group and, above 32 rakes, the sums together
(csrc/phase_log.cuh). The states and log weights of the per-tree engines, bit
for bit, on both sides of these fan-ins, and not slower than those engines."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


def broom(children, leaves):
    """A root with `children` children of `leaves` leaves each: the children's
    gathers of one round all have that fan-in."""
    inner = np.repeat(np.arange(1, children + 1), leaves)
    return np.concatenate([[-1], np.zeros(children, np.int64), inner])


def outputs(ws, model, uniforms):
    view = ws.maximum_a_posteriori_prepared(model)
    out = [np.array(view.log_weights), np.array(view.states)]
    return out + [np.array(ws.posterior_sample_prepared(model, uniforms).states)]


def check(ws, model, uniforms):
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    got = outputs(ws, model, uniforms)
    launches = ws.launches
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs(ws, model, uniforms)):
        assert np.array_equal(a, b)
    return launches


# Children enough for the round to run grid-wide (csrc/runtime.cc, SetLogRounds).
@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states,children", [(3, 700), (4, 700), (8, 90), (13, 45), (20, 40)])
def test_grid_wide_rounds(gpu, states, children, scalar):
    rng = np.random.default_rng(states)
    shapes = [broom(children, n) for n in (1, 15, 16, 17, 33)] + [broom(2, 700)]
    plans = gpu.Plan.many(shapes)
    nodes = sum(p.num_nodes for p in plans)
    edges = sum(p.num_edges for p in plans)
    ws = gpu.Workspace()
    ws.reserve_forest(plans, states, kind="maximum,sampling", scalar=scalar)
    launches = check(ws, gpu.BatchedModelView(
        None, states, len(plans), (rng.random(nodes * states) + 0.05).astype(scalar),
        (rng.random(edges * states ** 2) + 0.01).astype(scalar)), rng.random(nodes).astype(scalar))
    assert launches >= 4  # a gather, the wide gathers, the tail, the rakes' states


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states,items", [(4, 3), (8, 1), (20, 2)])
@pytest.mark.parametrize("leaves", [31, 32, 33, 64, 65, 1000])
def test_tails(gpu, states, items, leaves, scalar):
    rng = np.random.default_rng(states + leaves)
    plan = gpu.Plan(broom(3, leaves))
    ws = gpu.Workspace()
    ws._reserve("maximum,sampling", plan, states, items, 0, scalar, None)
    check(ws, gpu.BatchedModelView(
        plan, states, items, (rng.random(items * plan.num_nodes * states) + 0.05).astype(scalar),
        (rng.random(plan.num_edges * states ** 2) + 0.01).astype(scalar)),
        rng.random(items * plan.num_nodes).astype(scalar))


@pytest.mark.parametrize("shape", [broom(1, 5000), broom(100, 50)], ids=["star", "brooms"])
def test_time(gpu, shape):
    """Ten times and more the per-tree engines' while one group took a gather's
    rakes one after the other."""
    plan = gpu.Plan(shape)
    ws = gpu.Workspace()
    ws.reserve_maximum(plan, 8, 1, scalar=np.float32)
    rng = np.random.default_rng(1)
    model = gpu.BatchedModelView(plan, 8, 1,
                                 (rng.random(plan.num_nodes * 8) + 0.05).astype(np.float32),
                                 (rng.random(plan.num_edges * 64) + 0.01).astype(np.float32))

    def kernel_ms():
        return min(ws.maximum_a_posteriori_prepared(model).timings.kernel_ms for _ in range(5))

    phases = kernel_ms()
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    assert phases <= 1.5 * kernel_ms()
