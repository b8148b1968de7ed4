"""MAP and sampling tails of one warp a tree (csrc/runtime.cc, LogTail): more
trees than the chip holds blocks of four warps, up to 4 states and 256 nodes in
single precision; the per-tree engines' bits there and beside it."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

ITEMS = 1500


@pytest.mark.parametrize("states,nodes,scalar,single", [
    (1, 15, np.float32, True), (2, 1, np.float32, True), (2, 63, np.float32, True),
    (3, 256, np.float32, True), (4, 255, np.float32, True), (4, 257, np.float32, False),
    (2, 63, np.float64, False), (5, 63, np.float32, False)])
@pytest.mark.parametrize("shape", ["recursive", "star"])
def test_bits(gpu, shape, states, nodes, scalar, single):
    rng = np.random.default_rng(nodes + states)
    plan = gpu.Plan(np.array([-1] + [0] * (nodes - 1)) if shape == "star"
                    else synthetic.random_recursive(rng, nodes))
    ws = gpu.Workspace()
    ws._reserve("maximum,sampling", plan, states, ITEMS, 0, scalar, None)
    total = ITEMS * nodes
    model = gpu.BatchedModelView(plan, states, ITEMS,
                                 (rng.random(total * states) + 0.05).astype(scalar),
                                 (rng.random(plan.num_edges * states ** 2) + 0.01).astype(scalar))
    uniforms = rng.random(total).astype(scalar)

    def outputs():
        view = ws.maximum_a_posteriori_prepared(model)
        out = [np.array(view.log_weights), np.array(view.states)]
        return out + [np.array(ws.posterior_sample_prepared(model, uniforms).states)]

    got = outputs()
    assert (ws.launches == 1) == single
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs()):
        assert np.array_equal(a, b)
