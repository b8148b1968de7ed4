"""MAP and sampling rounds whose rakes are launched apart from their sums
(csrc/runtime.cc, SplitRound): the per-tree engines' states and log weights, bit
for bit, for fan-ins up to and above those that get a block of their own, in
calls of more trees than have tails, and not slower than those engines."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib

pytestmark = pytest.mark.gpu

ITEMS = 3000  # more than the chip holds tail blocks of any kernel


def batch(gpu, states, leaves, scalar, kind="maximum,sampling"):
    rng = np.random.default_rng(leaves)
    plan = gpu.Plan(np.array([-1] + [0] * leaves + [1, 1, 2]))
    ws = gpu.Workspace()
    ws._reserve(kind, plan, states, ITEMS, 0, scalar, None)
    nodes = ITEMS * plan.num_nodes
    model = gpu.BatchedModelView(plan, states, ITEMS,
                                 (rng.random(nodes * states) + 0.05).astype(scalar),
                                 (rng.random(plan.num_edges * states ** 2) + 0.01).astype(scalar))
    return ws, model, rng.random(nodes).astype(scalar)


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states", [3, 4, 7, 8, 20])
@pytest.mark.parametrize("leaves", [4, 15, 16, 17, 18, 40])
def test_bits(gpu, states, leaves, scalar):
    ws, model, uniforms = batch(gpu, states, leaves, scalar)

    def outputs():
        view = ws.maximum_a_posteriori_prepared(model)
        out = [np.array(view.log_weights), np.array(view.states)]
        return out + [np.array(ws.posterior_sample_prepared(model, uniforms).states)]

    got = outputs()
    assert ws.launches > 1
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs()):
        assert np.array_equal(a, b)


def test_time(gpu):
    """Twice the per-tree engines' time and more while one group took a gather's
    rakes one after the other."""
    ws, model, _ = batch(gpu, 4, 15, np.float64, "maximum")

    def kernel_ms():
        return min(ws.maximum_a_posteriori_prepared(model).timings.kernel_ms for _ in range(5))

    phases = kernel_ms()
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    assert phases <= 1.2 * kernel_ms()
