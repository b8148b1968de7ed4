"""Where a batch up to 4 states runs a tree per block and where a launch per
round and kind (csrc/runtime.cc, TreeLayout), on both sides of the line for 152
SMs; the same bits."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("states,compute,nodes,limit", [
    (4, np.float64, 3, 304), (4, np.float64, 61, 456), (2, np.float64, 61, 456),
    (4, None, 3, 608), (4, None, 61, 1216), (2, None, 61, 1216)])
def test_items_a_launch(gpu, states, compute, nodes, limit):
    rng = np.random.default_rng(nodes)
    plan = gpu.Plan(synthetic.leaf_splitting(rng, nodes))
    ws = gpu.Workspace()
    ws.reserve_marginals(plan, states, limit + 1, compute=compute)
    values = rng.random((limit + 1) * nodes * states) + 0.05
    edges = rng.random(plan.num_edges * states ** 2) + 0.01

    def outputs(items):
        view = ws.posterior_marginals_prepared(
            gpu.BatchedModelView(plan, states, items, values[:items * nodes * states], edges))
        return [np.array(view.log_partitions), np.array(view.nodes), np.array(view.edges)]

    inside = outputs(limit)
    assert ws.launches == 1
    outside = outputs(limit + 1)
    assert ws.launches > 1
    for a, b in zip(inside, outside):
        assert np.array_equal(a, b[:a.size])
