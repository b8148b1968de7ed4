"""First-round rakes of the batch API with an item per lane
(csrc/phase_items.cuh, ItemPhaseKernel) against the per-tree engines, bit for
bit: padded and exact state counts, full and ragged last warps, dense and
categorical inputs, trees whose first round takes the kernel (600 rakes and
more) with wide and narrow gathers."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

STATES = [5, 8, 11, 16, 19, 20, 24, 27, 32]


def outputs(ws, model):
    view = ws.posterior_marginals_prepared(model)
    return [np.array(view.log_partitions), np.array(view.nodes), np.array(view.edges)]


def check(ws, model):
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    got = outputs(ws, model)
    assert np.all(np.isfinite(got[0]))
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs(ws, model)):
        assert np.array_equal(a, b)
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES, stripes=2)
    for a, b in zip(got, outputs(ws, model)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("items", [32, 33, 95])
@pytest.mark.parametrize("states", STATES)
def test_categorical(gpu, states, items, scalar):
    rng = np.random.default_rng(states + items)
    categories = states - 1
    parents = synthetic.leaf_splitting(rng, 2601)
    plan = gpu.Plan(parents)
    observed = synthetic.leaves(parents)
    ws = gpu.Workspace()
    ws.reserve_categorical_marginals(plan, states, items + 2, categories, observed, scalar=scalar)
    view = ws.categorical_inputs(items)
    view.observations[:] = rng.integers(0, categories, view.observations.size)
    view.root_potential[:] = rng.random(states) + 0.1
    view.emission_potentials[:] = rng.random(categories * states) + 0.1
    view.edge_potentials[:] = synthetic.stochastic_edges(rng, plan.num_edges, states, 0.7, scalar)
    check(ws, view)


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states,items", [(7, 40), (8, 64), (20, 63), (32, 33)])
def test_dense(gpu, states, items, scalar):
    rng = np.random.default_rng(7 * states)
    parents = np.concatenate([synthetic.random_recursive(rng, 1500), np.zeros(700, np.int64)])
    plan = gpu.Plan(parents)
    nodes = items * plan.num_nodes * states
    ws = gpu.Workspace()
    ws.reserve_marginals(plan, states, items, scalar=scalar)
    check(ws, gpu.BatchedModelView(
        plan, states, items, (rng.random(nodes) + 0.05).astype(scalar),
        synthetic.lognormal(rng, plan.num_edges * states * states, 1.0, 0.02, scalar)))
