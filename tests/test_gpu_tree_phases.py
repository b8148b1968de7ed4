"""Small batches with a whole tree per block (csrc/phase_tree.cuh,
TreePhaseKernel) against the per-tree engines: every input and arithmetic
width, dense and categorical inputs, one node to the largest trees that fit,
on both sides of the rule's limits; bit for bit (log Z in FP64 included)."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

TYPES = [(np.float32, None), (np.float64, None), (np.float32, np.float64),
         (np.float64, np.float64)]


def outputs(ws, model):
    view = ws.posterior_marginals_prepared(model)
    out = [np.array(view.log_partitions), np.array(view.nodes), np.array(view.edges)]
    launches = ws.launches
    out.append(np.array(ws.log_partition_function_prepared(model).values))
    out.append(np.array(ws.partition_function_prepared(model).values))
    return out, launches


def check(ws, model, single):
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    got, launches = outputs(ws, model)
    assert (launches == 1) == single
    assert np.array_equal(got[0], got[3]) and np.all(np.isfinite(got[0]))
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs(ws, model)[0]):
        assert np.array_equal(a, b)
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES, stripes=2)
    for a, b in zip(got, outputs(ws, model)[0]):
        assert np.array_equal(a, b)


def parents(rng, nodes, shape):
    if shape == "star":
        return np.array([-1] + [0] * (nodes - 1))
    return (synthetic.random_recursive(rng, nodes) if shape == "recursive"
            else synthetic.caterpillar(nodes))


@pytest.mark.parametrize("scalar,compute", TYPES)
@pytest.mark.parametrize("nodes,shape", [(1, "recursive"), (2, "recursive"), (3, "star"),
                                         (130, "star"), (511, "caterpillar"),
                                         (512, "recursive"), (513, "recursive")])
@pytest.mark.parametrize("states,items", [(1, 3), (2, 1), (3, 5), (4, 2), (4, 40)])
def test_dense(gpu, states, items, nodes, shape, scalar, compute):
    rng = np.random.default_rng(31 * states + nodes)
    plan = gpu.Plan(parents(rng, nodes, shape))
    ws = gpu.Workspace()
    ws.reserve_marginals(plan, states, items, scalar=scalar, compute=compute)
    model = gpu.BatchedModelView(
        plan, states, items, (rng.random(items * nodes * states) + 0.05).astype(scalar),
        synthetic.lognormal(rng, plan.num_edges * states * states, 0.7,
                            0.05 if states > 2 else 0.0, scalar))
    check(ws, model, nodes <= 512 or items >= 32)


@pytest.mark.parametrize("scalar,compute", TYPES)
@pytest.mark.parametrize("nodes,items", [(61, 1), (999, 33), (999, 31), (2600, 40)])
def test_categorical(gpu, nodes, items, scalar, compute):
    rng = np.random.default_rng(nodes)
    states, categories = 4, 6
    tree = synthetic.leaf_splitting(rng, nodes)
    plan = gpu.Plan(tree)
    observed = np.concatenate([[0], synthetic.leaves(tree)]).astype(np.uint32)
    ws = gpu.Workspace()
    ws.reserve_categorical_marginals(plan, states, items + 1, categories, observed,
                                     scalar=scalar, compute=compute)
    view = ws.categorical_inputs(items)
    view.observations[:] = rng.integers(0, categories, view.observations.size)
    view.root_potential[:] = rng.random(states) + 0.1
    view.emission_potentials[:] = rng.random(categories * states) + 0.1
    view.edge_potentials[:] = synthetic.stochastic_edges(rng, plan.num_edges, states, 0.7, scalar)
    # 2,600 nodes do not fit; FP64 arithmetic of 999 nodes takes 264 KB.
    check(ws, view, items >= 32 and nodes < 1000 and compute is None or nodes <= 512)
