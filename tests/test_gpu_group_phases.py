"""Lane-group phase kernels (csrc/phase_groups.cuh, 4 < K <= 32) against the
per-tree engines, bit for bit: every tile shape at its padded state count, one
below and at the first count above it (16-byte rows and padded rows), every
input and arithmetic width, forests and the batch API's shared topology."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

STATES = [5, 7, 8, 9, 12, 15, 16, 17, 19, 20, 21, 24, 25, 28, 29, 32]
TYPES = [(np.float32, None), (np.float64, None), (np.float32, np.float64),
         (np.float64, np.float64)]


def outputs(ws, model):
    view = ws.posterior_marginals_prepared(model)
    out = [np.array(view.log_partitions), np.array(view.nodes), np.array(view.edges)]
    out.append(np.array(ws.log_partition_function_prepared(model).values))
    return out


def check(ws, model):
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    got = outputs(ws, model)
    assert np.array_equal(got[0], got[3]) and np.all(np.isfinite(got[0]))
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_TEAMS)
    for a, b in zip(got, outputs(ws, model)):
        assert np.array_equal(a, b)
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES, stripes=3)
    for a, b in zip(got, outputs(ws, model)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("scalar,compute", TYPES)
@pytest.mark.parametrize("states", STATES)
def test_forest(gpu, states, scalar, compute):
    rng = np.random.default_rng(100 + states)
    shapes = [synthetic.random_recursive(rng, n) for n in (1, 2, 33, 400)]
    shapes += [synthetic.caterpillar(150), np.arange(-1, 70),
               np.array([-1] + [0] * 40), synthetic.spine_heavy(rng, 300)]
    plans = gpu.Plan.many(shapes)
    nodes = sum(p.num_nodes for p in plans)
    edges = sum(p.num_edges for p in plans)
    ws = gpu.Workspace()
    ws.reserve_forest(plans, states, kind="marginals", scalar=scalar, compute=compute)
    check(ws, gpu.BatchedModelView(
        None, states, len(plans), (rng.random(nodes * states) + 0.05).astype(scalar),
        synthetic.lognormal(rng, edges * states * states, 1.0, 0.05, scalar)))


@pytest.mark.parametrize("scalar,compute", TYPES)
@pytest.mark.parametrize("states,items", [(5, 33), (8, 1), (13, 5), (20, 3), (20, 40), (31, 2)])
def test_batch(gpu, states, items, scalar, compute):
    rng = np.random.default_rng(200 + states)
    parents = synthetic.leaf_splitting(rng, 61)
    plan = gpu.Plan(parents)
    observed = synthetic.leaves(parents)
    ws = gpu.Workspace()
    ws.reserve_categorical_marginals(plan, states, items + 2, states, observed, scalar=scalar,
                                     compute=compute)
    view = ws.categorical_inputs(items)
    view.observations[:] = rng.integers(0, states, view.observations.size)
    view.root_potential[:] = rng.random(states) + 0.1
    view.emission_potentials[:] = rng.random(states * states) + 0.1
    view.edge_potentials[:] = synthetic.stochastic_edges(rng, plan.num_edges, states, 0.7, scalar)
    check(ws, view)
