"""MAP and sampling on the phase schedule (csrc/phase_log.cuh) against the
per-tree engines: the same states and the same log weights, bit for bit, at
the fan-ins where a gather's pairwise sums change place (register levels up to
31 rakes, scratch levels from 32 on), on both sides of every padded state
count, and with all, some or none of a tree's rounds in the tail launch."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


def star(n):
    return np.array([-1] + [0] * (n - 1), dtype=np.int64)


def trees(rng):
    shapes = [star(n) for n in (1, 2, 4, 32, 33, 34, 65, 129, 700)]
    shapes += [synthetic.caterpillar(n) for n in (5, 64, 901)]
    shapes += [synthetic.random_recursive(rng, n) for n in (40, 2500)]
    shapes += [np.arange(-1, 299), synthetic.spine_heavy(rng, 800, 0.7)]
    return shapes


def run(ws, model, uniforms):
    result = ws.maximum_a_posteriori_prepared(model)
    out = [np.array(result.log_weights), np.array(result.states)]
    out.append(np.array(ws.posterior_sample_prepared(model, uniforms).states))
    return out


def check(ws, model, uniforms):
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    got = run(ws, model, uniforms)
    for threshold in (1, 1 << 31):
        ws.set_tuning(threshold, schedule=_lib.THMM_SCHEDULE_TEAMS)
        for a, b in zip(got, run(ws, model, uniforms)):
            assert np.array_equal(a, b)
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES, stripes=3)
    for a, b in zip(got, run(ws, model, uniforms)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("scalar", [np.float32, np.float64])
@pytest.mark.parametrize("states", [1, 2, 3, 4, 5, 8, 9, 16, 17, 20, 21, 32])
def test_forest(gpu, states, scalar):
    rng = np.random.default_rng(states)
    plans = gpu.Plan.many(trees(rng))
    nodes = sum(p.num_nodes for p in plans)
    edges = sum(p.num_edges for p in plans)
    ws = gpu.Workspace()
    ws.reserve_forest(plans, states, kind="maximum,sampling", scalar=scalar)
    values = synthetic.lognormal(rng, edges * states * states, 1.0,
                                 0.05 if states > 4 else 0.0, scalar)
    model = gpu.BatchedModelView(None, states, len(plans),
                                 (rng.random(nodes * states) + 0.05).astype(scalar), values)
    check(ws, model, rng.random(nodes).astype(scalar))


@pytest.mark.parametrize("states,items", [(3, 1), (4, 33), (8, 5), (20, 7), (29, 2)])
@pytest.mark.parametrize("nodes", [1, 40, 1500])
def test_batch(gpu, states, items, nodes):
    rng = np.random.default_rng(7 * states + nodes)
    plan = gpu.Plan(synthetic.random_recursive(rng, nodes))
    observed = np.arange(0, nodes, 2, dtype=np.uint32)
    ws = gpu.Workspace()
    flags = "maximum,sampling"
    ws._reserve_categorical(flags, plan, states, items + 1, states, observed, 0, np.float32, None)
    view = ws.categorical_inputs(items)
    view.observations[:] = rng.integers(0, states + 1, view.observations.size)
    view.observations[view.observations == states] = 0
    view.root_potential[:] = rng.random(states) + 0.1
    view.emission_potentials[:] = rng.random(states * states) + 0.1
    view.edge_potentials[:] = rng.random(view.edge_potentials.size) + 0.01
    check(ws, view, rng.random(items * nodes).astype(np.float32))
