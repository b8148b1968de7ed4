"""Graph replay of prepared calls (a call of 8 launches and more, from its tenth
repeat on) and of the device-only step: new inputs, other operations, retuning,
sampling errors and more graphs than are kept give the bits of a fresh
workspace, and building a graph takes no notice of what other threads do to the
device."""
import threading

import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

STATES = 8


def plans_of(gpu, rng):
    return gpu.Plan.many([synthetic.random_recursive(rng, n) for n in (900, 2500, 40)])


def workspace(gpu, plans):
    ws = gpu.Workspace()
    ws.reserve_forest(plans, STATES, kind="marginals,maximum,sampling", scalar=np.float32)
    return ws


def model_of(gpu, plans, seed):
    rng = np.random.default_rng(seed)
    nodes = sum(p.num_nodes for p in plans)
    edges = sum(p.num_edges for p in plans)
    return (gpu.BatchedModelView(None, STATES, len(plans),
                                 (rng.random(nodes * STATES) + 0.05).astype(np.float32),
                                 (rng.random(edges * STATES ** 2) + 0.01).astype(np.float32)),
            rng.random(nodes).astype(np.float32))


def call(ws, operation, model, uniforms):
    if operation == "marginals":
        view = ws.posterior_marginals_prepared(model)
        return [np.array(view.log_partitions), np.array(view.nodes), np.array(view.edges)]
    if operation == "logz":
        return [np.array(ws.log_partition_function_prepared(model).values)]
    if operation == "map":
        view = ws.maximum_a_posteriori_prepared(model)
        return [np.array(view.log_weights), np.array(view.states)]
    return [np.array(ws.posterior_sample_prepared(model, uniforms).states)]


def same(got, expected):
    for a, b in zip(got, expected, strict=True):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("operation", ["marginals", "logz", "map", "sample"])
def test_prepared_calls_with_new_factors(gpu, operation):
    plans = plans_of(gpu, np.random.default_rng(1))
    ws = workspace(gpu, plans)
    other = "map" if operation == "marginals" else "marginals"
    for seed in range(30):
        model, uniforms = model_of(gpu, plans, seed)
        same(call(ws, operation, model, uniforms),
             call(workspace(gpu, plans), operation, model, uniforms))
        if seed == 12:  # another operation and back
            same(call(ws, other, model, uniforms),
                 call(workspace(gpu, plans), other, model, uniforms))
        if seed == 15:
            ws.set_tuning(256, schedule=_lib.THMM_SCHEDULE_PHASES, phase_rounds=2)
        if seed == 27 and operation == "sample":
            bad = uniforms.copy()
            bad[5] = 1.5
            with pytest.raises(gpu.InvalidArgument):
                ws.posterior_sample_prepared(model, bad)


def test_replay_after_a_sampling_error(gpu):
    plans = plans_of(gpu, np.random.default_rng(2))
    ws = workspace(gpu, plans)
    model, uniforms = model_of(gpu, plans, 3)
    expected = call(workspace(gpu, plans), "sample", model, uniforms)
    for _ in range(12):
        same(call(ws, "sample", model, uniforms), expected)
    with pytest.raises(gpu.InvalidArgument):
        ws.posterior_sample_prepared(model, np.full_like(uniforms, 1.0))
    same(call(ws, "sample", model, uniforms), expected)


def test_more_graphs_than_are_kept(gpu):
    """Device-only steps and prepared calls over 300 batch sizes (at most 256
    graphs are kept), twice round, then one of them often enough to have its
    graph built in the place of another's."""
    rng = np.random.default_rng(4)
    plan = gpu.Plan(synthetic.random_recursive(rng, 60))
    capacity = 300
    ws = gpu.Workspace()
    ws.reserve_marginals(plan, 5, capacity, scalar=np.float32)
    nodes = (rng.random(capacity * plan.num_nodes * 5) + 0.05).astype(np.float32)
    edges = (rng.random(plan.num_edges * 25) + 0.01).astype(np.float32)

    def model(batch):
        return gpu.BatchedModelView(plan, 5, batch, nodes[:batch * plan.num_nodes * 5], edges)

    expected = np.array(ws.log_partition_function_prepared(model(capacity)).values)
    for _ in range(2):
        for batch in range(1, capacity + 1):
            view = ws.log_partition_function_prepared(model(batch))
            assert np.array_equal(view.values, expected[:batch])
            ws.enqueue(_lib.THMM_OP_LOG_PARTITION)
            launches = ws.launches
            ws.enqueue(_lib.THMM_OP_LOG_PARTITION)
            assert ws.launches == launches
    for batch in (capacity, 1, capacity - 1):
        for _ in range(12):
            view = ws.log_partition_function_prepared(model(batch))
            assert np.array_equal(view.values, expected[:batch])
            ws.enqueue(_lib.THMM_OP_LOG_PARTITION)
    ws.synchronize()


def test_another_thread_synchronises_the_device(gpu):
    """A device-wide synchronisation in one thread while another's calls build
    and replay graphs: neither fails."""
    torch = pytest.importorskip("torch")
    plans = plans_of(gpu, np.random.default_rng(5))
    ws = workspace(gpu, plans)
    model, uniforms = model_of(gpu, plans, 6)
    expected = call(ws, "marginals", model, uniforms)
    torch.cuda.synchronize()
    errors, done = [], threading.Event()

    def synchronise():
        try:
            while not done.is_set():
                torch.cuda.synchronize()
        except Exception as error:  # noqa: BLE001
            errors.append(error)

    thread = threading.Thread(target=synchronise)
    thread.start()
    try:
        for _ in range(60):
            ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES)  # drops the graphs
            for _ in range(11):
                got = call(ws, "marginals", model, uniforms)
            same(got, expected)
            ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES)
            ws.enqueue(_lib.THMM_OP_MARGINALS)
            ws.synchronize()
    finally:
        done.set()
        thread.join()
    assert not errors, errors[0]
