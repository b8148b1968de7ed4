"""Log Z alone of small trees, 5 to 8 states in the batch API: one launch of the
per-tree engine (csrc/runtime.cc, OneLaunch) where the rounds would cost more, on
both sides of the rule and by stripes; the marginals' log Z, bit for bit."""
import numpy as np
import pytest

from parallel_tree_hmm_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scalar,compute", [(np.float32, None), (np.float64, None),
                                            (np.float64, np.float64)])
@pytest.mark.parametrize("states,nodes,items,shape,single", [
    (5, 3, 1, "recursive", True), (5, 48, 7, "recursive", True),
    (5, 49, 7, "recursive", False), (8, 31, 2048, "recursive", True),
    (8, 31, 2049, "recursive", False), (7, 200, 33, "star", True),
    (9, 31, 5, "recursive", False), (6, 1, 3, "recursive", True)])
def test_log_partition(gpu, states, nodes, items, shape, single, scalar, compute):
    rng = np.random.default_rng(nodes)
    plan = gpu.Plan(np.array([-1] + [0] * (nodes - 1)) if shape == "star"
                    else synthetic.random_recursive(rng, nodes))
    ws = gpu.Workspace()
    ws.reserve_marginals(plan, states, items, scalar=scalar, compute=compute)
    assert ws.tuning["schedule"] == _lib.THMM_SCHEDULE_PHASES
    model = gpu.BatchedModelView(plan, states, items,
                                 (rng.random(items * nodes * states) + 0.05).astype(scalar),
                                 (rng.random(plan.num_edges * states ** 2) + 0.01).astype(scalar))
    expected = np.array(ws.posterior_marginals_prepared(model).log_partitions)
    assert np.array_equal(ws.log_partition_function_prepared(model).values, expected)
    assert (ws.launches == 1) == single
    raw = np.array(ws.partition_function_prepared(model).values)
    for _ in range(2):
        ws.enqueue(_lib.THMM_OP_LOG_PARTITION)
    ws.synchronize()
    assert np.array_equal(ws.log_partition_function_prepared(model).values, expected)
    ws.set_tuning(1024, schedule=_lib.THMM_SCHEDULE_PHASES, stripes=3)
    assert np.array_equal(ws.log_partition_function_prepared(model).values, expected)
    assert np.array_equal(ws.partition_function_prepared(model).values, raw)
