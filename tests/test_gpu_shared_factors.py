"""Batch API, 5 to 32 states: every item reads the same edge matrices. A state
count that fills its tile, whose matrices come in 16-byte copies, takes no
longer than one state less."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def kernel_ms(gpu, states):
    rng = np.random.default_rng(states)
    plan = gpu.Plan(np.array([-1, 0, 0]))
    items = 8192
    ws = gpu.Workspace()
    ws.reserve_marginals(plan, states, items, scalar=np.float32)
    model = gpu.BatchedModelView(plan, states, items,
                                 (rng.random(items * 3 * states) + 0.05).astype(np.float32),
                                 (rng.random(2 * states ** 2) + 0.01).astype(np.float32))
    return min(ws.posterior_marginals_prepared(model).timings.kernel_ms for _ in range(10))


@pytest.mark.parametrize("states", [8, 16, 20])
def test_one_matrix_for_many_items(gpu, states):
    assert kernel_ms(gpu, states) <= 1.5 * kernel_ms(gpu, states - 1)
