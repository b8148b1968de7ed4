"""Workspaces are independent of each other (include/thmm_gb300.h): calls of
several threads, each on a workspace of its own, succeed and give the bits that
they give alone."""
import threading

import numpy as np
import pytest

from parallel_tree_hmm_gb300 import synthetic

pytestmark = pytest.mark.gpu


def outputs(ws, model):
    view = ws.posterior_marginals_prepared(model)
    return [np.array(view.log_partitions), np.array(view.nodes), np.array(view.edges)]


def run_together(tasks):
    """Runs every task in a thread of its own, started together; raises the first
    exception of any of them."""
    errors = []
    start = threading.Barrier(len(tasks))

    def body(task):
        try:
            start.wait()
            task()
        except Exception as error:  # noqa: BLE001
            errors.append(error)

    threads = [threading.Thread(target=body, args=(task,)) for task in tasks]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    if errors:
        raise errors[0]


@pytest.mark.parametrize("states,compute", [(4, None), (3, np.float64)])
def test_trees_per_block_of_several_sizes(gpu, states, compute):
    """A tree per block (csrc/phase_tree.cuh) above 48 KB of shared memory, the
    same kernel at a size of its own in each thread."""
    sizes = (320, 380, 440, 500)
    tasks = []
    for index, nodes in enumerate(sizes):
        rng = np.random.default_rng(nodes + states)
        plan = gpu.Plan(synthetic.random_recursive(rng, nodes))
        ws = gpu.Workspace()
        ws.reserve_marginals(plan, states, 2, compute=compute)
        model = gpu.BatchedModelView(plan, states, 2,
                                     rng.random(2 * nodes * states) + 0.05,
                                     rng.random(plan.num_edges * states * states) + 0.01)
        expected = outputs(ws, model)
        assert ws.launches == 1

        def task(ws=ws, model=model, expected=expected):
            for _ in range(1500):
                ws.posterior_marginals_prepared(model)
            for a, b in zip(outputs(ws, model), expected):
                assert np.array_equal(a, b)

        tasks.append(task)
    run_together(tasks)
