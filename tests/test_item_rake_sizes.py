"""The trees and item counts of tests/test_gpu_item_rakes.py reach the kernels that
it is about: the first round of each has warps of 32 items enough for the rule in
csrc/phase_groups_launch.cuh, gathers and rakes alike."""
import pathlib
import re

import numpy as np
import pytest

from parallel_tree_hmm_gb300 import synthetic

LAUNCH = (pathlib.Path(__file__).resolve().parent.parent / "parallel_tree_hmm_gb300" / "csrc" /
          "phase_groups_launch.cuh")


def check(thmm, parents, items):
    needed = int(re.search(r"kItemWarps = (\d+);", LAUNCH.read_text()).group(1))
    plan = thmm.Plan(parents)
    kind, first, count = plan.batches[0]
    assert (kind, first) == (0, 0)  # the first round's rakes
    parent_of = dict(zip(plan.edge_children.tolist(), plan.edge_parents.tolist()))
    gathers = {parent_of[leaf] for leaf in plan.rakes[:count, 1].tolist()}
    tiles = (items + 31) // 32
    assert min(len(gathers), count) * tiles >= needed


@pytest.mark.parametrize("items", [32, 33, 95])
@pytest.mark.parametrize("states", [5, 8, 11, 16, 19, 20, 24, 27, 32])
def test_categorical(thmm, states, items):
    rng = np.random.default_rng(states + items)
    check(thmm, synthetic.leaf_splitting(rng, 2601), items)


@pytest.mark.parametrize("states,items", [(7, 40), (8, 64), (20, 63), (32, 33)])
def test_dense(thmm, states, items):
    rng = np.random.default_rng(7 * states)
    check(thmm, np.concatenate([synthetic.random_recursive(rng, 1500), np.zeros(700, np.int64)]),
          items)
