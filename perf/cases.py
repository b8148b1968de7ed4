"""Performance cases: the calls that users of this package make, from one small
tree whose latency counts to forests of millions of nodes.

Three ways of calling are covered. A *call* is a prepared call of the
accelerator API on host data: inputs from pinned staging (or the caller's own
arrays) to results in host memory. A *sites* case is the batch API with one
topology and many items, inputs and results on the device. A *forest* is many
trees of their own shapes and edge factors, inputs and results on the device,
as in a training loop or a pipeline that makes its factors on the GPU; each
pass declares its inputs ready and enqueues one step.

Shapes and distributions are those of bench.py and of the tests: random
recursive trees, caterpillars, full binary trees, Galton-Watson trees and
path-heavy trees; row-stochastic (Dirichlet) or lognormal edge factors;
categorical leaves or dense node factors.
"""
import math

import numpy as np
import torch

import parallel_tree_hmm_gb300 as thmm
from parallel_tree_hmm_gb300 import _lib

_OPERATIONS = {
    "logz": _lib.THMM_OP_LOG_PARTITION,
    "marginals": _lib.THMM_OP_MARGINALS,
    "map": _lib.THMM_OP_MAXIMUM,
    "sample": _lib.THMM_OP_SAMPLE,
}
_KINDS = {"logz": "", "marginals": "marginals", "map": "maximum", "sample": "sampling"}


def _case(api, op, shape, states, trees, low, high, **more):
    """`trees` trees with node counts log-spaced over [low, high]; for the
    batch API ("call" and "sites") one tree of `high` nodes and `trees` items."""
    case = {"api": api, "op": op, "shape": shape, "states": states, "trees": trees,
            "low": low, "high": high, "scalar": 4, "compute": "default",
            "categorical": True, "edge_alpha": 0.5, "edge_sigma": 0.0, "zeros": 0.0}
    case.update(more)
    return case


def listed():
    cases = {
        # One small tree scored at a time (an interactive or per-request call)
        # with the API's default double precision and the caller's own arrays.
        "call-small": _case("call", "logz", "recursive", 3, 1, 127, 127, scalar=8,
                            categorical=False, edge_alpha=1.0),
        # The reference's own batch: 64 items on one 1,000-node binary tree,
        # new factors on each call (kFactors), double precision, from pinned
        # host inputs to host marginals.
        "call-binary": _case("call", "marginals", "binary", 4, 64, 999, 999, scalar=8,
                             edge_alpha=1.0),
        # A batch of uneven trees decoded from host data.
        "call-map": _case("forest-call", "map", "mixed", 8, 48, 150, 6000),
        # DNA-like alignment: many sites on one binary tree, shared edges.
        "sites-k4": _case("sites", "marginals", "binary", 4, 4096, 1999, 1999, edge_alpha=1.0),
        # Protein-like alignment: 20 states on the batch API.
        "sites-k20": _case("sites", "marginals", "binary", 20, 500, 399, 399, edge_alpha=1.0),
        # The headline forest: 4,096 uneven trees, half of them caterpillars.
        "forest-k4": _case("forest", "marginals", "mixed", 4, 4096, 200, 20000),
        # Likelihoods alone in full FP64 arithmetic, 3 states (rows that are
        # no multiple of 16 bytes).
        "forest-k3-f64": _case("forest", "logz", "mixed", 3, 512, 200, 20000, scalar=8,
                               compute="f64"),
        # Gradients of sum log Z for dense factors with exact zeros.
        "gradient-k20": _case("forest", "marginals", "recursive", 20, 256, 5000, 5000,
                              categorical=False, edge_sigma=1.5, zeros=0.02),
        # MAP reconstruction and posterior sampling of Galton-Watson trees.
        "gw-map-k8": _case("forest", "map", "galton-watson", 8, 320, 1000, 50000,
                           edge_alpha=0.3),
        "gw-sample-k8": _case("forest", "sample", "galton-watson", 8, 320, 1000, 50000,
                              edge_alpha=0.3),
        # Path-heavy trees with dense transition factors above 32 states.
        "dense-k64": _case("forest", "marginals", "spine", 64, 64, 2000, 2000,
                           categorical=False, edge_sigma=2.0, zeros=0.05),
        "dense-k128": _case("forest", "marginals", "spine", 128, 64, 500, 500,
                            categorical=False, edge_sigma=2.0, zeros=0.05),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    family = rng.choice(["call", "forest-call", "sites", "forest", "gradient", "gw", "dense"])
    scalar = rng.choice([4, 4, 8])
    compute = "f64" if scalar == 8 and rng.random() < 0.5 else "default"
    if family == "call":
        states, nodes = _log_uniform(rng, 2, 32), _log_uniform(rng, 5, 3000)
        items = max(1, min(_log_uniform(rng, 1, 256), 4_000_000 // (nodes * states * states)))
        return _case("call", rng.choice(list(_OPERATIONS)), rng.choice(["recursive", "binary"]),
                     states, items, nodes, nodes, scalar=scalar, compute=compute,
                     categorical=rng.random() < 0.5, edge_alpha=1.0)
    if family == "forest-call":
        states = _log_uniform(rng, 2, 16)
        high = _log_uniform(rng, 200, 20000)
        trees = max(1, min(_log_uniform(rng, 1, 256), 8_000_000 // (high * states * states)))
        return _case("forest-call", rng.choice(list(_OPERATIONS)), "mixed", states, trees,
                     min(high, 100), high, scalar=scalar, compute=compute)
    if family == "sites":
        states, nodes = _log_uniform(rng, 2, 32), _log_uniform(rng, 101, 4001)
        items = _log_uniform(rng, 64, 16384)
        items = max(32, min(items, 120_000_000 // (nodes * states * states)))
        return _case("sites", rng.choice(["logz", "marginals"]), "binary", states, items, nodes,
                     nodes, edge_alpha=1.0)
    if family == "forest":
        states = rng.choice([2, 3, 4, 4, _log_uniform(rng, 5, 32)])
        high = _log_uniform(rng, 1000, 20000)
        low = min(200, high)
        trees = _log_uniform(rng, 64, 4096)
        mean = (high - low) / math.log(high / low)
        trees = max(16, min(trees, int((250e6 if states <= 4 else 80e6) / scalar * 4 / 2 /
                                       (mean * states * states))))
        return _case("forest", rng.choice(["logz", "marginals"]), "mixed", states, trees, low,
                     high, scalar=scalar, compute=compute)
    if family == "gradient":
        states, nodes = _log_uniform(rng, 8, 32), _log_uniform(rng, 500, 5000)
        trees = max(8, min(_log_uniform(rng, 32, 1024), 400_000_000 // (nodes * states * states)))
        return _case("forest", "marginals", "recursive", states, trees, nodes, nodes,
                     categorical=False, edge_sigma=1.5, zeros=0.02)
    if family == "gw":
        states, high = _log_uniform(rng, 3, 16), _log_uniform(rng, 5000, 50000)
        trees = max(8, min(_log_uniform(rng, 16, 320), 150_000_000 // (high * states * states)))
        return _case("forest", rng.choice(["map", "sample"]), "galton-watson", states, trees,
                     1000, high, edge_alpha=0.3)
    states = rng.randint(33, 128)
    nodes = _log_uniform(rng, 200, 2000)
    most = 128_000 if states <= 64 else 32_000
    trees = max(4, min(_log_uniform(rng, 16, 128), most // nodes))
    return _case("forest", rng.choice(["logz", "marginals", "marginals"]), "spine", states,
                 trees, nodes, nodes, compute=rng.choice(["default", "default", "bf16"]),
                 categorical=False, edge_sigma=2.0, zeros=0.05)


# ------------------------------------------------------------------- inputs
def _batch_api(case):
    return case["api"] in ("call", "sites")


def _sizes(case):
    """Node counts of the trees; the same for every seed."""
    if _batch_api(case):
        n = case["high"]
        return np.array([n - 1 + n % 2 if case["shape"] == "binary" else n], dtype=np.int64)
    low, high = math.log(case["low"]), math.log(case["high"])
    if case["shape"] == "galton-watson":  # caps spread evenly, as a uniform draw's
        return np.linspace(case["low"], case["high"], case["trees"]).round().astype(np.int64)
    return np.exp(np.linspace(low, high, case["trees"])).round().astype(np.int64)


def _recursive(rng, n):
    parents = np.floor(rng.random(n) * np.arange(n)).astype(np.int64)
    parents[0] = -1
    return parents


def _binary(rng, n):
    """Full binary tree by splitting a uniform leaf until it has n nodes."""
    parents, leaves = [-1], [0]
    for u in rng.random(n // 2):
        index = int(u * len(leaves))
        node, first = leaves[index], len(parents)
        parents += [node, node]
        leaves[index] = first
        leaves.append(first + 1)
    return np.array(parents, dtype=np.int64)


def _caterpillar(n):
    spine = (n + 1) // 2
    return np.concatenate([[-1], np.arange(spine - 1), np.arange(n - spine)]).astype(np.int64)


def _spine(rng, n):
    parents = _recursive(rng, n)
    keep = rng.random(n) < 0.95
    keep[0] = False
    parents[keep] = np.flatnonzero(keep) - 1
    return parents


def _galton_watson(rng, n):
    """Breadth-first Poisson(2) tree grown to n nodes."""
    while True:
        counts = rng.poisson(2.0, size=n)
        born = 1 + np.cumsum(counts)
        if (born[:-1] > np.arange(1, n)).all():
            return np.concatenate([[-1], np.repeat(np.arange(n), counts)])[:n].astype(np.int64)


def _trees(case, seed):
    rng = np.random.default_rng(seed)
    sizes = rng.permutation(_sizes(case))
    trees = []
    for index, n in enumerate(sizes):
        n = int(n)
        shape = case["shape"]
        if shape == "mixed":
            shape = "recursive" if index % 2 == 0 else "caterpillar"
        trees.append(_recursive(rng, n) if shape == "recursive" else
                     _binary(rng, n) if shape == "binary" else
                     _caterpillar(n) if shape == "caterpillar" else
                     _spine(rng, n) if shape == "spine" else _galton_watson(rng, n))
    return trees


def _leaves(parents):
    has_child = np.zeros(len(parents), dtype=bool)
    has_child[parents[1:]] = True
    return np.flatnonzero(~has_child).astype(np.uint32)


def _rows(rng, rows, states, alpha, dtype):
    """Dirichlet(alpha) rows on the GPU."""
    if alpha == 0.5:  # squared normals
        values = torch.randn(rows, states, generator=rng, device="cuda", dtype=dtype).square_()
    elif alpha == 1.0:
        values = torch.empty(rows, states, device="cuda", dtype=dtype).exponential_(generator=rng)
    else:
        shape = torch.full((rows, states), alpha, device="cuda", dtype=dtype)
        values = torch._standard_gamma(shape, generator=rng)
    values /= values.sum(dim=1, keepdim=True)
    return values.nan_to_num_(1.0 / states)


def _model(case, seed):
    """The inputs of one pass as GPU tensors, made from the seed alone."""
    trees = _trees(case, seed)
    rng = torch.Generator(device="cuda")
    rng.manual_seed(seed)
    K = case["states"]
    dtype = torch.float64 if case["scalar"] == 8 else torch.float32
    items = case["trees"] if _batch_api(case) else 1
    nodes = sum(len(p) for p in trees)
    edges = nodes - len(trees)
    model = {"trees": trees, "items": items, "nodes": nodes, "edges": edges}
    if case["edge_sigma"] > 0:
        values = torch.randn(edges * K * K, generator=rng, device="cuda", dtype=dtype)
        values.mul_(case["edge_sigma"]).exp_()
        drop = torch.rand(values.shape, generator=rng, device="cuda") < case["zeros"]
        model["edge_potentials"] = values.masked_fill_(drop, 0.0)
    else:
        model["edge_potentials"] = _rows(rng, edges * K, K, case["edge_alpha"], dtype).view(-1)
    if case["categorical"]:
        observed = [_leaves(p) for p in trees]
        count = sum(len(o) for o in observed) * items
        model["observed"] = observed
        model["root_potential"] = _rows(rng, 1, K, 1.0, dtype).view(-1)
        model["emission_potentials"] = _rows(rng, K, K, 2.0, dtype).view(-1)
        model["observations"] = torch.randint(0, K, (count,), generator=rng, device="cuda",
                                              dtype=torch.uint8)
    else:
        model["node_potentials"] = torch.randn(nodes * items * K, generator=rng, device="cuda",
                                               dtype=dtype).exp_()
    if case["op"] == "sample":
        draws = torch.rand(nodes * items, generator=rng, device="cuda", dtype=dtype)
        model["uniforms"] = draws.clamp_(max=1 - 2.0 ** -20)
    return model


_INPUTS = ("node_potentials", "edge_potentials", "observations", "root_potential",
           "emission_potentials", "uniforms")


def prepare(case, seed):
    """Plans, a reserved workspace and the inputs where the caller has them:
    in the workspace's device buffers, or in host memory for a call."""
    model = _model(case, seed)
    K = case["states"]
    plans = thmm.Plan.many(model["trees"])
    ws = thmm.Workspace()
    on_device = case["api"] in ("sites", "forest")
    kind = ",".join(p for p in (_KINDS[case["op"]], "device" if on_device else "") if p)
    scalar = np.float64 if case["scalar"] == 8 else np.float32
    compute = {"default": None, "f64": np.float64, "bf16": "bf16"}[case["compute"]]
    if not _batch_api(case):
        if case["categorical"]:
            ws.reserve_forest_categorical(plans, K, K, model["observed"], kind=kind,
                                          scalar=scalar, compute=compute)
        else:
            ws.reserve_forest(plans, K, kind=kind, scalar=scalar, compute=compute)
    else:
        suffix = "_" + _KINDS[case["op"]] if _KINDS[case["op"]] else ""
        if case["categorical"]:
            getattr(ws, "reserve_categorical" + suffix)(plans[0], K, model["items"], K,
                                                        model["observed"][0], scalar=scalar,
                                                        compute=compute)
        else:
            getattr(ws, "reserve" + suffix)(plans[0], K, model["items"], scalar=scalar,
                                            compute=compute)
    state = {"case": case, "ws": ws, "plans": plans, "operation": _OPERATIONS[case["op"]]}
    if on_device:
        buffers = ws.device_buffers()
        for name in _INPUTS:
            if name in model:
                buffers[name].copy_(model[name])
        torch.cuda.synchronize()
        results = _Results(ws, values=buffers["values"])
        if case["op"] == "marginals":
            results.update(nodes=buffers["node_marginals"], edges=buffers["edge_marginals"])
        elif case["op"] in ("map", "sample"):
            results["states"] = buffers["states"].view(torch.int32)
        state["results"] = results
        return state
    host = {name: model[name].cpu().numpy() for name in _INPUTS if name in model}
    if case["categorical"]:
        view = ws.categorical_inputs()
        for name in ("observations", "root_potential", "emission_potentials", "edge_potentials"):
            getattr(view, name)[:] = host[name]
    elif case["trees"] == 1:  # the caller's own arrays
        view = ws.inputs()
        view.node_potentials, view.edge_potentials = host["node_potentials"], host["edge_potentials"]
    else:
        view = ws.inputs()
        view.node_potentials[:] = host["node_potentials"]
        view.edge_potentials[:] = host["edge_potentials"]
    state["view"] = view
    if case["op"] == "sample":
        state["uniforms"] = ws.uniforms()
        state["uniforms"][:] = host["uniforms"]
    if case["categorical"]:
        # Observations stay resident; each pass brings new factors.
        _call(state, thmm.CategoricalInputUpdate.kAll)
    return state


class _Results(dict):
    """Results that live in a workspace, which they keep."""

    def __init__(self, owner, **results):
        super().__init__(results)
        self.owner = owner


def _call(state, update):
    ws, view, op = state["ws"], state["view"], state["case"]["op"]
    if op == "logz":
        return _Results(ws, values=ws.log_partition_function_prepared(view, update).values)
    if op == "marginals":
        result = ws.posterior_marginals_prepared(view, update)
        return _Results(ws, values=result.log_partitions, nodes=result.nodes, edges=result.edges)
    if op == "map":
        result = ws.maximum_a_posteriori_prepared(view, update)
        return _Results(ws, values=result.log_weights, states=result.states.view(np.int32))
    states = ws.posterior_sample_prepared(view, state["uniforms"], update).states
    return _Results(ws, states=states.view(np.int32))


def run(state):
    """One pass: a prepared call on the host inputs, or one device step on
    inputs that were just written."""
    if "view" in state:
        return _call(state, thmm.CategoricalInputUpdate.kFactors
                     if state["case"]["categorical"] else None)
    state["ws"].device_inputs_ready()
    state["ws"].enqueue(state["operation"])
    return state["results"]


# --------------------------------------------------------------------- work
def work(case):
    """Inputs read once and outputs written once; the operations of one pass
    of messages over each edge (and one back for marginals)."""
    K, S = case["states"], case["scalar"]
    sizes = _sizes(case)
    items = case["trees"] if _batch_api(case) else 1
    nodes = int(sizes.sum()) * items
    edges_in = int((sizes - 1).sum())
    edges = edges_in * items
    moved = edges_in * K * K * S + len(sizes) * items * S
    moved += nodes // 2 if case["categorical"] else nodes * K * S
    flops = edges * 2 * K * K
    if case["op"] == "marginals":
        moved += nodes * K * S + edges * K * K * S
        flops += edges * 4 * K * K
    elif case["op"] in ("map", "sample"):
        moved += nodes * 4 + (nodes * S if case["op"] == "sample" else 0)
    return {"bytes": moved, "flops": flops}


# -------------------------------------------------------------------- exact
def _depths(parent):
    """Depth of every node by pointer doubling (a root is its own parent)."""
    jump = parent.clone()
    depth = (parent != torch.arange(len(parent), device=parent.device)).long()
    while True:
        step = depth[jump]
        if not bool(step.any()):
            return depth
        depth = depth + step
        jump = jump[jump]


def exact(case, seed):
    """Message passing level by level in 64 bits: sum-product (log Z, node and
    edge marginals) or max-product (the MAP log weight)."""
    model = _model(case, seed)
    K, items, trees = case["states"], model["items"], model["trees"]
    f64 = torch.float64
    starts = np.cumsum([0] + [len(p) for p in trees])
    parent = np.concatenate([np.concatenate([[s], p[1:] + s]) for p, s in zip(trees, starts)])
    roots = torch.as_tensor(starts[:-1], device="cuda")
    one_edges = model["edge_potentials"].to(f64).view(-1, K, K)
    is_root = np.zeros(len(parent), dtype=bool)
    is_root[starts[:-1]] = True
    edge_of = torch.as_tensor(np.cumsum(~is_root) - 1, device="cuda")
    n = model["nodes"]
    parent = torch.as_tensor(parent, device="cuda")
    depth = _depths(parent)
    if case["categorical"]:
        phi = torch.ones(items, n, K, device="cuda", dtype=f64)
        phi[:, roots] = model["root_potential"].to(f64)
        seen = np.concatenate([o.astype(np.int64) + s for o, s in zip(model["observed"], starts)])
        seen = torch.as_tensor(seen, device="cuda")
        emission = model["emission_potentials"].to(f64).view(K, K)
        phi[:, seen] *= emission[model["observations"].long()].view(items, -1, K)
    else:
        phi = model["node_potentials"].to(f64).view(items, n, K).clone()
    # Nodes in depth order, so that a level is a slice; items innermost.
    order = torch.argsort(depth, stable=True)
    rank = torch.empty_like(order)
    rank[order] = torch.arange(n, device="cuda")
    up = phi[:, order].log_().transpose(0, 1).contiguous()  # [node, item, state]
    del phi
    above = rank[parent[order]]
    edge_at = edge_of[order]
    bounds = torch.cumsum(torch.bincount(depth), 0).tolist()
    levels = list(zip(bounds[:-1], bounds[1:]))
    maximum = case["op"] == "map"
    for a, b in reversed(levels):
        matrix = one_edges[edge_at[a:b]]  # [node, parent state, child state]
        top = up[a:b].amax(dim=2, keepdim=True)
        if maximum:
            message = (matrix.log()[:, None] + up[a:b, :, None]).amax(dim=3)
        else:
            weight = torch.exp(up[a:b] - top)
            message = torch.log(torch.einsum("npc,nic->nip", matrix, weight)) + top
        up.index_add_(0, above[a:b], message)
    at_root = up[: len(trees)]  # depth 0, in tree order
    if maximum:
        return {"values": at_root.amax(dim=2).transpose(0, 1).reshape(-1), "states": None}
    log_z = torch.logsumexp(at_root, dim=2)
    values = log_z.transpose(0, 1).reshape(-1)
    if case["op"] == "sample":
        return ({"states": None} if case["api"] in ("call", "forest-call")
                else {"values": values, "states": None})
    if case["op"] == "logz":
        return {"values": values}
    node_out = torch.empty_like(up)
    node_out[: len(trees)] = torch.exp(at_root - log_z[:, :, None])
    edge_out = torch.empty(items, model["edges"], K, K, device="cuda", dtype=f64)
    for a, b in levels:
        matrix = one_edges[edge_at[a:b]]
        weight = torch.exp(up[a:b] - up[a:b].amax(dim=2, keepdim=True))
        total = torch.einsum("npc,nic->nip", matrix, weight)
        ratio = torch.where(total > 0, node_out[above[a:b]] / total, torch.zeros_like(total))
        joint = ratio[:, :, :, None] * matrix[:, None] * weight[:, :, None]
        node_out[a:b] = joint.sum(dim=2)
        edge_out[:, edge_at[a:b]] = joint.transpose(0, 1)
    nodes = torch.empty_like(node_out)
    nodes[order] = node_out
    return {"values": values, "nodes": nodes.transpose(0, 1).reshape(-1),
            "edges": edge_out.view(-1)}
