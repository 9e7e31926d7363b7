"""The work a user of this package has it do, as timed cases: walks of both kinds from the smallest demo batch to a graph of
half a billion edges, the skip-gram pairs made of them, graphs that are built before they are walked, and host arrays.

A case is a dict of plain values. ``kind`` says which program it stands for:

* ``uniform``   ``random_walk`` on CUDA tensors. ``draws`` is where its random numbers come from: ``given`` (a ``rand`` array, as in
  the reference's own call) or ``kernel`` (``rand=None``). ``graph``: ``plain`` passes ``rowptr, col``; ``fused`` a
  ``WalkGraph`` with fused edge records that the program keeps.
* ``node2vec``  ``rejection_sampling`` on CUDA tensors. ``graph``: ``plain`` passes ``rowptr, col`` and leaves the rest to the
  operator; ``search`` forbids the edge hash set; ``hash`` keeps a ``WalkGraph`` with the hash set, ``filter`` one
  with the triangle filter too.
* ``skipgram``  one training batch: walks, negative rows, and the context windows of both.
* ``new_graph`` an edge list becomes a CSR, a prepared graph and one epoch of walks in the same pass.
* ``host``      either operator on host arrays, the result landing in host memory.

Graphs are R-MAT with the benchmark's parameters; ids are squeezed to ``nodes`` so that any number of nodes is possible. All
outputs are node and edge ids, so every comparison is exact."""
import math

import torch

from mlx_cluster_b200 import (WalkGraph, context_windows, csr_from_edges, graphs, negative_walks, random_walk,
                              rejection_sampling)

#: (p, q) pairs of the tests and the benchmark; (1, 1) is what most node2vec users leave in place.
PQ = ((1.0, 1.0), (0.5, 2.0), (4.0, 0.25), (0.25, 4.0), (1.0, 2.0))


def _uniform(name, nodes, edges, starts, length, *, draws="given", graph="plain", directed=False, return_edges=False):
    return dict(name=name, kind="uniform", nodes=nodes, edges=edges, starts=starts, length=length, draws=draws, graph=graph,
                directed=directed, return_edges=return_edges)


def _node2vec(name, nodes, edges, starts, length, p, q, *, graph="plain", directed=False, return_edges=False):
    return dict(name=name, kind="node2vec", nodes=nodes, edges=edges, starts=starts, length=length, p=p, q=q, graph=graph,
                directed=directed, return_edges=return_edges)


def _skipgram(name, nodes, edges, starts, walks_per_node, length, context, p, q):
    return dict(name=name, kind="skipgram", nodes=nodes, edges=edges, starts=starts, walks_per_node=walks_per_node,
                length=length, context=context, p=p, q=q)


def _new_graph(name, nodes, edges, starts, length, p, q):
    return dict(name=name, kind="new_graph", nodes=nodes, edges=edges, starts=starts, length=length, p=p, q=q)


def _host(name, walk, nodes, edges, starts, length, p, q):
    return dict(name=name, kind="host", walk=walk, nodes=nodes, edges=edges, starts=starts, length=length, p=p, q=q)


def listed():
    return [
        # the reference's demo call: a citation-sized graph, 2,000 starts, five steps, its own rand array
        _uniform("uniform_demo", 2708, 5278, 2000, 5),
        # the node2vec demo: every node of that graph, 20 steps, nothing but the positional arguments
        _node2vec("node2vec_demo", 2708, 5278, 2708, 20, 0.5, 2.0),
        # one step of a node2vec training loop: 128 nodes, ten walks each, positive and negative windows of ten
        _skipgram("skipgram_batch", 2708, 5278, 128, 10, 20, 10, 1.0, 1.0),
        # a follower graph walked along its edges' direction, odd sizes, the edges wanted too (edge features)
        _uniform("uniform_directed_edges", 300007, 3000017, 200001, 33, directed=True, return_edges=True),
        # a middling graph, draws made in the kernel
        _uniform("uniform_kernel_draws", 1 << 20, 16 << 20, 1 << 20, 80, draws="kernel"),
        # the benchmark's uniform workload: a prepared graph, every node, 80 steps, the caller's rand array
        _uniform("uniform_rmat22", 1 << 22, 16 << 22, 1 << 22, 80, graph="fused"),
        # a graph that is not worth its hash set (or a device without room for one): binary searches
        _node2vec("node2vec_search", 500009, 5000011, 500009, 40, 1.0, 2.0, graph="search", directed=True),
        # the benchmark's light node2vec workload on a graph prepared with the hash set
        _node2vec("node2vec_rmat22_p1q2", 1 << 22, 16 << 22, 1 << 22, 40, 1.0, 2.0, graph="hash"),
        # the benchmark's headline: strong rejection on half a billion edges, the prepared graph of a long training
        _node2vec("node2vec_rmat24", 1 << 24, 16 << 24, 1 << 24, 80, 0.25, 4.0, graph="filter"),
        # the pairs of a whole epoch over a graph of 100,000 nodes
        _skipgram("skipgram_epoch", 100003, 1600033, 100003, 1, 40, 10, 1.0, 1.0),
        # edges arrive, are made a graph, and the graph is walked once from every node
        _new_graph("new_graph_rmat20", 1 << 20, 16 << 20, 1 << 20, 40, 0.5, 2.0),
        # numpy-side users: host arrays in, a host matrix out
        _host("host_node2vec", "node2vec", 262147, 4000037, 262147, 80, 0.25, 4.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("uniform", "uniform", "uniform", "node2vec", "node2vec", "node2vec", "node2vec", "skipgram", "skipgram",
                       "new_graph", "new_graph", "host", "host"))
    p, q = rng.choice(PQ)
    graph = {"uniform": rng.choice(("plain", "plain", "fused")),
             "node2vec": rng.choice(("plain", "search", "hash", "filter"))}.get(kind, "plain")
    most = 1 << {"host": 19, "new_graph": 21, "skipgram": 18}.get(kind, 20 if graph == "search" else 22)
    nodes = _log_int(rng, 1000, most)
    edges = int(nodes * rng.uniform(2.0, 16.0))
    starts = max(1, int(nodes * rng.choice((1.0, rng.random(), rng.random()))))
    length = _log_int(rng, 5, 100)
    if kind == "uniform":
        return _drop_name(_uniform("", nodes, edges, starts, min(length, 80), draws=rng.choice(("given", "given", "kernel")),
                                   graph=graph, directed=rng.random() < 0.3, return_edges=rng.random() < 0.2))
    if kind == "node2vec":
        return _drop_name(_node2vec("", nodes, edges, starts, min(length, 80), p, q, graph=graph,
                                    directed=graph != "filter" and rng.random() < 0.3, return_edges=rng.random() < 0.2))
    if kind == "skipgram":
        batch = min(starts, _log_int(rng, 64, 200000))
        walks = rng.choice((1, 5, 10)) if batch < 10000 else 1
        length = min(length, 60)
        return _drop_name(_skipgram("", nodes, edges, batch, walks, length, rng.randint(2, min(10, length)), p, q))
    if kind == "new_graph":
        return _drop_name(_new_graph("", nodes, edges, starts, min(length, 80), p, q))
    return _drop_name(_host("", rng.choice(("uniform", "node2vec", "node2vec")), nodes, edges, starts, length, p, q))


def _drop_name(case):
    del case["name"]
    return case


def _edge_list(case, seed, device):
    """``edges`` R-MAT edges over ``nodes`` ids, as an edge list arrives: repeats and loops among them."""
    scale = max(1, (case["nodes"] - 1).bit_length())
    factor = max(1, -(-case["edges"] // (1 << scale)))
    src, dst = graphs.rmat_edges(scale, factor, seed=seed, device=device)
    if src.numel() > case["edges"] or case["nodes"] != 1 << scale:
        # a prefix is as good a sample as the whole: the edges are drawn independently
        src, dst = ((t[:case["edges"]] * case["nodes"]) >> scale for t in (src, dst))
    return src, dst


def _starts(case, gen, device):
    """The epoch's nodes in random order (a batch is a part of them)."""
    return torch.randperm(case["nodes"], generator=gen, device=device)[:case["starts"]].contiguous()


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    state = {"case": case, "seed": seed}
    src, dst = _edge_list(case, seed, dev)
    start = _starts(case, gen, dev)
    if case["kind"] == "new_graph":
        state.update(src=src, dst=dst, start=start)
        return state
    rowptr, col = csr_from_edges(src, dst, case["nodes"], symmetrize=not case.get("directed", False))
    col = col.clone()  # the program keeps the trimmed array, not the buffer it was cut from
    del src, dst
    if case["kind"] == "skipgram":
        start = start.repeat(case["walks_per_node"])
    n, length = start.numel(), case["length"]
    if case["kind"] == "uniform" and case["draws"] == "given" or case.get("walk") == "uniform":
        state["rand"] = torch.rand((n, length), generator=gen, device=dev)
    if case["kind"] == "host":
        state.update({k: state[k].cpu() for k in ("rand",) if k in state})
        state.update(rowptr=rowptr.cpu(), col=col.cpu(), start=start.cpu())
        return state
    state.update(rowptr=rowptr, col=col, start=start)
    graph, undirected = case.get("graph", "plain"), not case.get("directed", False)
    if graph == "fused":
        state["graph"] = WalkGraph(rowptr, col, fused=True)
    elif graph == "hash":
        state["graph"] = WalkGraph(rowptr, col, symmetric=undirected, edgeset=True)
    elif graph == "filter":
        state["graph"] = WalkGraph(rowptr, col, symmetric=True, trifilter=True)
    return state


def run(state):
    case, seed = state["case"], state["seed"]
    kind, length = case["kind"], case["length"]
    if kind == "uniform":
        return random_walk(state["rowptr"], state["col"], state["start"], state.get("rand"), length, graph=state.get("graph"),
                           seed=seed, return_edges=case["return_edges"])
    if kind == "node2vec":
        return rejection_sampling(state["rowptr"], state["col"], state["start"], length, case["p"], case["q"], seed=seed,
                                  graph=state.get("graph"), edgeset=False if case["graph"] == "search" else "auto",
                                  return_edges=case["return_edges"])
    if kind == "skipgram":
        walks = rejection_sampling(state["rowptr"], state["col"], state["start"], length, case["p"], case["q"], seed=seed)
        negatives = negative_walks(state["start"], length, case["nodes"], seed=seed)
        return context_windows(walks, case["context"]), context_windows(negatives, case["context"])
    if kind == "new_graph":
        rowptr, col = csr_from_edges(state["src"], state["dst"], case["nodes"])
        graph = WalkGraph(rowptr, col, symmetric=True, edgeset=True)
        walks = rejection_sampling(rowptr, col, state["start"], length, case["p"], case["q"], seed=seed, graph=graph)
        return rowptr, walks  # (how many columns remain depends on the repeats in the list; the walks are made of them)
    if case["walk"] == "uniform":
        return random_walk(state["rowptr"], state["col"], state["start"], state["rand"], length)
    return rejection_sampling(state["rowptr"], state["col"], state["start"], length, case["p"], case["q"], seed=seed,
                              symmetric=True)


def work(case):
    """Each input read once and each output written once. Of the graph a pass needs no more than it visits: row bounds and one
    column entry, 24 bytes, per step, or the whole CSR where that is less."""
    n, length = case["starts"] * case.get("walks_per_node", 1), case["length"]
    steps = n * length
    entries = case["edges"] * (1 if case.get("directed", False) else 2)
    csr = 8 * (case["nodes"] + 1) + 8 * entries
    visited = min(24 * steps, csr)
    walks = 8 * n * (length + 1) + (8 * steps if case.get("return_edges", False) else 0)
    if case["kind"] == "skipgram":
        windows = n * (length + 2 - case["context"])
        return {"bytes": 8 * n + visited + 2 * 8 * windows * case["context"], "flops": 0}
    if case["kind"] == "new_graph":
        return {"bytes": 16 * case["edges"] + csr + 8 * n + walks, "flops": 0}
    rand = 4 * steps if case.get("draws") == "given" or case.get("walk") == "uniform" else 0
    # of host arrays the batch and the walk matrix cross the bus; the graph stays on the device from the first call on
    return {"bytes": 8 * n + rand + visited + walks, "flops": 0}


def tolerance(case):
    return "exact"
