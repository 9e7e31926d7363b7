"""The per-edge structures of a graph against numpy: reverse positions (directed, symmetric, loops, edges without a reverse,
hubs beside short rows, isolated nodes, edge counts around a warp's chunk) and the edge hash set's members."""
import numpy as np
import pytest
import torch

from mlx_cluster_b200 import _lib
from mlx_cluster_b200.ops import WalkGraph

pytestmark = pytest.mark.gpu


def _csr(nodes, pairs):
    pairs = np.unique(pairs, axis=0)
    rowptr = np.zeros(nodes + 1, dtype=np.int64)
    np.cumsum(np.bincount(pairs[:, 0], minlength=nodes), out=rowptr[1:])
    return rowptr, pairs


def _reverse_positions(nodes, pairs):
    key = pairs[:, 0] * nodes + pairs[:, 1]
    back = pairs[:, 1] * nodes + pairs[:, 0]
    at = np.minimum(np.searchsorted(key, back), len(key) - 1)
    return np.where(key[at] == back, at, 0xffffffff)


def _members(table):
    table = table.cpu().numpy().view(np.uint64)
    return np.sort(table[table != np.uint64(0xffffffffffffffff)])


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("nodes,edges", [(1, 1), (3, 4), (40, 255), (40, 257), (5000, 2600), (70000, 300000), (33, 1000)])
def test_reverse_positions_and_edge_set(cuda, nodes, edges, symmetric):
    rng = np.random.default_rng(nodes + edges)
    skew = (rng.random((edges, 2)) ** 3 * nodes).astype(np.int64)  # hubs at the low ids, isolated nodes at the high ones
    pairs = np.concatenate([skew, skew[:, ::-1]]) if symmetric else skew
    rowptr, pairs = _csr(nodes, pairs)
    graph = WalkGraph(torch.from_numpy(rowptr).to(cuda), torch.from_numpy(pairs[:, 1].copy()).to(cuda), edgeset=True)
    joined = graph.colrev.cpu().numpy().view(np.uint64)
    np.testing.assert_array_equal(joined & np.uint64(0xffffffff), pairs[:, 1].astype(np.uint64))
    np.testing.assert_array_equal((joined >> np.uint64(32)).astype(np.int64), _reverse_positions(nodes, pairs))
    np.testing.assert_array_equal(_members(graph.edgeset),
                                  np.sort(pairs[:, 0].astype(np.uint64) << np.uint64(32) | pairs[:, 1].astype(np.uint64)))


def test_unsorted_rows_are_seen(cuda):
    rowptr = np.array([0, 300, 300, 600], dtype=np.int64)
    col = np.concatenate([np.arange(300), np.arange(300)]) % 3
    graph = WalkGraph(torch.from_numpy(rowptr).to(cuda), torch.from_numpy(col).to(cuda), edgeset=True)
    assert graph.rows_sorted is False and graph.colrev is None
    ok = np.array([0, 1, 2], dtype=np.int64)
    graph = WalkGraph(torch.tensor([0, 3, 3, 3]).to(cuda), torch.from_numpy(ok).to(cuda), edgeset=True)
    assert graph.rows_sorted is True and graph.colrev is not None
    assert _lib.last_kernel() == "colrev_build_kernel"
