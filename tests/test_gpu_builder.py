"""The builder's candidate search on the GPU against the host search: same candidates, hence
byte-identical structures (tree arrays, delta CSR), on graphs of every shape the host tests use."""
import numpy as np
import pytest
import torch

from cbm4gnn_b200 import graphs
from cbm4gnn_b200.cbm import cbm_matrix
from helpers import with_self_loops

pytestmark = pytest.mark.gpu


def _both(ei, alpha, normalized=False):
    e = torch.from_numpy(np.ascontiguousarray(ei)).to(torch.int32)
    ones = torch.ones(e.shape[1])
    host = cbm_matrix(e, ones, alpha=alpha, normalized=normalized)
    gpu = cbm_matrix(e, ones, alpha=alpha, normalized=normalized, build_device=torch.cuda.current_device())
    assert gpu.build_info["candidates_on_gpu"] is True and host.build_info["candidates_on_gpu"] is False
    assert gpu.build_info["n_candidates"] == host.build_info["n_candidates"]
    assert torch.equal(host.mst_row, gpu.mst_row) and torch.equal(host.mst_col, gpu.mst_col)
    for a, b in ((host._crow, gpu._crow), (host._dcol, gpu._dcol), (host._dval, gpu._dval), (host._parent, gpu._parent)):
        assert np.array_equal(a, b)
    return host, gpu


@pytest.mark.parametrize("alpha", [0, 1, 3, 8, 64])
def test_copy_model_graphs(alpha):
    _both(graphs.make_graph("c1"), alpha)
    _both(with_self_loops(graphs.make_graph("c2", scale=0.2)), alpha, normalized=True)


@pytest.mark.parametrize("alpha", [0, 4, 16])
def test_high_similarity_graph(alpha):
    host, _ = _both(with_self_loops(graphs.copy_model(6000, 0.95, 20, 77)), alpha, normalized=True)
    assert host.build_info["n_delta"] < host.nnz


def test_small_random_and_block_model_graphs():
    for seed in range(6):
        _both(graphs.erdos_renyi(40 + seed, 0.3, seed), seed % 3)
    _both(with_self_loops(graphs.make_graph("c3", scale=0.05)), 2, normalized=True)


def test_nested_rows_with_long_prefixes():
    """Row i = {0..i}: every pair of rows intersects and the tree is one chain."""
    n = 700
    rows = np.repeat(np.arange(n), np.arange(1, n + 1))
    cols = np.concatenate([np.arange(i + 1) for i in range(n)])
    host, _ = _both(np.stack([rows, cols]), 0)
    assert host.build_info["depth"] == n


def test_negative_alpha_and_directed_pattern():
    rng = np.random.default_rng(3)
    mask = rng.random((120, 120)) < 0.2
    np.fill_diagonal(mask, True)
    ei = np.stack(np.nonzero(mask))
    for alpha in (-3, 0, 5):
        _both(ei, alpha, normalized=True)


def test_config4_full_size_on_the_gpu():
    """The high-degree configuration at full size: identical structure.  (Measured: the search takes
    9 s on 16 host threads and 2 s through the GPU; no timing is asserted, host core counts vary.)"""
    ei = with_self_loops(graphs.make_graph("c4"))
    host, gpu = _both(ei, 4, normalized=True)
    assert gpu.build_info["seconds_candidates"] < 30.0


@pytest.mark.parametrize("lengths", [(1, 2, 31, 32, 33, 64, 255, 256, 257), (511, 512, 513, 4095, 4096, 4097, 5000, 9000)])
def test_rows_at_the_edges_of_the_sorts(lengths):
    """Rows as long as a warp's registers, a warp's and a block's shared memory hold, one more and one less, each with a near
    copy that can be its child."""
    n = 9000
    rng = np.random.default_rng(sum(lengths))
    pattern = [rng.integers(0, n, 3) for _ in range(n)]
    for i, length in enumerate(lengths):
        pattern[2 * i] = rng.choice(n, length, replace=False)
        pattern[2 * i + 1] = np.concatenate([pattern[2 * i][: max(1, length - 2)], rng.integers(0, n, 2)])
    key = np.unique(np.concatenate([v * n + p for v, p in enumerate(pattern)] + [np.array([n * n - 1])]))
    host, _ = _both(np.stack([key // n, key % n]), 0)
    assert host.build_info["depth"] > 1


@pytest.mark.parametrize("group", [18, 29, 30, 31, 32, 33, 60])
def test_parents_at_the_edge_of_a_warps_table(group):
    """Groups of like rows whose prefixes list just as many rows as a warp counts in shared memory (704), some fewer and
    some more (23 columns of 29 - 33 rows each); with 60 rows to a group all go to the blocks."""
    rng = np.random.default_rng(group)
    rows = []
    for g in range(40):
        common = np.arange(40) + 40 * g
        rows += [np.delete(common, rng.integers(0, 40, rng.integers(0, 3))) for _ in range(group + g % 2)]
    n = max(len(rows), 1600)  # (40 groups of 40 columns)
    key = np.unique(np.concatenate([v * n + r for v, r in enumerate(rows)]))
    host, _ = _both(np.stack([key // n, key % n]), 0)
    assert host.build_info["depth"] > 2
