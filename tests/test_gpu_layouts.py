"""Operand layouts and widths at which the product kernels change form: row groups of 1 - 16 lanes, the last
partial vector of a row, operands that are copied to aligned rows first, results whose rows are not aligned."""
import ctypes

import numpy as np
import pytest
import torch

from cbm4gnn_b200 import _lib, graphs
from cbm4gnn_b200.cbm import cbm_matrix
from helpers import chains, near_cliques, sparse_product, waiting_rows, with_self_loops

pytestmark = pytest.mark.gpu
TOL = dict(atol=1e-4, rtol=1e-4)


@pytest.fixture(scope="module", params=["split rows", "waiting rows"])
def copy_graph(request):
    """Split rows, and rows that wait in the tree but not in the product in one pass, which has them lifted; or a split row and
    a chain of rows that wait there too."""
    if request.param == "split rows":
        ei = with_self_loops(graphs.copy_model(3000, 0.9, 8, 11))
    else:
        rest = np.arange(500, 1100)
        ei = np.concatenate([chains(500, 1), np.stack([rest, rest]), np.stack([np.full(400, 500), np.arange(600, 1000)])], axis=1)
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=2, normalized=True)
    assert (np.diff(c._crow) > 192).any() and c.build_info["depth"] > 2  # split rows and waiting rows
    made = c.plan(0).schedule(columns=64)
    assert made["n_partial"] > 0 and (waiting_rows(c) > 300) == (request.param == "waiting rows")
    return ei, c


def _buffer(rows, width, pitch):
    return torch.full((rows, pitch), 7.0, device="cuda")[:, :width]


@pytest.mark.parametrize("f", [1, 3, 4, 5, 8, 9, 16, 17, 31, 33, 47, 64, 65, 100, 127, 129, 131, 257])
@pytest.mark.parametrize("aligned_x,aligned_y", [(True, True), (True, False), (False, True), (False, False)])
def test_widths_and_pitches(copy_graph, f, aligned_x, aligned_y):
    ei, c = copy_graph
    x = np.random.default_rng(f).standard_normal((c.num_rows, f)).astype(np.float32)
    up = -(-f // 4) * 4
    xd = _buffer(c.num_rows, f, up if aligned_x else up + 1)
    yd = _buffer(c.num_rows, f, up if aligned_y else up + 1)
    xd.copy_(torch.from_numpy(x))
    want = sparse_product(ei, x, True)
    c.omp_mkl_csr_fused_spmm_update(xd, yd)
    c.plan(0).status()
    np.testing.assert_allclose(yd.cpu().numpy(), want, **TOL)
    if up != f or not aligned_y:  # nothing is written beside the result's columns
        pad = yd.as_strided((c.num_rows, yd.stride(0) - f), (yd.stride(0), 1), f)
        assert torch.equal(pad, torch.full_like(pad, 7.0))
    two = torch.full_like(yd, 7.0)
    c.seq_mkl_csr_spmm(xd, two)
    c.seq_mkl_csr_fused_update(two)
    np.testing.assert_allclose(two.cpu().numpy(), want, **TOL)
    torch.testing.assert_close(c.seq_torch_csr_fused_matmul(xd), yd, atol=0, rtol=1e-6)


@pytest.fixture(scope="module", params=[2, 40, "near cliques"])
def community_graph(request):
    """Enough rows with common columns that the plan works on them community by community (16 384 and more); with 40
    expected links per node rows also share a parent, so that some of them wait in the tree; near cliques' rows wait in the
    product in one pass too."""
    n = 16384 + 5
    if request.param == "near cliques":
        ei = near_cliques(n, 80, 0.1, 5)
    else:
        ei = with_self_loops(graphs.stochastic_block_model(n, 400, 3.5, 0.8, 8.0 if request.param == 2 else 40.0, 1.0, 5))
    ei = np.concatenate([ei, [[7] * 700, list(range(1000, 1700))]], axis=1)  # one row that is split
    key = np.unique(ei[0] * n + ei[1])
    ei = np.stack([key // n, key % n])
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=2, normalized=True)
    made = c.plan(0).schedule()
    assert made["n_chunks"] > 0 and made["n_partial"] > 0 and made["n_items"] > made["n_prefix"]
    assert request.param == 2 or c.build_info["depth"] > 1
    in_one_pass = c.plan(0).schedule(columns=64)
    assert in_one_pass["n_chunks"] > 0 and (waiting_rows(c) > 8000) == (request.param == "near cliques")
    return ei, c


@pytest.mark.parametrize("f", [5, 16, 61, 64, 65, 100, 128, 129, 200])
@pytest.mark.parametrize("pad", [0, 1, 3])
def test_rows_in_community_order(community_graph, f, pad):
    ei, c = community_graph
    x = np.random.default_rng(f).standard_normal((c.num_rows, f)).astype(np.float32)
    xd, yd = _buffer(c.num_rows, f, f + pad), _buffer(c.num_rows, f, f + pad)
    xd.copy_(torch.from_numpy(x))
    want = sparse_product(ei, x, True)
    for _ in range(2):
        c.omp_mkl_csr_fused_spmm_update(xd, yd)
    c.plan(0).status()
    np.testing.assert_allclose(yd.cpu().numpy(), want, **TOL)
    two = torch.full_like(yd, 7.0)
    c.seq_mkl_csr_spmm(xd, two)
    c.seq_mkl_csr_fused_update(two)
    np.testing.assert_allclose(two.cpu().numpy(), want, **TOL)
    own, sent = _buffer(c.num_rows, f, f + pad), _buffer(c.num_rows, f, f + pad)
    _deliver(c, xd, own, sent, relu=True)
    assert torch.equal(own, yd) and torch.equal(sent, yd.relu())


def _deliver(c, x, y, to, relu=False):
    """The product with its rows also stored to a further buffer."""
    _lib.check(_lib.lib().cbm_b200_spmm_update_bcast(
        c.plan(0).handle, x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), x.size(1), 1, int(relu), 1,
        (ctypes.c_void_p * 1)(to.data_ptr()), torch.cuda.current_stream().cuda_stream))


@pytest.fixture(scope="module")
def many_rows():
    """So many rows that wait for nobody that a warp claims several (256 for each SM and more): narrow ones are then
    worked on side by side."""
    ei = with_self_loops(graphs.copy_model(45000, 0.6, 4, 3))
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=8, normalized=True, build_device=0)
    length = np.diff(c._crow)
    made = c.plan(0).schedule()
    assert made["n_chunks"] == 0 and made["n_prefix"] - made["n_partial"] > 37888 and (length > 192).any()
    return ei, c


@pytest.mark.parametrize("f", [3, 13, 17, 29, 32, 33, 47, 61, 64])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_rows_side_by_side(many_rows, f, pad):
    """Narrow rows: right, and with the same bits whether several share a warp (the product) or each has its own
    (delivery to further buffers)."""
    ei, c = many_rows
    n, pitch = c.num_rows, -(-f // 4) * 4 + pad
    x = np.random.default_rng(f).standard_normal((n, f)).astype(np.float32)
    xd, yd, own, sent = (_buffer(n, f, pitch) for _ in range(4))
    xd.copy_(torch.from_numpy(x))
    c.omp_mkl_csr_fused_spmm_update(xd, yd)
    _deliver(c, xd, own, sent)
    c.plan(0).status()
    np.testing.assert_allclose(yd.cpu().numpy(), sparse_product(ei, x, True), **TOL)
    assert torch.equal(own, yd) and torch.equal(sent, yd)
    pad_of = yd.as_strided((n, pitch - f), (pitch, 1), f)
    assert torch.equal(pad_of, torch.full_like(pad_of, 7.0))


@pytest.mark.parametrize("n,mu,deg_in", [(60_000, 3.5, 12.0), (200_000, 4.0, 8.0)])
def test_plans_of_one_graph_are_the_same(n, mu, deg_in):
    ei = with_self_loops(graphs.stochastic_block_model(n, n // 50, mu, 0.8, deg_in, 3.0, 5))
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=2, normalized=True, build_device=0)
    first, in_one_pass = c.plan(0).schedule(), c.plan(0).schedule(columns=64)
    assert first["n_chunks"] > 0  # rows in the order of communities found on the GPU
    assert in_one_pass["n_chunks"] > 0 and in_one_pass["fingerprint"] != first["fingerprint"]  # (with rows lifted)
    for _ in range(4):
        c._plans.clear()
        assert c.plan(0).schedule() == first and c.plan(0).schedule(columns=64) == in_one_pass


@pytest.mark.parametrize("rows,f,aligned,slab", [(4, 1_000_000, True, 0), (4, 909_312, True, 0), (4, 909_440, True, 0), (6, 300_000, False, 0),
                                                 (3, 227_328, False, 0), (3, 227_392, False, 0), (5, 230_000, True, 32)])
def test_more_slabs_than_warps(rows, f, aligned, slab):
    """Few rows by so many columns that there are more column slabs than resident warps (7 104 of 128 columns on 148 SMs,
    3 552 of 64 where rows are not aligned), and just as many."""
    ei = np.stack([np.repeat(np.arange(rows), rows), np.tile(np.arange(rows), rows)])
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=100, normalized=True)
    if slab:
        c.plan(0).tune(slab_width=slab)
    x = np.random.default_rng(f).standard_normal((rows, f)).astype(np.float32)
    xd, yd = _buffer(rows, f, f if aligned else f + 1), _buffer(rows, f, f if aligned else f + 1)
    xd.copy_(torch.from_numpy(x))
    c.omp_mkl_csr_fused_spmm_update(xd, yd)
    c.plan(0).status()
    np.testing.assert_allclose(yd.cpu().numpy(), sparse_product(ei, x, True), **TOL)


@pytest.fixture(scope="module")
def waiting_chains():
    """So many waiting rows (a quarter of the resident warps and more) that claims are drawn in more than one round, and one
    row that is split."""
    ei = chains(400, 7)
    rest = np.arange(2800, 3400)
    ei = np.concatenate([ei, np.stack([rest, rest]), np.stack([np.full(400, 2800), np.arange(2900, 3300)])], axis=1)
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=2, normalized=True)
    assert waiting_rows(c) > 1776 and c.plan(0).schedule(columns=64)["n_partial"] > 0
    return ei, c


@pytest.mark.parametrize("slab,form", [(0, 0), (64, 0), (256, 0), (512, 0), (0, 1)])
@pytest.mark.parametrize("f,pad", [(512, 0), (512, 1), (515, 0), (40, 0)])
def test_every_form_waits(waiting_chains, slab, form, f, pad):
    """One, two and four vectors or values a lane, aligned and not, bulk copies, and the allocation-free product."""
    ei, c = waiting_chains
    x = np.random.default_rng(f).standard_normal((c.num_rows, f)).astype(np.float32)
    xd, yd, static = (_buffer(c.num_rows, f, f + pad) for _ in range(3))
    xd.copy_(torch.from_numpy(x))
    c.plan(0).tune(slab_width=slab, form=form)
    try:
        c.omp_mkl_csr_fused_spmm_update(xd, yd)
        _lib.check(_lib.lib().cbm_b200_spmm_update_static(c.plan(0).handle, xd.data_ptr(), f + pad, static.data_ptr(), f + pad, f, 1,
                                                          torch.cuda.current_stream().cuda_stream))
        c.plan(0).status()
    finally:
        c.plan(0).tune()
    np.testing.assert_allclose(yd.cpu().numpy(), sparse_product(ei, x, True), **TOL)
    torch.testing.assert_close(static, yd, **TOL)


@pytest.mark.parametrize("n,p_copy,links,by_tree_from", [(3000, 0.95, 20, 500), (6000, 0.9, 8, 1024), (4096, 0.8, 3, None)])
def test_wide_products_go_by_the_tree_where_it_saves_much(n, p_copy, links, by_tree_from):
    ei = with_self_loops(graphs.copy_model(n, p_copy, links, 3))
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=4, normalized=True, build_device=0)
    tree, narrow = c.plan(0).schedule(), c.plan(0).schedule(columns=128)
    assert tree != narrow and waiting_rows(c) < (c._parent != c.num_rows).sum()
    for f in (128, 500, 1024):
        goes_by = c.plan(0).schedule(columns=f)
        assert goes_by == (tree if by_tree_from is not None and f >= by_tree_from else narrow)
        x = torch.randn((c.num_rows, f), generator=torch.Generator(device="cuda").manual_seed(f), device="cuda")
        y, own, sent, static = (torch.full_like(x, float("nan")) for _ in range(4))
        c.omp_mkl_csr_fused_spmm_update(x, y)
        _deliver(c, x, own, sent)
        rc = _lib.lib().cbm_b200_spmm_update_static(c.plan(0).handle, x.data_ptr(), f, static.data_ptr(), f, f, 1,
                                                    torch.cuda.current_stream().cuda_stream)
        c.plan(0).status()
        np.testing.assert_allclose(y.cpu().numpy(), sparse_product(ei, x.cpu().numpy(), True), **TOL)
        assert torch.equal(own, y) and torch.equal(sent, y)
        if rc == 0:
            torch.testing.assert_close(static, y, **TOL)
        else:
            assert b"bytes of scratch" in _lib.lib().cbm_b200_last_error()
