"""Kernels whose blocks are set up while the one before them on the stream is ending (cbm_launch.cuh) see all of what it
wrote: a chain of calls issued in one go gives the bits of the same calls waited for one by one."""
import numpy as np
import pytest
import torch

from cbm4gnn_b200 import dense, graphs
from cbm4gnn_b200.cbm import cbm_matrix
from helpers import chains, near_cliques, waiting_rows, with_self_loops

pytestmark = pytest.mark.gpu


def _chain(c, f, after):
    """Products there and back between the same two buffers, whose rows share cache lines where `f` is odd, the operand
    changed by torch's kernels too; maps, their gradients and the sum of its parts behind them."""
    gen = torch.Generator(device="cuda").manual_seed(f)
    x, y = torch.randn((2, c.num_rows, f), generator=gen, device="cuda")
    w = torch.randn((f, f), generator=gen, device="cuda") / f ** 0.5
    seen = []
    for _ in range(4):
        c.omp_mkl_csr_fused_spmm_update(x, y)
        after()
        c.omp_mkl_csr_fused_spmm_update(y, x)
        after()
        h = dense.dense_forward(x, w)
        after()
        g = dense.dense_grad_weight(h, y)
        after()
        gx = dense.dense_grad_input(h, g / g.norm(), relu_output=x)
        after()
        x.copy_(gx).div_(gx.norm())
        after()
        w = w + g / g.norm()
        after()
        seen += [h, g, gx, y.clone()]
    return seen


# kind of graph: rows, whether rows wait for a parent in the product in one pass, whether the plan is in community order
KINDS = {"split rows": (3000, False, False), "few communities": (11793, False, False), "chains": (2800, True, False),
         "communities": (70_000, False, True), "near cliques": (17_000, True, True)}


@pytest.fixture(scope="module", params=KINDS)
def matrix(request):
    ei = {"split rows": lambda: graphs.copy_model(3000, 0.9, 8, 11), "few communities": lambda: graphs.make_graph("c3", scale=0.05),
          "chains": lambda: chains(400, 7), "communities": lambda: graphs.stochastic_block_model(70_000, 1400, 3.5, 0.8, 12.0, 3.0, 5),
          "near cliques": lambda: near_cliques(17_000, 80, 0.1, 5)}[request.param]()
    ei = ei if KINDS[request.param][1] else with_self_loops(ei)
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=2, normalized=True, build_device=0)
    made, (rows, waits, clustered) = c.plan(0).schedule(columns=64), KINDS[request.param]
    assert c.num_rows == rows and (made["n_chunks"] > 0) == clustered
    # Rows that wait: the normalized wait; in community order, on up to 65 536 rows or from 65 columns on: the chunk kernel's.
    assert (waiting_rows(c) > 1000) == waits
    # Up to 64 columns, more than 65 536 rows and 256 for each of 148 SMs that never wait: the staged narrow kernel.
    assert request.param != "communities" or rows > 65_536 and made["n_prefix"] - made["n_partial"] >= 37_888
    return c


# widths: row groups of a few lanes, two odd pitches (the operand is copied to aligned rows first), whole slabs, several
@pytest.mark.parametrize("f", [8, 33, 47, 64, 128, 260])
def test_calls_in_one_go_give_the_bits_of_calls_one_by_one(matrix, f):
    want = _chain(matrix, f, torch.cuda.synchronize)
    got = _chain(matrix, f, lambda: None)
    matrix.plan(0).status()
    assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(bool(torch.isfinite(a).all()) for a in got)


def test_captured_branches_that_join(matrix):
    """A product and a map on two branches of a captured graph, and a map of both behind the join."""
    x, y = torch.randn((2, matrix.num_rows, 64), device="cuda")
    w = torch.randn((64, 64), device="cuda")
    side = torch.cuda.Stream()

    def work():
        here = torch.cuda.current_stream()
        matrix.omp_mkl_csr_fused_spmm_update(x, y)
        side.wait_stream(here)
        with torch.cuda.stream(side):
            a = dense.dense_forward(x, w)
        b = dense.dense_forward(y, w)
        here.wait_stream(side)
        return dense.dense_grad_weight(a, b)

    first = torch.cuda.Stream()
    with torch.cuda.stream(first):  # workspaces grow outside the capture
        want = work().clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = work()
    x.mul_(2)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    assert np.isfinite(float(want.norm()))
    assert torch.equal(got, want * 4)  # (of powers of two, nothing is rounded)


def test_first_product_of_a_plan_may_be_a_captured_one():
    """Two column slabs of rows that park no sums by the tree: 100 roots of 60 entries, children with 50 more, 1 000 short
    rows.  Lifted, the children are cut in two and would need more workspace than a plan begins with."""
    roots, short = 100, 1000
    n = 2 * roots + short
    mst_row = np.full(n + 2, roots, np.int32)
    mst_row[:roots + 1] = np.arange(roots + 1)
    mst_row[n + 1] = n
    mst_col = np.concatenate([np.arange(roots, 2 * roots), np.arange(roots), np.arange(2 * roots, n)]).astype(np.int32)
    rows = [np.arange(60) + i for i in range(roots)] + [np.arange(60, 110) + i for i in range(roots)] + [np.arange(3) + i for i in range(short)]
    crow = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    c = cbm_matrix.from_arrays(mst_row, mst_col, crow, col, np.ones(len(col), np.float32))
    x = torch.randn((n, 256), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    y = torch.empty_like(x)
    c.plan(0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c.omp_mkl_csr_spmm_update(x, y)
    graph.replay()
    c.plan(0).status()
    want = torch.stack([x.double()[torch.from_numpy(r).cuda()].sum(0) for r in rows])
    want[roots:2 * roots] += want[:roots]
    torch.testing.assert_close(y.double(), want, atol=1e-4, rtol=1e-4)


@pytest.mark.parametrize("f", [16, 64, 256])
@pytest.mark.parametrize("entry", ["spmm_update", "update"])
def test_a_captured_product_waits_in_every_replay(entry, f):
    """A chain of rows, each of which waits for the one before: replays see their own launch's rows, not those that the
    replay before left."""
    n = 1500
    ei = np.stack([np.repeat(np.arange(n), np.arange(1, n + 1)), np.concatenate([np.arange(i + 1) for i in range(n)])])
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=0)
    x = torch.randn((n, f), generator=torch.Generator(device="cuda").manual_seed(f), device="cuda")
    y = torch.empty_like(x)

    def work():
        if entry == "update":
            c.seq_mkl_csr_spmm(x, y)
            c.omp_mkl_csr_update(y)
        else:
            c.omp_mkl_csr_spmm_update(x, y)

    work()  # workspaces grow outside the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    for scale in (1.0, -2.0, 0.5):
        x.mul_(scale)
        for _ in range(2):
            y.fill_(float("nan"))
            graph.replay()
            got = y.clone()
            work()
            c.plan(0).status()
            assert torch.equal(got, y)
        torch.testing.assert_close(got.double(), x.double().cumsum(0), atol=1e-3, rtol=1e-4)  # (sums of up to 1 500)


def test_a_captured_product_outlives_the_growth_of_its_workspaces():
    """Wider products of the plan replace its flags, parked sums and the operand's aligned copy; a graph goes on with those it
    was captured with."""
    ei = with_self_loops(graphs.copy_model(3000, 0.95, 20, 77))
    c = cbm_matrix(torch.from_numpy(ei).to(torch.int32), torch.ones(ei.shape[1]), alpha=4, normalized=True, build_device=0)
    gen = torch.Generator(device="cuda").manual_seed(2)
    x, y = torch.randn((2, c.num_rows, 301), generator=gen, device="cuda")  # (copied to aligned rows first)
    c.omp_mkl_csr_fused_spmm_update(x, y)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c.omp_mkl_csr_fused_spmm_update(x, y)
    for f in (1001, 2003):
        wide, out = torch.randn((2, c.num_rows, f), generator=gen, device="cuda")
        c.omp_mkl_csr_fused_spmm_update(wide, out)
        x.mul_(-0.5)
        y.fill_(float("nan"))
        graph.replay()
        again = torch.empty_like(out)
        c.omp_mkl_csr_fused_spmm_update(wide, again)
        want = torch.empty_like(y)
        c.omp_mkl_csr_fused_spmm_update(x, want)
        c.plan(0).status()
        assert torch.equal(y, want) and torch.equal(out, again)
