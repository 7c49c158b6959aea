"""The allocation-free product entry point against the ordinary one.

``cbm_b200_spmm_update_static`` exists for callers that may not allocate device memory while they
run (all memory handed to their own pool, a stream capture in progress, a latency budget that an
allocation's device synchronisation would break).  It runs the same kernel as the ordinary entry
points but keeps its ready flags and partial sums in a fixed array inside the library, which is
shared between calls and keeps the previous call's contents.  The test therefore makes two calls in
a row, with different operands and a plan that has long rows (so partial sums are in play), and
requires each to reproduce the ordinary entry point exactly (both run the same arithmetic in the
same order) and to agree with an independent float64 CSR product of the same matrix.  The file name sorts last so that a run that stops at the first failure has already
exercised everything else.
"""
import ctypes

import numpy as np
import pytest
import torch

from cbm4gnn_b200 import _lib, graphs
from cbm4gnn_b200.cbm import cbm_matrix
from cbm4gnn_b200.utility import add_self_loops

pytestmark = pytest.mark.gpu


def _call(fn, plan, x, y, f, *extra):
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(fn(plan.handle, x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), f, *extra, stream))


def test_static_scratch_product_matches_twice_in_a_row():
    L = _lib.lib()
    ei = add_self_loops(torch.from_numpy(graphs.make_graph("c1")))
    c = cbm_matrix(ei.to(torch.int32), torch.ones(ei.shape[1]), alpha=0, normalized=True)
    assert int(np.diff(c._crow).max()) > 192       # some rows are cut into segments
    plan = c.plan(torch.cuda.current_device())
    n = c.num_rows
    gen = torch.Generator(device="cuda").manual_seed(7)
    import scipy.sparse as sp
    e = ei.numpy()
    a64 = sp.csr_matrix((np.ones(e.shape[1]), (e[0], e[1])), shape=(n, n))
    s = np.asarray(a64.sum(1)).ravel() ** -0.5
    a64_norm = sp.diags(s) @ a64 @ sp.diags(s)
    for normalized, f in ((1, 500), (0, 64)):
        x = torch.randn((n, f), device="cuda", generator=gen)
        want = torch.empty((n, f), device="cuda")
        _call(L.cbm_b200_fused_spmm_update if normalized else L.cbm_b200_spmm_update, plan, x, want, f)
        got = torch.full((n, f), float("nan"), device="cuda")
        _call(L.cbm_b200_spmm_update_static, plan, x, got, f, normalized)
        plan.status()
        torch.testing.assert_close(got, want, atol=1e-4, rtol=1e-4)
        assert torch.equal(got, want)
        # and both against an independent float64 CSR product of the same matrix
        # the plan carries the normalized structure (delta values +-s_col): without the row
        # scales of the fused form it computes A D^-1/2 x
        ref = a64_norm if normalized else a64 @ sp.diags(s)
        np.testing.assert_allclose(got.cpu().numpy(), ref @ x.cpu().numpy().astype(np.float64), atol=1e-4, rtol=1e-4)


def test_static_scratch_rejects_oversized_products():
    L = _lib.lib()
    # nested rows: row i holds columns 0..i, so one row alone has far more than 192 entries and
    # the operand is wide: the partial sums do not fit the fixed array
    n = 4000
    rows = np.repeat(np.arange(n), np.arange(1, n + 1))
    cols = np.concatenate([np.arange(i + 1) for i in range(n)])
    c = cbm_matrix(torch.from_numpy(np.stack([rows, cols])).to(torch.int32), torch.ones(rows.size), alpha=100000)
    plan = c.plan(torch.cuda.current_device())
    f = 1024
    x = torch.zeros((n, f), device="cuda")
    y = torch.zeros((n, f), device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = L.cbm_b200_spmm_update_static(plan.handle, x.data_ptr(), f, y.data_ptr(), f, f, 0, stream)
    assert rc == 1
    msg = L.cbm_b200_last_error().decode()
    assert "bytes of scratch" in msg and str(8 << 20) in msg


def _hubs_on_blocks():
    """470 000 short rows, which leave little of the fixed array, and 20 of 2 000 entries."""
    n = 470_000
    rng = np.random.default_rng(3)
    ei = graphs.stochastic_block_model(n, n // 50, 3.5, 0.8, 3.0, 1.0, 5)
    hub = np.repeat(np.arange(20) * 1000, 2000)
    key = np.unique(np.concatenate([ei[0] * n + ei[1], hub * n + rng.integers(0, n, hub.size), np.arange(n) * (n + 1)]))
    return np.stack([key // n, key % n])


@pytest.mark.parametrize("make,alpha", [(lambda: add_self_loops(torch.from_numpy(graphs.copy_model(50_000, 0.7, 5, 3))).numpy(), 8),
                                        (_hubs_on_blocks, 2)])
def test_what_is_refused_does_not_depend_on_how_finely_rows_are_cut(make, alpha):
    """Parked sums that do not all fit the fixed array are those of the longest rows; as long as a schedule with rows cut at
    192 entries would fit, the product runs, with the ordinary entry point's bits."""
    L = _lib.lib()
    ei = torch.from_numpy(make())
    c = cbm_matrix(ei.to(torch.int32), torch.ones(ei.shape[1]), alpha=alpha, normalized=True, build_device=0)
    plan, n = c.plan(0), c.num_rows
    made, length = plan.schedule(), np.diff(c._crow)
    coarse = int((-(-length[length > 192] // 128) - 1).sum())
    assert made["segment"] == 64 and 0 < coarse < made["n_partial"]
    gen = torch.Generator(device="cuda").manual_seed(7)
    for f, pad in ((500, 0), (500, 4), (497, 3), (499, 0), (480, 0), (401, 0)):
        slabs, unaligned, odd = -(-f // 128), (f + pad) % 4 != 0, f % 4 != 0 or (f + pad) % 4 != 0
        assert 4 * slabs * (n + coarse + 128 * coarse) < 8 << 20 < 4 * slabs * (n + made["n_partial"] * 129)
        x = torch.randn((n, f + pad), device="cuda", generator=gen)[:, :f]
        want, got = (torch.full((n, f + pad), float("nan"), device="cuda")[:, :f] for _ in range(2))
        rc = L.cbm_b200_spmm_update_static(plan.handle, x.data_ptr(), f + pad, got.data_ptr(), f + pad, f, 1,
                                           torch.cuda.current_stream().cuda_stream)
        if odd and n > 400_000:  # counted in slabs of 64 columns: more flags than room
            assert rc == 1 and b"bytes of scratch" in L.cbm_b200_last_error()
            continue
        _lib.check(rc)
        _call(L.cbm_b200_fused_spmm_update, plan, x, want, f)
        plan.status()
        # an unaligned operand of this size is copied to aligned rows by the ordinary entry point, and its sums are added
        # in another order where the last slab is narrow: within fp32 rounding of the longest row
        torch.testing.assert_close(got, want, atol=0 if not unaligned else 1e-5, rtol=0 if not unaligned else 1e-5)


@pytest.mark.parametrize("f", [16, 64, 128])
def test_more_claims_by_the_lifted_rows_than_by_the_tree(f):
    """37 000 rows and 1 500 children that are lifted: by the tree one round of claims does (fewer than 256 rows for each of
    148 SMs wait for nobody), as the product goes there are more."""
    L = _lib.lib()
    roots, children = 37_000, 1_500
    n = roots + children
    mst_row = np.full(n + 2, children, np.int32)
    mst_row[:children + 1] = np.arange(children + 1)
    mst_row[n + 1] = n
    mst_col = np.concatenate([np.arange(roots, n), np.arange(roots)]).astype(np.int32)
    crow = np.concatenate([[0], np.cumsum(np.where(np.arange(n) < roots, 3, 2))]).astype(np.int32)
    col = np.concatenate([(np.arange(roots)[:, None] + [0, 1, 2]).ravel(), (np.arange(children)[:, None] + [3, 4]).ravel()])
    c = cbm_matrix.from_arrays(mst_row, mst_col, crow, col.astype(np.int32), np.ones(len(col), np.float32))
    x = torch.randn((n, f), generator=torch.Generator(device="cuda").manual_seed(f), device="cuda")
    y = torch.full((n, f), float("nan"), device="cuda")
    want = x.double()[:roots] + x.double()[1:roots + 1] + x.double()[2:roots + 2]
    want = torch.cat([want, want[:children] + x.double()[3:children + 3] + x.double()[4:children + 4]])
    for _ in range(2):
        _call(L.cbm_b200_spmm_update_static, c.plan(0), x, y.fill_(float("nan")), f, 0)
        c.plan(0).status()
        torch.testing.assert_close(y.double(), want, atol=1e-5, rtol=1e-5)  # (sums of five)
