"""Host builder of the product (libcbm_b200.so) against the restated builder and its invariants."""
import ctypes

import numpy as np
import pytest
import torch

from cbm4gnn_b200 import _lib, graphs
from cbm4gnn_b200.cbm import cbm_matrix
from oracle import cbm_oracle as orc
from helpers import with_self_loops


def _cbm(ei, alpha=0, normalized=False):
    e = torch.from_numpy(ei).to(torch.int32)
    return cbm_matrix(e, torch.ones(e.shape[1]), alpha=alpha, normalized=normalized)


@pytest.mark.parametrize("alpha", [1, 2, 3, 4])   # the values tests/test_cbm_creation.py:31-39 sweeps
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_structure_valid_and_optimal(seed, alpha):
    ei = graphs.erdos_renyi(25, 0.5, seed)
    c = _cbm(ei, alpha)
    assert c is not None
    c.check_format(torch.from_numpy(ei))
    ref = orc.build_structure(ei, alpha)
    # the optimum weight is unique even where the optimal tree is not
    assert c.build_info["n_delta"] == ref["weight"]
    assert c.mst_row.dtype == torch.int32 and c.mst_col.dtype == torch.int32
    assert c.mst_row.numel() == c.num_rows + 2 and c.mst_col.numel() == c.num_rows
    assert c.deltas.layout == torch.sparse_csr and tuple(c.deltas.shape) == (c.num_rows, c.num_rows)
    assert c.deltas.values().dtype == torch.float32


def test_structure_optimal_against_networkx():
    nx = pytest.importorskip("networkx")
    ei = graphs.make_graph("c1", scale=0.03)
    n = int(ei.max()) + 1
    c = _cbm(ei, 0)
    g = nx.DiGraph()
    for u, v, w in orc.candidate_edges(ei, n, 0):
        if not g.has_edge(u, v) or g[u][v]["weight"] > w:
            g.add_edge(u, v, weight=w)
    ref = nx.minimum_spanning_arborescence(g)
    assert c.build_info["n_delta"] == sum(d["weight"] for _, _, d in ref.edges(data=True))


def test_candidate_rule_respected():
    """Every tree edge u -> v below the virtual root satisfies h(u, v) < |v| - alpha
    (cbm/cbm_extensions.cpp:93-101) and carries exactly h(u, v) delta entries."""
    alpha = 2
    ei = graphs.make_graph("c1", scale=0.2)
    c = _cbm(ei, alpha)
    n = c.num_rows
    rows = orc.pattern_rows(ei, n)
    dl = np.diff(c._crow)
    for v in range(n):
        u = int(c._parent[v])
        if u == n:
            assert dl[v] == rows[v].size
        else:
            h = np.setxor1d(rows[u], rows[v]).size
            assert h < rows[v].size - alpha and dl[v] == h


@pytest.mark.parametrize("alpha", [0, 1, 5, 40, -3])
def test_candidate_set_equals_all_pairs_enumeration(alpha):
    """The builder finds candidates through a rare-column prefix instead of visiting every
    intersecting pair; the set must be the one the all-pairs rule of cbm/cbm_extensions.cpp:75-102
    yields."""
    for ei in (graphs.make_graph("c1", scale=0.15), graphs.erdos_renyi(40, 0.4, 9),
               graphs.copy_model(400, 0.95, 6, 3)):
        n = int(ei.max()) + 1
        c = _cbm(ei, alpha)
        ref = orc.candidate_edges(ei, n, alpha)
        assert c.build_info["n_candidates"] == len(ref)
        assert c.build_info["n_delta"] == orc.build_structure(ei, alpha)["weight"]


def test_deterministic_and_thread_independent():
    ei = graphs.make_graph("c1", scale=0.25)
    e = torch.from_numpy(ei).to(torch.int32)
    a = cbm_matrix(e, torch.ones(e.shape[1]), alpha=1, n_threads=1)
    b = cbm_matrix(e, torch.ones(e.shape[1]), alpha=1, n_threads=4)
    for x, y in ((a.mst_row, b.mst_row), (a.mst_col, b.mst_col)):
        assert torch.equal(x, y)
    assert np.array_equal(a._crow, b._crow) and np.array_equal(a._dcol, b._dcol)
    assert np.array_equal(a._dval, b._dval)


def test_normalized_values_are_signed_multipliers():
    ei = with_self_loops(graphs.erdos_renyi(30, 0.3, 5))
    c = _cbm(ei, 2, normalized=True)
    c.check_format(torch.from_numpy(ei))
    mult = c.col_multiplier.numpy()
    np.testing.assert_array_equal(mult, orc.row_multiplier(ei, c.num_rows))
    np.testing.assert_array_equal(np.abs(c._dval), mult[c._dcol])


def test_coo_export_is_breadth_first_and_equivalent():
    ei = graphs.erdos_renyi(25, 0.5, 11)
    row, col = ei[0].astype(np.int32), ei[1].astype(np.int32)
    n = int(ei.max()) + 1
    L = _lib.lib()
    h = ctypes.c_void_p(0)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    _lib.check(L.cbm_b200_build(p(row), p(col), row.shape[0], n, 2, None, 0, ctypes.byref(h)))
    nd = ctypes.c_int64()
    _lib.check(L.cbm_b200_built_info(h, ctypes.byref(nd), None, None, None, None))
    mst_row, mst_col = np.empty(n + 2, np.int32), np.empty(n, np.int32)
    crow, dcol, dval = np.empty(n + 1, np.int32), np.empty(nd.value, np.int32), np.empty(nd.value, np.float32)
    _lib.check(L.cbm_b200_built_export_csr(h, p(mst_row), p(mst_col), p(crow), p(dcol), p(dval), None))
    cr, cc, cv = np.empty(nd.value, np.int32), np.empty(nd.value, np.int32), np.empty(nd.value, np.float32)
    _lib.check(L.cbm_b200_built_export_coo(h, p(cr), p(cc), p(cv)))
    L.cbm_b200_built_free(h)
    # the reference coalesces its COO output into CSR (cbm/cbm.py:120-141): same matrix
    o = np.lexsort((cc, cr))
    assert np.array_equal(cc[o], dcol) and np.array_equal(cv[o], dval)
    assert np.array_equal(np.bincount(cr, minlength=n), np.diff(crow))
    # rows appear in breadth-first order of the tree
    first = [r for i, r in enumerate(cr.tolist()) if i == 0 or cr[i - 1] != r]
    bfs = []
    frontier = [n]
    while frontier:
        nxt = []
        for u in frontier:
            nxt.extend(mst_col[mst_row[u]:mst_row[u + 1]].tolist())
        bfs.extend(nxt)
        frontier = nxt
    # the walk is a queue, not level-synchronous, but children stay in mst_col order: same sequence
    assert first == [v for v in bfs if crow[v + 1] > crow[v]]


def test_edge_cases():
    # a row without entries (node 2 has only an incoming edge) and duplicate input entries
    ei = np.array([[0, 0, 1, 1, 3, 3, 0], [1, 2, 0, 2, 0, 1, 1]], dtype=np.int64)
    c = _cbm(ei, 0)
    c.check_format(torch.from_numpy(ei))
    assert c.num_rows == 4 and c.build_info["n_delta"] <= 6
    # single entry
    c1 = _cbm(np.array([[0], [0]]), 0)
    assert c1.num_rows == 1 and c1.build_info["n_delta"] == 1
    # identical rows compress to nothing below the first
    ei = np.array([[0, 0, 1, 1, 2, 2], [3, 4, 3, 4, 3, 4]], dtype=np.int64)
    c2 = _cbm(ei, 0)
    assert c2.build_info["n_delta"] == 2
    c2.check_format(torch.from_numpy(ei))
    # large alpha forbids every non-virtual edge
    c3 = _cbm(graphs.erdos_renyi(25, 0.5, 3), alpha=1000)
    assert c3.build_info["n_root_children"] == c3.num_rows and c3.build_info["depth"] == 1


def test_builder_rejects_bad_input():
    L = _lib.lib()
    h = ctypes.c_void_p(0)
    row = np.array([0, 5], dtype=np.int32)
    col = np.array([1, 0], dtype=np.int32)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    assert L.cbm_b200_build(p(row), p(col), 2, 3, 0, None, 0, ctypes.byref(h)) == 1
    assert b"out of range" in L.cbm_b200_last_error()
    assert L.cbm_b200_build(None, None, 2, 3, 0, None, 0, ctypes.byref(h)) == 1
    with pytest.raises(ValueError):
        cbm_matrix(torch.zeros((3, 4), dtype=torch.int32), torch.ones(4))


def test_save_load_round_trip_and_compression_ratio(tmp_path):
    ei = with_self_loops(graphs.make_graph("c1", scale=0.2))
    c = _cbm(ei, 2, normalized=True)
    path = tmp_path / "c.pt"
    c.save(path)
    d = cbm_matrix.load(path)
    assert torch.equal(c.mst_row, d.mst_row) and torch.equal(c.mst_col, d.mst_col)
    assert np.array_equal(c._crow, d._crow) and np.array_equal(c._dcol, d._dcol) and np.array_equal(c._dval, d._dval)
    assert torch.equal(c.col_multiplier, d.col_multiplier) and d.alpha == 2 and d.normalized
    assert d.is_symmetric() == c.is_symmetric()
    d.check_format(torch.from_numpy(ei))
    # the reference's metric: CSR elements over CBM elements (benchmark/utility.py:45-64)
    n, nnz, nd = c.num_rows, ei.shape[1], c.build_info["n_delta"]
    want = ((n + 1) + 2 * nnz) / ((n + 1) + 2 * nd + (n + 2) + n)
    assert abs(c.compression_ratio() - want) < 1e-12 and abs(d.compression_ratio() - want) < 1e-12


def test_alpha_search_byte_model():
    from cbm4gnn_b200.alpha_search import product_bytes, search_alpha
    ei = torch.from_numpy(graphs.copy_model(1500, 0.95, 8, 5))
    best, table = search_alpha(ei, f=64, alphas=(0, 2, 8, 1000), measure=False)
    assert [r["alpha"] for r in table] == [0, 2, 8, 1000]
    nd = [r["n_delta"] for r in table]
    assert nd == sorted(nd) and table[-1]["n_root_children"] == int(ei.max()) + 1
    assert best == min(table, key=lambda r: (r["bytes"], r["alpha"]))["alpha"] and best != 1000
    r = table[0]
    assert r["bytes"] == product_bytes(int(ei.max()) + 1, r["n_delta"], r["n_root_children"], 64)


def test_structure_is_pinned_byte_for_byte():
    """Same seed, same structure: digests of (mst_row, mst_col, delta row pointers, columns, signs)
    for two seeded graphs.  A change here means the builder's output changed (tie-breaking, order
    of children, candidate rule) and every stored structure and measurement with it."""
    import hashlib

    def digest(c):
        h = hashlib.sha256()
        for a in (c.mst_row.numpy(), c.mst_col.numpy(), c._crow, c._dcol, np.sign(c._dval).astype(np.int8)):
            h.update(np.ascontiguousarray(a).tobytes())
        return h.hexdigest()

    c = _cbm(graphs.make_graph("c1"), 0)
    assert c.build_info["n_delta"] == 77490
    assert digest(c) == "ef3d6b5c798651d5488d8e9447f7b25098500866faf946e00aaae1aca00752b4"
    c = _cbm(with_self_loops(graphs.make_graph("c2", scale=0.1)), 8, normalized=True)
    assert c.build_info["n_delta"] == 300192
    assert digest(c) == "f096072e632b1da7ae1c82abf0c7dc8819e6cb691a62e957f0437f1c72097aba"


def test_random_small_patterns_are_valid_and_optimal():
    """Property check of the arborescence solver and the candidate search on arbitrary (also
    non-symmetric, also rank-deficient) small patterns: the structure must reproduce the matrix and
    its weight must equal the optimum found by the independent O(V*E) solver of the restatement.
    Small dense patterns produce many ties and nested cycles, the hard cases of the contraction."""
    hyp = pytest.importorskip("hypothesis")
    st = pytest.importorskip("hypothesis.strategies")

    @hyp.settings(max_examples=60, deadline=None, derandomize=True)
    @hyp.given(st.integers(2, 11), st.integers(0, 2 ** 31 - 1), st.floats(0.15, 0.9), st.integers(0, 3))
    def check(n, seed, p, alpha):
        rng = np.random.default_rng(seed)
        mask = rng.random((n, n)) < p
        mask[n - 1, rng.integers(0, n)] = True          # the matrix is n x n: last row is not empty
        ei = np.stack(np.nonzero(mask)).astype(np.int64)
        if int(ei.max()) + 1 != n:
            mask[rng.integers(0, n), n - 1] = True
            ei = np.stack(np.nonzero(mask)).astype(np.int64)
        c = _cbm(ei, alpha)
        c.check_format(torch.from_numpy(ei))
        ref = orc.build_structure(ei, alpha)
        assert c.build_info["n_delta"] == ref["weight"]
        assert c.build_info["n_candidates"] == len(orc.candidate_edges(ei, n, alpha))

    check()


def test_gpu_build_entry_point_falls_back_to_the_host_search():
    """Without a usable CUDA device the GPU-assisted builder runs the host search and says so; the
    structure is the one cbm_b200_build emits."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present: the GPU search itself is covered by the gpu tests")
    from cbm4gnn_b200.cbm import cbm_matrix
    ei = torch.from_numpy(graphs.make_graph("c1", scale=0.2)).to(torch.int32)
    a = cbm_matrix(ei, torch.ones(ei.shape[1]), alpha=2)
    b = cbm_matrix(ei, torch.ones(ei.shape[1]), alpha=2, build_device=0)
    assert b.build_info["candidates_on_gpu"] is False
    assert torch.equal(a.mst_row, b.mst_row) and torch.equal(a.mst_col, b.mst_col)
    assert np.array_equal(a._dcol, b._dcol) and np.array_equal(a._dval, b._dval)


def test_check_format_rejects_corrupted_structures():
    """The validator has to fail on: a wrong matrix, a flipped delta sign, a zero delta, a column
    removed that the parent does not hold."""
    import torch
    from cbm4gnn_b200.cbm import cbm_matrix
    ei = graphs.make_graph("c1", scale=0.1)
    e = torch.from_numpy(ei).to(torch.int32)
    c = cbm_matrix(e, torch.ones(e.shape[1]), alpha=0)
    c.check_format(e)
    with pytest.raises(ValueError, match="Format is incorrect"):
        c.check_format(e[:, :-2])                       # two entries of the matrix missing
    keep = c._dval.copy()
    neg = np.nonzero(c._dval < 0)[0]
    assert neg.size > 0                                 # the graph compresses: some deltas remove columns
    c._dval[neg[0]] = 1.0
    with pytest.raises(ValueError, match="Format is incorrect"):
        c.check_format(e)
    c._dval[:] = keep
    c._dval[0] = 0.0
    with pytest.raises(ValueError, match="Failed with the edge index"):
        c.check_format(e)
    c._dval[:] = keep
    root_child = int(c.mst_col[c.mst_row[c.num_rows]])  # a child of the virtual root removes nothing
    k = c._crow[root_child]
    c._dval[k] = -1.0
    with pytest.raises(ValueError, match="Format is incorrect"):
        c.check_format(e)
    c._dval[:] = keep
    c.check_format(e)


@pytest.mark.parametrize("dtype,device", [(torch.float64, None), (torch.bfloat16, None), (torch.float32, "meta")])
def test_multiplier_and_deltas_whatever_the_defaults_of_torch(dtype, device):
    """The row degrees are 32-bit floats in host memory also where new tensors are by default something else."""
    ei = torch.from_numpy(with_self_loops(graphs.copy_model(300, 0.8, 3, 1))).to(torch.int32)
    values = torch.ones(ei.shape[1])
    want = cbm_matrix(ei, values, alpha=2, normalized=True)
    torch.set_default_dtype(dtype)
    torch.set_default_device(device)
    try:
        got = cbm_matrix(ei, values, alpha=2, normalized=True)
    finally:
        torch.set_default_dtype(torch.float32)
        torch.set_default_device(None)
    assert got.col_multiplier.dtype == torch.float32 and torch.equal(got.col_multiplier, want.col_multiplier)
    assert np.array_equal(got._dcol, want._dcol) and np.array_equal(got._dval, want._dval)


@pytest.mark.parametrize("room", [12, 13, 14, 14.5, 15, 15.5])
def test_memory_that_runs_out_is_an_error_not_an_abort(room):
    """The counting sort of an unsorted edge list allocates before its threads start: a process whose memory is limited so
    that the row pointers and the sorted columns (12 bytes a row here) fit and the threads' counters do not gets a
    status back."""
    import os
    import subprocess
    import sys
    code = f"""
import ctypes, resource
import numpy as np
L = ctypes.CDLL({_lib.LIB_PATH!r})
L.cbm_b200_last_error.restype = ctypes.c_char_p
def build(n):
    row = np.arange(n, dtype=np.int32)[::-1].copy()
    out, p = ctypes.c_void_p(), ctypes.c_void_p(row.ctypes.data)
    return row, lambda: L.cbm_b200_build(p, p, ctypes.c_int64(n), n, 0, None, 0, ctypes.byref(out))
row, run = build(300_000)
assert run() == 0  # the threads are there now
n = 8_000_000
row, run = build(n)
used = int(next(s for s in open("/proc/self/status") if s.startswith("VmSize")).split()[1]) * 1024
resource.setrlimit(resource.RLIMIT_AS, (used + int({room} * n), resource.getrlimit(resource.RLIMIT_AS)[1]))
print(run(), L.cbm_b200_last_error().decode())
"""
    _lib.lib()  # (built)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, OMP_NUM_THREADS="4"))
    assert done.returncode == 0 and "memory" in done.stdout, (done.returncode, done.stdout, done.stderr[-300:])


@pytest.mark.parametrize("normalized", [False, True])
@pytest.mark.parametrize("edge,message", [([-1, 0], "negative row"), ([0, -1], "out of range"), ([2**31 - 1, 0], "too large")])
def test_indices_out_of_range_are_refused(edge, message, normalized):
    with pytest.raises(RuntimeError, match=message):
        cbm_matrix(torch.tensor([[0, 1, edge[0]], [0, 1, edge[1]]]), torch.ones(3), normalized=normalized)
