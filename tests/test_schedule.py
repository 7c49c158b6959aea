"""The host-side schedule of a plan (no GPU): sizes and the pre-launch checks."""
import ctypes

import numpy as np
import pytest
import torch

from cbm4gnn_b200 import _lib, graphs
from cbm4gnn_b200.cbm import cbm_matrix
from cbm4gnn_b200.sharding import partition_subtrees
from helpers import with_self_loops


def _cbm(ei, alpha=0, normalized=False):
    e = torch.from_numpy(np.ascontiguousarray(ei)).to(torch.int32)
    return cbm_matrix(e, torch.ones(e.shape[1]), alpha=alpha, normalized=normalized)


def _schedule(c, perm=None, n_labels=0, own=None, mst_col=None):
    L = _lib.lib()
    n = c.num_rows
    p = lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)
    out = [ctypes.c_int32() for _ in range(4)]
    mult = None if c.col_multiplier is None else c.col_multiplier.numpy()
    mc = c.mst_col.numpy() if mst_col is None else mst_col
    b, e = own if own else (0, n_labels or n)
    perm32 = None if perm is None else np.ascontiguousarray(perm, dtype=np.int32)
    rc = L.cbm_b200_schedule_info(n, p(c.mst_row.numpy()), p(mc), p(c._crow), p(c._dcol), p(c._dval), p(mult),
                                  p(perm32), n_labels, b, e, *[ctypes.byref(o) for o in out])
    return rc, [o.value for o in out]


def _expected(c, rows=None):
    dl = np.diff(c._crow)
    rows = np.arange(c.num_rows) if rows is None else rows
    split = dl[rows] > 192
    n_partial = int((-(-dl[rows][split] // 128) - 1).sum())
    easy = int(((c._parent[rows] == c.num_rows) & ~split).sum())
    return len(rows) + n_partial, n_partial + easy, n_partial, len(rows)


@pytest.mark.parametrize("make", [
    lambda: _cbm(graphs.erdos_renyi(25, 0.5, 1), 2),
    lambda: _cbm(graphs.make_graph("c1"), 0),
    lambda: _cbm(with_self_loops(graphs.make_graph("c1", scale=0.5)), 1, normalized=True),
    lambda: _cbm(with_self_loops(graphs.copy_model(2000, 0.95, 20, 3)), 4, normalized=True),
])
def test_schedule_sizes_and_checks(make):
    c = make()
    rc, got = _schedule(c)
    assert rc == 0, _lib.lib().cbm_b200_last_error()
    assert tuple(got) == _expected(c)


def test_schedule_of_a_chain_and_of_a_hub():
    n = 600
    rows = np.repeat(np.arange(n), np.arange(1, n + 1))
    cols = np.concatenate([np.arange(i + 1) for i in range(n)])
    c = _cbm(np.stack([rows, cols]), 0)                 # one chain of depth n: nothing but waiting items
    rc, got = _schedule(c)
    assert rc == 0 and tuple(got) == (n, 1, 0, n)
    c = _cbm(np.stack([rows, cols]), 100000)            # no compression: long rows are split
    rc, got = _schedule(c)
    assert rc == 0 and tuple(got) == _expected(c) and got[2] > 0


def test_schedule_of_shards_and_refusals():
    c = _cbm(with_self_loops(graphs.make_graph("c1")), 0, normalized=True)
    n = c.num_rows
    part = partition_subtrees(c, 3)
    total_rows = 0
    for g in range(3):
        rc, got = _schedule(c, perm=part.perm, n_labels=part.n_labels, own=part.offsets(g))
        assert rc == 0, _lib.lib().cbm_b200_last_error()
        mine = np.nonzero(part.perm // part.shard_rows == g)[0]
        assert tuple(got) == _expected(c, mine)
        total_rows += got[3]
    assert total_rows == n
    # an owned range that cuts a subtree
    deep = int(np.nonzero(c._parent != n)[0][0])
    rc, _ = _schedule(c, perm=np.arange(n), n_labels=n, own=(deep, deep + 1))
    assert rc == 1 and b"cuts a subtree" in _lib.lib().cbm_b200_last_error()
    # a tree with a repeated child is not a tree
    mc = c.mst_col.numpy().copy()
    mc[0] = mc[1]
    rc, _ = _schedule(c, mst_col=mc)
    assert rc == 3
    # labels that collide
    perm = np.arange(n)
    perm[1] = 0
    rc, _ = _schedule(c, perm=perm, n_labels=n)
    assert rc == 1


def _as_planned(c, labels=None):
    n = c.num_rows
    p = lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)
    out, mark = [ctypes.c_int32() for _ in range(5)], ctypes.c_uint64()
    mult = None if c.col_multiplier is None else c.col_multiplier.numpy()
    labels = None if labels is None else np.ascontiguousarray(labels, dtype=np.int32)
    rc = _lib.lib().cbm_b200_schedule_as_planned(n, p(c.mst_row.numpy()), p(c.mst_col.numpy()), p(c._crow), p(c._dcol), p(c._dval),
                                                 p(mult), p(labels), *[ctypes.byref(o) for o in out], ctypes.byref(mark))
    return rc, [o.value for o in out], mark.value


def _hub_graph():
    """A tree some levels deep, a row of 700 entries and rows of odd length."""
    ei = with_self_loops(graphs.copy_model(1500, 0.9, 8, 11))
    n = int(ei.max()) + 1
    key = np.unique(np.concatenate([ei[0] * n + ei[1], 7 * n + np.arange(700, 1400)]))
    return np.stack([key // n, key % n])


@pytest.mark.parametrize("make,segment", [(lambda: _cbm(_hub_graph(), 2, normalized=True), 64),
                                          (lambda: _cbm(with_self_loops(graphs.copy_model(1000, 0.95, 40, 3)), 1000), 128)])
@pytest.mark.parametrize("communities", [None, 1, 7, 300])
def test_schedule_by_the_rules_of_a_plan(make, segment, communities):
    """Rows cut by the length of the mean row; with communities also the order, the chunks and the paired entries pass the
    checks (every item behind those it waits for, chunks that hold their items' entries)."""
    c = make()
    n, length = c.num_rows, np.diff(c._crow)
    assert (length.mean() <= 64) == (segment == 64) and (length % 2).any()
    labels = None if communities is None else np.random.default_rng(1).integers(0, communities, n)
    rc, got, mark = _as_planned(c, labels)
    assert rc == 0, _lib.lib().cbm_b200_last_error()
    split = length > 3 * segment // 2
    n_partial = int((-(-length[split] // segment) - 1).sum())
    easy = int(((c._parent == n) & ~split).sum())
    assert got[:3] == [n + n_partial, n_partial + easy, n_partial] and got[4] == segment and n_partial > 0
    assert (got[3] > 0) == (labels is not None) and got[3] * 32 >= (got[0] if labels is not None else 0)
    assert _as_planned(c, labels)[2] == mark
    if labels is not None and communities > 1:
        assert mark != _as_planned(c)[2]


def test_labels_out_of_range_are_refused():
    c = _cbm(graphs.erdos_renyi(25, 0.5, 1), 2)
    for label in (-1, c.num_rows):
        assert _as_planned(c, np.full(c.num_rows, label))[0] == 1


@pytest.mark.parametrize("room", [2, 6, 12, 30, 60])
@pytest.mark.parametrize("entry", ["schedule_info", "schedule_as_planned"])
def test_memory_that_runs_out_is_an_error_not_an_abort(entry, room):
    """A schedule of 8 000 000 rows takes over 100 bytes a row; with less (``room`` bytes) the call returns."""
    import os
    import subprocess
    import sys
    code = f"""
import ctypes, resource
import numpy as np
L = ctypes.CDLL({_lib.LIB_PATH!r})
L.cbm_b200_last_error.restype = ctypes.c_char_p
n = 8_000_000
col, val, crow = np.arange(n, dtype=np.int32), np.ones(n, np.float32), np.arange(n + 1, dtype=np.int32)
row = np.zeros(n + 2, np.int32)
row[n + 1] = n  # every row a child of the virtual root
p = lambda a: ctypes.c_void_p(a.ctypes.data)
rest = [None, 0, 0, n, None, None, None, None] if {entry!r} == "schedule_info" else [None] * 7
used = int(next(s for s in open("/proc/self/status") if s.startswith("VmSize")).split()[1]) * 1024
resource.setrlimit(resource.RLIMIT_AS, (used + {room} * n, resource.getrlimit(resource.RLIMIT_AS)[1]))
print(L.cbm_b200_{entry}(n, p(row), p(col), p(crow), p(col), p(val), None, *rest), L.cbm_b200_last_error().decode())
"""
    _lib.lib()  # (built)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, OMP_NUM_THREADS="2"))
    assert done.returncode == 0 and "memory" in done.stdout, (done.returncode, done.stdout, done.stderr[-300:])


def _lifted(c, labels=None):
    n = c.num_rows
    p = lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)
    mult = None if c.col_multiplier is None else c.col_multiplier.numpy()
    labels = None if labels is None else np.ascontiguousarray(labels, dtype=np.int32)
    lifted, parent, crow = ctypes.c_int32(), np.empty(n, np.int32), np.empty(n + 1, np.int64)
    call = lambda cap, col, val: _lib.lib().cbm_b200_schedule_lifted(
        n, p(c.mst_row.numpy()), p(c.mst_col.numpy()), p(c._crow), p(c._dcol), p(c._dval), p(mult), p(labels), ctypes.byref(lifted),
        p(parent), p(crow), cap, p(col), p(val))
    assert call(0, None, None) == 0, _lib.lib().cbm_b200_last_error()
    col, val = np.empty(crow[n], np.int32), np.empty(crow[n], np.float32)
    assert call(len(col), col, val) == 0
    return lifted.value, parent, crow, col, val


def _nested(n):
    return np.stack([np.repeat(np.arange(n), np.arange(1, n + 1)), np.concatenate([np.arange(i + 1) for i in range(n)])])


@pytest.mark.parametrize("ei,alpha,normalized,some_stay", [
    (with_self_loops(graphs.copy_model(1500, 0.9, 8, 11)), 2, True, False),     # split rows, some levels
    (graphs.copy_model(3000, 0.8, 3, 5), 0, False, False),                      # a dozen levels that save next to nothing
    (with_self_loops(graphs.copy_model(3000, 0.97, 60, 3)), 4, True, None),     # savings of all sizes
    (_nested(400), 0, False, True), (_nested(400), 0, True, True),              # a chain: whole rows would be 100 times the entries
])
@pytest.mark.parametrize("communities", [None, 7])
def test_lifted_rows_are_whole_rows(ei, alpha, normalized, some_stay, communities):
    c = _cbm(ei, alpha, normalized=normalized)
    n = c.num_rows
    labels = None if communities is None else np.random.default_rng(1).integers(0, communities, n)
    lifted, parent, crow, col, val = _lifted(c, labels)
    moved = parent != c._parent
    assert lifted == moved.sum() and np.all(parent[moved] == n)
    assert some_stay is None or (parent != n).any() == some_stay
    assert lifted > 0 or some_stay
    mult = np.ones(n, np.float32) if not normalized else c.col_multiplier.numpy()
    key = np.unique(ei[0].astype(np.int64) * n + ei[1])
    whole = np.split(key % n, np.searchsorted(key // n, np.arange(1, n)))
    for v in range(n):
        a, b = slice(crow[v], crow[v + 1]), slice(c._crow[v], c._crow[v + 1])
        if moved[v]:
            assert np.array_equal(col[a], whole[v]) and np.array_equal(val[a], mult[whole[v]])
        else:
            assert np.array_equal(col[a], c._dcol[b]) and np.array_equal(val[a], c._dval[b])


@pytest.mark.parametrize("spoil", ["value", "order"])
def test_a_structure_that_is_no_signed_pattern_is_not_lifted(spoil):
    """Values that do not cancel, and columns out of order, are taken as they are: no row is computed from other entries."""
    c = _cbm(graphs.copy_model(3000, 0.8, 3, 5), 0)
    assert _lifted(c)[0] > 0
    c._dval, c._dcol = c._dval.copy(), c._dcol.copy()
    minus = next(v for v in range(c.num_rows) if (c._dval[c._crow[v]:c._crow[v + 1]] < 0).any() and c._crow[v + 1] - c._crow[v] > 1)
    at = slice(c._crow[minus], c._crow[minus + 1])
    if spoil == "value":
        c._dval[at] *= 1.5
    else:
        c._dcol[at], c._dval[at] = c._dcol[at][::-1].copy(), c._dval[at][::-1].copy()
    lifted, parent, crow, col, val = _lifted(c)
    assert lifted == 0 and np.array_equal(parent, c._parent)
    assert np.array_equal(col, c._dcol) and np.array_equal(val, c._dval)


def _csr_as_planned(n_rows, n_cols, labels, seed=0):
    rng = np.random.default_rng(seed)
    crow = np.arange(0, 8 * n_rows + 1, 8, dtype=np.int32)
    col = np.sort(rng.integers(0, n_cols, (n_rows, 8)), axis=1).astype(np.int32)
    val, labels = np.ones(8 * n_rows, np.float32), np.ascontiguousarray(labels, dtype=np.int32)
    p = lambda a: ctypes.c_void_p(a.ctypes.data)
    out, mark = [ctypes.c_int32() for _ in range(5)], ctypes.c_uint64()
    rc = _lib.lib().cbm_b200_csr_schedule_as_planned(n_rows, n_cols, p(crow), p(col), p(val), p(labels),
                                                     *[ctypes.byref(o) for o in out], ctypes.byref(mark))
    assert rc == 0, _lib.lib().cbm_b200_last_error()
    return [o.value for o in out]


@pytest.mark.parametrize("n_rows,n_cols", [(300, 299), (300, 300), (300, 301), (200, 1000), (1000, 200), (1, 5)])
def test_only_square_matrices_are_ordered_by_community(n_rows, n_cols):
    """A column number is a row's number only where there are as many of them: nobody looks for communities, whose search
    follows columns to rows, in other matrices."""
    n_items, n_prefix, n_partial, n_chunks, _ = _csr_as_planned(n_rows, n_cols, np.arange(n_rows) % 3 % n_rows)
    assert n_items == n_prefix == n_rows and n_partial == 0
    assert (n_chunks > 0) == (n_rows == n_cols)


@pytest.mark.parametrize("warps", [2368, 3552, 7104])
def test_one_round_has_a_warp_for_every_claim(warps):
    """From no slab to a warp up to several times as many slabs as there are warps, where there can be no such round."""
    group_of = _lib.lib().cbm_b200_one_round_group
    for n_slabs in [1, 2, 3, 4, 7, 111, warps // 4, warps // 2 - 1, warps // 2, warps // 2 + 1, warps - 1, warps, warps + 1, 7813, 40_000]:
        for n_prefix in [1, 2, 3, 4, 5, 8, 63, 1000]:
            for n_waiting in [0, 1, 5, 500]:
                group = group_of(n_prefix, n_waiting, n_slabs, warps)
                waiting = n_waiting * n_slabs
                fits = lambda g: -(-n_prefix // g) * n_slabs + waiting <= warps
                if waiting >= warps // 4 or n_slabs + waiting > warps:  # (all of a slab's prefix to one warp)
                    assert group == 0
                else:
                    assert 1 <= group <= n_prefix and fits(group) and (group == 1 or not fits(group - 1))


def _run_on_pairs(pairs, more, body):
    """``body`` in a process of its own, on a structure of ``pairs`` rows of 4 entries and as many children with ``more``
    entries beside their parent's: all children are lifted."""
    import os
    import subprocess
    import sys
    code = f"""
import ctypes, os, resource, threading
import numpy as np
L = ctypes.CDLL({_lib.LIB_PATH!r})
L.cbm_b200_last_error.restype = ctypes.c_char_p
pairs, more = {pairs}, {more}
n = 2 * pairs
row = np.full(n + 2, pairs, np.int32)
row[0], row[n + 1] = 0, n
row[1:pairs + 1] = np.arange(1, pairs + 1)  # row i has the child pairs + i
col = np.concatenate([np.arange(pairs, n), np.arange(pairs)]).astype(np.int32)
length = np.concatenate([np.full(pairs, 4), np.full(pairs, more)])
crow = np.concatenate([[0], np.cumsum(length)]).astype(np.int32)
dcol = np.concatenate([np.tile(np.arange(4), pairs), np.tile(np.arange(4, 4 + more), pairs)]).astype(np.int32)
val = np.ones(len(dcol), np.float32)
p = lambda a: ctypes.c_void_p(a.ctypes.data)
def lifted():
    count = ctypes.c_int32(-1)
    rc = L.cbm_b200_schedule_lifted(n, p(row), p(col), p(crow), p(dcol), p(val), None, None, ctypes.byref(count), None, None,
                                    ctypes.c_int64(0), None, None)
    return rc, count.value
{body}
"""
    _lib.lib()  # (built)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                          env=dict(os.environ, OMP_NUM_THREADS="4", MALLOC_MMAP_THRESHOLD_="65536", MALLOC_ARENA_MAX="1"))
    assert done.returncode == 0, (done.returncode, done.stdout, done.stderr[-300:])
    return done.stdout


def test_one_team_of_threads_makes_both_schedules():
    """Beside the calling thread's team (4 with it) there is one thread more, not a second team."""
    said = _run_on_pairs(12_000, 100, """
base, most, done = threading.active_count(), 0, False
def watch():
    global most
    while not done:
        most = max(most, len(os.listdir("/proc/self/task")))
before = len(os.listdir("/proc/self/task"))
watcher = threading.Thread(target=watch)
watcher.start()
for _ in range(20):
    assert lifted() == (0, pairs)
done = True
watcher.join()
print(most - before - 1)
""")
    assert 1 <= int(said) <= 3 + 1


def test_a_plan_without_memory_for_lifted_rows_goes_by_its_tree():
    """With less and less memory: both schedules, then the tree's alone, then an error."""
    said = _run_on_pairs(200_000, 10, """
assert lifted() == (0, pairs)
used = int(next(s for s in open("/proc/self/status") if s.startswith("VmSize")).split()[1]) * 1024
hard = resource.getrlimit(resource.RLIMIT_AS)[1]
seen = []
for room in range(600, 0, -8):  # bytes a row
    resource.setrlimit(resource.RLIMIT_AS, (used + room * n, hard))
    rc, count = lifted()
    resource.setrlimit(resource.RLIMIT_AS, (hard, hard))
    assert rc == 0 or b"memory" in L.cbm_b200_last_error()
    seen.append((rc, count if rc == 0 else 0))
    if rc:
        break
print(sorted(set(seen)) == [(0, 0), (0, pairs), (seen[-1][0], 0)], sorted(set(seen)))
""")
    assert said.startswith("True"), said
