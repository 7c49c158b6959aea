"""Shared helpers of the test-suite (CPU side)."""
import ctypes

import numpy as np
import torch

from cbm4gnn_b200 import _lib
from cbm4gnn_b200.utility import add_self_loops


def with_self_loops(ei: np.ndarray) -> np.ndarray:
    return add_self_loops(torch.from_numpy(ei)).numpy()


def dense_product(ei: np.ndarray, x: np.ndarray, normalized: bool) -> np.ndarray:
    """float64 ``A @ x`` or ``D^-1/2 A D^-1/2 @ x`` (D = row degrees of the matrix as given)."""
    n = x.shape[0]
    a = np.zeros((n, n))
    a[ei[0], ei[1]] = 1.0
    if normalized:
        with np.errstate(divide="ignore"):
            s = a.sum(1) ** -0.5
        a = s[:, None] * a * s[None, :]
    return a @ x.astype(np.float64)


def sparse_product(ei: np.ndarray, x: np.ndarray, normalized: bool) -> np.ndarray:
    """The same through scipy CSR in float64, for sizes a dense matrix does not fit."""
    import scipy.sparse as sp
    n = x.shape[0]
    a = sp.csr_matrix((np.ones(ei.shape[1]), (ei[0], ei[1])), shape=(n, n))
    if normalized:
        s = np.asarray(a.sum(1)).ravel() ** -0.5
        a = sp.diags(s) @ a @ sp.diags(s)
    return a @ x.astype(np.float64)


def near_cliques(n: int, size: int, missing: float, seed: int) -> np.ndarray:
    """Communities of ``size`` nodes, numbers shuffled, that are complete but for a share ``missing`` of the links (self loops
    stay): rows save nearly all of their entries by a parent, and wait for it in a product in one pass too."""
    rng = np.random.default_rng(seed)
    label = rng.permutation(n)
    pairs = []
    for first in range(0, n, size):
        k = min(size, n - first)
        there = rng.random((k, k)) >= missing
        there = np.triu(there, 1)
        there = there | there.T | np.eye(k, dtype=bool)
        pairs.append(np.stack(np.nonzero(there)) + first)
    ei = label[np.concatenate(pairs, axis=1)]
    key = np.sort(ei[0] * n + ei[1])
    return np.stack([key // n, key % n])


def chains(length: int, count: int) -> np.ndarray:
    """``count`` chains of ``length`` rows: each names one column more than the one before, so that it waits for it, and is far
    too long to be computed whole instead."""
    row, col = np.repeat(np.arange(length), np.arange(1, length + 1)), np.concatenate([np.arange(i + 1) for i in range(length)])
    return np.concatenate([np.stack([row, col]) + k * length for k in range(count)], axis=1)


def waiting_rows(c) -> int:
    """Rows of a ``cbm_matrix`` that wait for their parent's in the product in one pass.  (By the schedule made without a GPU,
    whose choice of rows does not depend on their order.)"""
    n, p = c.num_rows, lambda a: None if a is None else ctypes.c_void_p(a.ctypes.data)
    mult = None if c.col_multiplier is None else c.col_multiplier.numpy()
    parent = np.empty(n, np.int32)
    _lib.check(_lib.lib().cbm_b200_schedule_lifted(n, p(c.mst_row.numpy()), p(c.mst_col.numpy()), p(c._crow), p(c._dcol), p(c._dval),
                                                   p(mult), None, None, p(parent), None, 0, None, None))
    return int((parent != n).sum())
