"""The dense half of a GCN layer on B200's tensor cores.

A layer of the reference is ``lin`` followed by ``propagate``
(gnns/graph_convolutional_network/cbm_gcn.py:21-24); ``lin`` is a bias-free fp32 map
``[N, in] x [in, out]``.  ``linear(x, weight)`` runs it, and ``autograd`` its two gradients, through
the library's fp32-accurate tensor-core GEMMs (``cbm_b200_dense_forward`` / ``_grad_input`` /
``_grad_weight``: operands split into three bf16 terms, fp32 accumulation), which keep the 1e-4
tolerance of the reference's tests that a single TF32 or BF16 pass would not.  CPU tensors go
through ``torch.nn.functional.linear``.
"""
from __future__ import annotations

import torch

from . import _lib
from .cbm import _raw_stream


_current_device = torch._C._cuda_getDevice


def _rows(t: torch.Tensor) -> torch.Tensor:
    """Row-major with unit column stride: as is, or a copy.  The maps take rows of any width at any
    pitch; 16-byte aligned ones are read four values at a time."""
    s = t.stride()
    return t if s[1] == 1 and s[0] >= t.size(1) else t.contiguous()


def _new_rows(n: int, width: int, like: torch.Tensor) -> torch.Tensor:
    """An uninitialised [n, width] tensor whose rows are 16-byte aligned."""
    if width % 4 == 0:
        return like.new_empty((n, width))
    return like.new_empty((n, -(-width // 4) * 4))[:, :width]


def _ld(t: torch.Tensor) -> int:
    return max(t.stride(0), t.size(1))


def _check(t: torch.Tensor, u: torch.Tensor, match: bool, what: str) -> None:
    """The kernels read as far as the sizes they are given say: operands that do not fit together are refused here."""
    if not match:
        raise RuntimeError(f"dense map: shape mismatch, {what} of {tuple(t.shape)} and {tuple(u.shape)}")
    if t.device != u.device:
        raise RuntimeError(f"dense map: operands on {t.device} and {u.device}")


def _call(name: str, dev: int, *args) -> None:
    """One library call on device ``dev``'s current stream."""
    fn = getattr(_lib.lib(), name)
    if _current_device() == dev:
        rc = fn(*args, _raw_stream(dev))
    else:
        with torch.cuda.device(dev):
            rc = fn(*args, _raw_stream(dev))
    if rc:
        _lib.check(rc)


def dense_forward(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor | None = None, relu: bool = False,
                  relu_in: bool = False) -> torch.Tensor:
    """``x @ w.T`` (``relu``: followed by ``max(., 0)`` in the GEMM's epilogue; ``relu_in``: of
    ``max(x, 0)``, taken as the operand is read) for CUDA fp32 ``x`` [N, in] and ``w`` [out, in];
    ``out`` (optional) is an [N, out] tensor that receives the result."""
    _check(x, w, x.dim() == 2 and w.dim() == 2 and x.size(1) == w.size(1), "x @ w.T")
    n, n_in, n_out = x.size(0), x.size(1), w.size(0)
    x, w = _rows(x), _rows(w)
    direct = (out is not None and out.shape == (n, n_out) and out.dtype == x.dtype and out.device == x.device
              and out.stride(1) == 1 and out.stride(0) >= n_out)  # anything else is copied to, or refused, by torch
    y = out if direct else _new_rows(n, n_out, x)
    args = (x.data_ptr(), _ld(x), w.data_ptr(), _ld(w), y.data_ptr(), _ld(y), n, n_in, n_out)
    if relu_in:
        _call("cbm_b200_dense_forward_of_relu", x.get_device(), *args, 1 if relu else 0)
    else:
        _call("cbm_b200_dense_forward_relu" if relu else "cbm_b200_dense_forward", x.get_device(), *args)
    return y if out is None or direct else out.copy_(y)


def dense_grad_input(gy: torch.Tensor, w: torch.Tensor, relu_output: torch.Tensor | None = None) -> torch.Tensor:
    """``gy @ w`` for ``gy`` [N, out], ``w`` [out, in].  With ``relu_output`` [N, in] (the output, or
    the input, of the ReLU this gradient flows back through) the result is zeroed where that is <= 0,
    in the GEMM's epilogue."""
    _check(gy, w, gy.dim() == 2 and w.dim() == 2 and gy.size(1) == w.size(0), "gy @ w")
    n, n_out, n_in = gy.size(0), gy.size(1), w.size(1)
    if relu_output is not None:
        _check(gy, relu_output, relu_output.shape == (n, n_in), "gy @ w and its mask")
    gy, w = _rows(gy), _rows(w)
    gx = _new_rows(n, n_in, gy)
    args = (gy.data_ptr(), _ld(gy), w.data_ptr(), _ld(w))
    to = (gx.data_ptr(), _ld(gx), n, n_in, n_out)
    if relu_output is None:
        _call("cbm_b200_dense_grad_input", gy.get_device(), *args, *to)
    else:
        h = _rows(relu_output)
        _call("cbm_b200_dense_grad_input_relu", gy.get_device(), *args, h.data_ptr(), _ld(h), *to)
    return gx


def dense_grad_weight(gy: torch.Tensor, x: torch.Tensor, relu_x: bool = False) -> torch.Tensor:
    """``gy.T @ x`` for ``gy`` [N, out], ``x`` [N, in]: the weight gradient [out, in] (``relu_x``: of
    ``max(x, 0)``).  The partial results of the row ranges go through a workspace from torch's
    allocator, which is stream-ordered: calls on different streams and threads do not share one."""
    _check(gy, x, gy.dim() == 2 and x.dim() == 2 and gy.size(0) == x.size(0), "gy.T @ x")
    n, n_out, n_in = gy.size(0), gy.size(1), x.size(1)
    gy, x = _rows(gy), _rows(x)
    gw = gy.new_empty((n_out, n_in))
    ws = gy.new_empty(_lib.lib().cbm_b200_dense_grad_weight_workspace(n, n_in, n_out) // 4)
    _call("cbm_b200_dense_grad_weight_of_relu" if relu_x else "cbm_b200_dense_grad_weight", gy.get_device(), gy.data_ptr(),
          _ld(gy), x.data_ptr(), _ld(x), gw.data_ptr(), n_in, n, n_in, n_out, ws.data_ptr(), 4 * ws.numel())
    return gw


class _DenseMap(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight):
        ctx.save_for_backward(x, weight)
        return dense_forward(x, weight)

    @staticmethod
    def backward(ctx, gy):
        x, weight = ctx.saved_tensors
        gx = dense_grad_input(gy, weight) if ctx.needs_input_grad[0] else None
        gw = dense_grad_weight(gy, x) if ctx.needs_input_grad[1] else None
        return gx, gw


class _DenseMapRelu(torch.autograd.Function):
    """``relu(x @ w.T)`` with the ReLU in the GEMM's epilogue; the gradient masks with the output."""

    @staticmethod
    def forward(ctx, x, weight):
        h = dense_forward(x, weight, relu=True)
        ctx.save_for_backward(x, weight, h)
        return h

    @staticmethod
    def backward(ctx, gh):
        x, weight, h = ctx.saved_tensors
        gy = torch.ops.aten.threshold_backward(gh, h, 0.0)  # gh where h > 0, else 0: one pass
        gx = dense_grad_input(gy, weight) if ctx.needs_input_grad[0] else None
        gw = dense_grad_weight(gy, x) if ctx.needs_input_grad[1] else None
        return gx, gw


def linear_relu(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``relu(x @ weight.T)`` in fp32 accuracy, differentiable in both arguments."""
    if not x.is_cuda:
        return torch.nn.functional.linear(x, weight).relu()
    if x.dtype != torch.float32 or weight.dtype != torch.float32:
        raise RuntimeError("dense map: fp32 operands expected")
    return _DenseMapRelu.apply(x, weight)


class _ReluMapThenMap(torch.autograd.Function):
    """``relu(p @ w1.T) @ w2.T``: the dense map that ends one layer, the ReLU between two layers and
    the dense map that opens the next one.  Forward: the ReLU in the first map's epilogue.
    Backward: the ReLU's mask in the epilogue of the second map's input gradient, so the hidden
    activations are never passed over by an elementwise kernel in either direction."""

    @staticmethod
    def forward(ctx, p, w1, w2):
        h = dense_forward(p, w1, relu=True)
        ctx.save_for_backward(p, w1, w2, h)
        return dense_forward(h, w2)

    @staticmethod
    def backward(ctx, gu):
        p, w1, w2, h = ctx.saved_tensors
        gw2 = dense_grad_weight(gu, h) if ctx.needs_input_grad[2] else None
        gp = gw1 = None
        if ctx.needs_input_grad[0] or ctx.needs_input_grad[1]:
            gz = dense_grad_input(gu, w2, relu_output=h)  # gradient at the first map's output, before its ReLU
            gp = dense_grad_input(gz, w1) if ctx.needs_input_grad[0] else None
            gw1 = dense_grad_weight(gz, p) if ctx.needs_input_grad[1] else None
        return gp, gw1, gw2


def relu_linear_linear(p: torch.Tensor, w1: torch.Tensor, w2: torch.Tensor) -> torch.Tensor:
    """``relu(p @ w1.T) @ w2.T`` in fp32 accuracy, differentiable in all three arguments."""
    if not p.is_cuda:
        return torch.nn.functional.linear(torch.nn.functional.linear(p, w1).relu(), w2)
    if p.dtype != torch.float32 or w1.dtype != torch.float32 or w2.dtype != torch.float32:
        raise RuntimeError("dense map: fp32 operands expected")
    return _ReluMapThenMap.apply(p, w1, w2)


def linear(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``x @ weight.T`` in fp32 accuracy, differentiable in both arguments."""
    if not x.is_cuda:
        return torch.nn.functional.linear(x, weight)
    if x.dtype != torch.float32 or weight.dtype != torch.float32:
        raise RuntimeError("dense map: fp32 operands expected")
    return _DenseMap.apply(x, weight)
