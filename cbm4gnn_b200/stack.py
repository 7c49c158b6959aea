"""The layers of a GCN stack (benchmark/parallel/benchmark_gcn_cpu.py:70-89) run as one differentiable step.

A stack is a list of ``steps``, two to a layer, in the order in which they run: a ``cbm_matrix`` stands for
its product, ``None`` for the dense map by the next of ``weights``; a ReLU lies between every two layers.
"""
from __future__ import annotations

import functools
from array import array

import torch
from torch.autograd import forward_ad

from . import _lib
from .cbm import _product, _raw_stream, result_pitch
from .dense import dense_forward, dense_grad_input, dense_grad_weight


def _stack_forward(x, steps, weights, kept=None):
    """A stack of layers as one list of ``steps``, two to a layer: a structure stands for its product, ``None``
    for the dense map by the next of ``weights``.  The ReLU in front of every layer but the first is taken by the
    map before it as it stores, else by the map after it as it reads, and is a pass of its own only between two
    products.  ``kept`` receives the operand of every step."""
    last, j = len(steps) - 1, 0
    for k, step in enumerate(steps):
        relu = k > 0 and k % 2 == 0  # a ReLU in front of this step
        if step is not None:
            if relu and steps[k - 1] is not None:
                x = x.relu()
            if kept is not None:
                kept.append(x if relu else None)  # (for the mask)
            x = _product(step, x)
        else:
            if kept is not None:
                kept.append(x)
            x = dense_forward(x, weights[j], relu=k % 2 == 1 and k < last, relu_in=relu and steps[k - 1] is not None)
            j += 1
    return x


class _Stack(torch.autograd.Function):
    """``_stack_forward`` as one differentiable step.  A function to a layer, or to a map and a product, costs the
    host more in the two passes than the launches in it (4096 rows, 500-64-7: 285 us a training step with four of
    them, 245 with one)."""

    @staticmethod
    def forward(ctx, x, steps, keep, *weights):
        """``keep``: a backward pass may follow; the operands of the steps are let go as they are used up otherwise."""
        if not keep:
            return _stack_forward(x, steps, weights)
        kept = []
        y = _stack_forward(x, steps, weights, kept)
        ctx.steps = steps
        ctx.save_for_backward(*weights, *kept)
        return y

    @staticmethod
    def backward(ctx, g):
        steps, needs = ctx.steps, ctx.needs_input_grad
        n, saved = len(needs) - 3, ctx.saved_tensors
        weights, kept = saved[:n], saved[n:]
        maps = [k for k, step in enumerate(steps) if step is None]
        # the gradient flows down to the features, or to the lowest map that wants one for its weight
        lowest = -1 if needs[0] else next(k for k, need in zip(maps, needs[3:]) if need)
        grads, j = [None] * n, n
        for k in range(len(steps) - 1, max(lowest, 0) - 1, -1):
            step, operand, relu = steps[k], kept[k], k > 0 and k % 2 == 0
            if step is not None:
                g = _product(step.transposed(), g)
                if relu:
                    g = torch.ops.aten.threshold_backward(g, operand, 0.0)
                continue
            j -= 1
            if needs[3 + j]:
                grads[j] = dense_grad_weight(g, operand, relu_x=relu and steps[k - 1] is not None)
            if k > lowest:
                g = dense_grad_input(g, weights[j], relu_output=operand if relu else None)
        return (g if needs[0] else None, None, None, *grads)


# ------------------------------------------------------------------------------- small graphs: listed calls
# Up to this many bytes of intermediate results the kernels of a pass are shorter than the Python that allocates
# for and issues them one by one (4096 rows, 500-64-7: 110 us of 245; 167 us with the lists).  The calls of a pass are then listed once
# for its sizes and issued by one library call, all intermediate results in one allocation.  Above it the host is
# ahead of the GPU anyway, and single allocations let go of what the backward pass does not read.
LISTED_BYTES = 64 << 20
_PRODUCT, _MAP, _GRAD_INPUT, _GRAD_WEIGHT, _WORDS = 0, 1, 2, 3, 13  # include/cbm_b200.h, cbm_b200_sequence


class _List:
    """Calls for ``cbm_b200_sequence``; ``room`` hands out pieces of the pass's one allocation, base ``base``."""

    def __init__(self, base):
        self.calls, self.base, self.floats = array("q"), base, 0

    def room(self, floats):
        at = self.base + (self.floats << 10)  # 256 x 4 bytes
        self.floats += -(-floats // 64) * 64
        return at

    def add(self, *words):
        self.calls.extend(words + (0,) * (_WORDS - len(words)))

    def issue(self, dev, bases):
        bases = array("q", bases)
        args = self.calls.buffer_info()[0], len(self.calls) // _WORDS, bases.buffer_info()[0], len(bases)
        if torch._C._cuda_getDevice() == dev:
            rc = _lib.lib().cbm_b200_sequence(*args, _raw_stream(dev))
        else:
            with torch.cuda.device(dev):
                rc = _lib.lib().cbm_b200_sequence(*args, _raw_stream(dev))
        if rc:
            _lib.check(rc)


def _pitch(width):
    return -(-width // 4) * 4


def _pitch_out(width, step):
    """Row pitch of what ``step`` leaves for the caller: as the product or the map called by itself."""
    return _pitch(width) if step is None else result_pitch(width)


@functools.lru_cache(maxsize=128)
def _forward_list(steps, shapes, n, ldx):
    """``steps``: (plan, normalized) or None; ``shapes``: of the weights.  Bases: x, the allocation, the result, the
    weights.  Also the place, leading dimension and width of every step's operand."""
    out, at, width, j, operands = _List(1), (0, ldx), shapes[0][1], 0, []
    last = len(steps) - 1
    for k, step in enumerate(steps):
        operands.append((*at, width))
        after = width if step else shapes[j][0]
        to = (out.room(n * _pitch(after)), _pitch(after)) if k < last else (2, _pitch_out(after, step))
        if step:
            out.add(_PRODUCT, step[0], *at, *to, width, step[1])
        else:
            relu_in = k > 0 and k % 2 == 0 and steps[k - 1] is not None
            out.add(_MAP, *at, 3 + j, width, *to, n, width, after, relu_in, k % 2 == 1 and k < last)
            j += 1
        at, width = to, after
    return out, operands


@functools.lru_cache(maxsize=128)
def _backward_list(steps, shapes, n, ldx, ldg, needs):
    """``steps`` with the plans of the transposed structures, ``needs``: which of x and the weights want a gradient.
    Bases: x, the forward pass's allocation, the gradient that comes in, this pass's allocation, the gradient of
    x, the weights, their gradients."""
    operands = _forward_list(steps, shapes, n, ldx)[1]
    maps = [k for k, step in enumerate(steps) if step is None]
    lowest = -1 if needs[0] else next(k for k, need in zip(maps, needs[1:]) if need)
    out, at, j = _List(3), (2, ldg), len(shapes)
    for k in range(len(steps) - 1, max(lowest, 0) - 1, -1):
        step, (place, ld, width), relu = steps[k], operands[k], k > 0 and k % 2 == 0
        to = None
        if k > lowest:
            to = (out.room(n * _pitch(width)), _pitch(width)) if k else (4, _pitch_out(width, step))
        if step:
            out.add(_PRODUCT, step[0], *at, *to, width, step[1])
        else:
            j -= 1
            after = shapes[j][0]
            if needs[1 + j]:
                space = _lib.lib().cbm_b200_dense_grad_weight_workspace(n, width, after)
                out.add(_GRAD_WEIGHT, *at, place, ld, 5 + len(shapes) + j, width, n, width, after,
                        relu and steps[k - 1] is not None, out.room(space // 4), space)
            if to:
                out.add(_GRAD_INPUT, *at, 5 + j, width, *((place, ld) if relu else (-1, 0)), *to, n, width, after)
        at = to
    return out


def _plans(structures, dev):
    return tuple(None if s is None else ((s._plans.get(dev) or s.plan(dev)).handle.value, s.col_multiplier is not None)
                 for s in structures)


def _rows_of(t):
    s = t.stride()
    return t if s[1] == 1 and s[0] >= t.size(1) else t.contiguous()


def _listed_forward(x, steps, shapes, weights):
    dev, n, x = x.get_device(), x.size(0), _rows_of(x)
    calls, _ = _forward_list(_plans(steps, dev), shapes, n, max(x.stride(0), x.size(1)))
    # a stack ends in a map to this width, or in a product of it
    width = shapes[-1][0]
    pitch = _pitch_out(width, steps[-1])
    y, space = x.new_empty((n, pitch)), x.new_empty(calls.floats)
    calls.issue(dev, [x.data_ptr(), space.data_ptr(), y.data_ptr(), *(w.data_ptr() for w in weights)])
    return (y if width == pitch else y[:, :width]), x, space


class _ListedStack(torch.autograd.Function):
    """``_Stack`` with the calls of each pass issued as one."""

    @staticmethod
    def forward(ctx, x, steps, shapes, *weights):
        y, x, space = _listed_forward(x, steps, shapes, weights)
        ctx.steps, ctx.shapes = steps, shapes
        ctx.save_for_backward(x, space, *weights)
        return y

    @staticmethod
    def backward(ctx, g):
        x, kept, *weights = ctx.saved_tensors
        # (a saved-tensor hook may hand them back in another layout)
        x, kept, weights = _rows_of(x), kept.contiguous(), [w.contiguous() for w in weights]
        shapes, needs = ctx.shapes, ctx.needs_input_grad
        dev, n, width, g = x.get_device(), x.size(0), x.size(1), _rows_of(g)
        calls = _backward_list(_plans([None if s is None else s.transposed() for s in ctx.steps], dev), shapes, n, max(x.stride(0), width),
                               max(g.stride(0), g.size(1)), (needs[0], *needs[3:]))
        space = x.new_empty(calls.floats)
        pitch = _pitch_out(width, ctx.steps[0])
        gx = x.new_empty((n, pitch)) if needs[0] else None
        gws = [x.new_empty(shape) if need else None for shape, need in zip(shapes, needs[3:])]
        calls.issue(dev, [x.data_ptr(), kept.data_ptr(), g.data_ptr(), space.data_ptr(), gx.data_ptr() if needs[0] else 0,
                          *(w.data_ptr() for w in weights), *(0 if gw is None else gw.data_ptr() for gw in gws)])
        if needs[0] and width != pitch:
            gx = gx[:, :width]
        return (gx, None, None, *gws)


def _listable(x, steps, shapes, weights):
    """Small, nothing between the calls but other calls (no ReLU in front of a product), operands that fit together."""
    n, width = x.shape if x.dim() == 2 else (0, 0)
    if n == 0 or 4 * n * (width + sum(2 * a for a, _ in shapes)) > LISTED_BYTES or any(s is not None for s in steps[2::2]):
        return False
    for (after, before), w in zip(shapes, weights):
        if before != width or not w.is_contiguous() or w.device != x.device:
            return False
        width = after
    return all(step is None or step.num_rows == n for step in steps)


def run_stack(x, steps, weights):
    """The result of the stack for CUDA fp32 ``x`` and ``weights``, differentiable in both.  Its function is gone round
    only where neither a backward pass can follow nor forward-mode differentiation is going on, which has to meet (and
    be refused by) it: applying a function to three layers takes the host 10 us of 55."""
    shapes = tuple(tuple(w.shape) for w in weights)
    keep = torch.is_grad_enabled() and (x.requires_grad or any(w.requires_grad for w in weights))
    listed = _listable(x, steps, shapes, weights)
    if keep or forward_ad._current_level >= 0:
        return _ListedStack.apply(x, steps, shapes, *weights) if listed else _Stack.apply(x, steps, keep, *weights)
    return _listed_forward(x, steps, shapes, weights)[0] if listed else _stack_forward(x, steps, weights)
