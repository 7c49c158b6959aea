"""GCN layers on the CBM product: ``forward(x, edge_index) = propagate(lin(x))``.

Mirrors gnns/graph_convolutional_network/cbm_gcn.py:10-75: a bias-free linear map with
Glorot-uniform weights (the reference uses torch_geometric's ``Linear(..., bias=False,
weight_initializer='glorot')``, restated here on ``torch.nn.Linear`` because torch_geometric is not
available offline) followed by the normalized CBM propagation.  ``GCNModel`` restates the stacked
benchmark model of benchmark/parallel/benchmark_gcn_cpu.py:70-89 (ReLU between layers, one CBM
structure shared by every layer).

The dense map and its gradients run on the tensor cores through the library's fp32-accurate GEMMs
(cbm4gnn_b200/dense.py), so that results stay within the 1e-4 tolerance the reference's tests use.
"""
from __future__ import annotations

import torch
from torch import nn

from .cbm import _product
from .dense import dense_forward, dense_grad_input, dense_grad_weight, linear, linear_relu
from .message_passing import CBMCudaMessagePassing


def _fp32_linear(lin: nn.Linear, x: torch.Tensor) -> torch.Tensor:
    return linear(x, lin.weight)


class CBMCudaGCN(CBMCudaMessagePassing):
    """``order``: "lin_first" is the reference's ``propagate(lin(x))`` (cbm_gcn.py:21-24);
    "propagate_first" computes ``lin(propagate(x))``, the same matrix product ``A (X W) = (A X) W``
    with the sparse product running at the input width; "auto" (default) propagates at the
    narrower of the two widths."""

    def __init__(self, in_channels: int, out_channels: int, alpha: int = 2, order: str = "auto"):
        super().__init__(normalize=True, alpha=alpha)
        if order not in ("auto", "lin_first", "propagate_first"):
            raise ValueError("order must be 'auto', 'lin_first' or 'propagate_first'")
        self.in_channels = in_channels
        self.out_channels = out_channels
        self.order = order
        self.lin = nn.Linear(in_channels, out_channels, bias=False)
        self.reset_parameters()

    def reset_parameters(self):
        nn.init.xavier_uniform_(self.lin.weight)  # Glorot-uniform

    def propagate_first(self) -> bool:
        return self.order == "propagate_first" or (self.order == "auto" and self.in_channels < self.out_channels)

    def product_width(self) -> int:
        return self.in_channels if self.propagate_first() else self.out_channels

    def propagate_only(self, x, edge_index):
        """The layer's sparse half alone: ``A_hat @ x``."""
        return CBMCudaMessagePassing.forward(self, edge_index, x=x)

    def forward(self, x, edge_index, relu: bool = False):
        """``relu``: apply the ReLU that follows this layer in a stack; when the dense map comes
        last in the layer it runs in the map's epilogue."""
        if self.propagate_first():
            p = super().forward(edge_index, x=x)
            return linear_relu(p, self.lin.weight) if relu else _fp32_linear(self.lin, p)
        x = _fp32_linear(self.lin, x)
        y = super().forward(edge_index, x=x)
        return y.relu() if relu else y


# Reference class names (cbm_gcn.py:10, 27, 44, 61).
class CBMSequentialMKLCSRSparseMatrixGCN(CBMCudaGCN):
    pass


class CBMParallelMKLCSRSparseMatrixGCN(CBMCudaGCN):
    pass


class CBMSequentialTorchCSRSparseMatrixGCN(CBMCudaGCN):
    two_step = True


class CBMParallelTorchCSRSparseMatrixGCN(CBMCudaGCN):
    two_step = True


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
                kept.append(x)
            x = _product(step, x)
        else:
            if kept is not None:
                kept.append(x)
            x = dense_forward(x, weights[j], relu=k % 2 == 1 and k < last, relu_in=relu and steps[k - 1] is not None)
            j += 1
    return x


class _Stack(torch.autograd.Function):
    """``_stack_forward`` as one differentiable step.  On a graph of a few thousand nodes the kernels of a training
    step take 110 us and everything else is the host's: a function to a layer, or to a map and a product, costs
    more in the two passes than the launches in it (4096 rows, 500-64-7: 285 us a step with four of them, 245 with one)."""

    @staticmethod
    def forward(ctx, x, steps, *weights):
        kept = []
        y = _stack_forward(x, steps, weights, kept)
        ctx.steps = steps
        ctx.save_for_backward(*weights, *kept)
        return y

    @staticmethod
    def backward(ctx, g):
        steps, needs = ctx.steps, ctx.needs_input_grad
        n = len(needs) - 2
        weights, kept = ctx.saved_tensors[:n], ctx.saved_tensors[n:]
        maps = [k for k, step in enumerate(steps) if step is None]
        # the gradient flows down to the features, or to the lowest map that wants one for its weight
        lowest = -1 if needs[0] else next(k for k, need in zip(maps, needs[2:]) if need)
        grads, j = [None] * n, n
        for k in range(len(steps) - 1, max(lowest, 0) - 1, -1):
            step, operand, relu = steps[k], kept[k], k > 0 and k % 2 == 0
            if step is not None:
                g = _product(step.transposed(), g)
                if relu:
                    g = torch.ops.aten.threshold_backward(g, operand, 0.0)
                continue
            j -= 1
            if needs[2 + j]:
                grads[j] = dense_grad_weight(g, operand, relu_x=relu and steps[k - 1] is not None)
            if k > lowest:
                g = dense_grad_input(g, weights[j], relu_output=operand if relu else None)
        return (g if needs[0] else None, None, *grads)


class GCNModel(nn.Module):
    """``len(widths) - 1`` GCN layers with ReLU between them, sharing one CBM structure."""

    def __init__(self, widths, structure=None, alpha: int = 2):
        super().__init__()
        if len(widths) < 3:
            raise ValueError("Number of layers must be at least 2")
        self.layers = nn.ModuleList(CBMCudaGCN(a, b, alpha=alpha) for a, b in zip(widths[:-1], widths[1:]))
        if structure is not None:
            self.share(structure)

    def product_widths(self):
        """Operand width of each layer's sparse product, in layer order."""
        return [layer.product_width() for layer in self.layers]

    def share(self, structure):
        for layer in self.layers:
            layer.cached_a_t = structure

    def forward(self, x, edge_index):
        """Layers of this library's own class run as one step (``_Stack``); where one was replaced, derived from,
        given hooks or told to go by two steps, or off the GPU, layer by layer."""
        layers = list(self.layers)
        if x.is_cuda and x.dtype == torch.float32 and all(map(_plain, layers)):
            steps, weights = [], []
            for layer in layers:
                structure = layer._structure(edge_index, x.dtype, x.device)
                steps += (structure, None) if layer.propagate_first() else (None, structure)
                weights.append(layer.lin.weight)
            if torch.is_grad_enabled() and (x.requires_grad or any(w.requires_grad for w in weights)):
                return _Stack.apply(x, steps, *weights)
            return _stack_forward(x, steps, weights)
        last = len(layers) - 1
        for i, layer in enumerate(layers):
            x = layer(x, edge_index, relu=i < last)
        return x


def _plain(layer) -> bool:
    if type(layer) is not CBMCudaGCN or layer.two_step:
        return False
    w = layer.lin.weight
    return w.is_cuda and w.dtype == torch.float32 and not (
        layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks or layer._backward_pre_hooks)
