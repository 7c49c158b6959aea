"""The dense-map kernels at the edges of their tiles, blocks and passes, against float64."""
import pytest
import torch

from cbm4gnn_b200 import _lib, dense, stack
from cbm4gnn_b200.gcn import GCNModel

pytestmark = pytest.mark.gpu


def _operand(rows, cols, pad, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((rows, cols + pad), generator=g, device="cuda")[:, :cols]


def _close(got, a, b):
    """Within 3e-7 of sum |a||b|, what fp32 accuracy of every product and sum allows."""
    want, scale = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    assert got.shape == want.shape
    assert float(((got.double() - want).abs() / scale.clamp(min=1e-30)).max()) < 3e-7


# rows: one, a tile's edge, more tiles than blocks; widths: one value, edges of the 16-, 32- and 64-deep steps, of the
# 16-, 64- and 128-wide tiles, a contraction of several passes (1433 columns beside 128 results)
@pytest.mark.parametrize("n,n_in,n_out", [(1, 1, 1), (127, 16, 15), (128, 17, 16), (129, 31, 17), (130, 33, 47), (257, 63, 64),
                                          (200, 65, 65), (100, 127, 128), (333, 129, 130), (150, 300, 256), (70, 1433, 128),
                                          (20000, 100, 257)])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_forward_and_gradients_at_tile_edges(n, n_in, n_out, pad):
    x, w, gy = _operand(n, n_in, pad, 1), _operand(n_out, n_in, pad, 2), _operand(n, n_out, pad, 3)
    xr = x.relu()
    _close(dense.dense_forward(x, w), x, w.t())
    _close(dense.dense_forward(x, w, relu_in=True), xr, w.t())
    assert torch.equal(dense.dense_forward(x, w, relu=True), dense.dense_forward(x, w).relu())
    gx = dense.dense_grad_input(gy, w)
    _close(gx, gy, w)
    masked = dense.dense_grad_input(gy, w, relu_output=x)  # the ReLU's input serves as well as its output
    assert torch.equal(masked, torch.where(x > 0, gx, torch.zeros_like(gx)))
    _close(dense.dense_grad_weight(gy, x), gy.t(), x)
    _close(dense.dense_grad_weight(gy, x, relu_x=True), gy.t(), xr)


def test_long_contraction_keeps_its_accuracy():
    """Sums over many rows and columns are carried rounded, not cut off: the result drifts by no more than a few
    units of fp32's last place."""
    x, gy, w = _operand(60000, 256, 0, 4), _operand(60000, 64, 0, 5), _operand(64, 256, 0, 9)
    for got, want in ((dense.dense_grad_weight(gy, x), gy.double().t() @ x.double()),
                      (dense.dense_forward(x, w), x.double() @ w.double().t())):
        assert float((got.double() - want).norm() / want.norm()) < 3e-7


@pytest.mark.parametrize("widths", [(6, 9, 20, 5), (20, 9, 6, 3), (20, 6, 9, 5), (6, 20, 5, 9), (6, 20, 7)])
@pytest.mark.parametrize("listed_bytes", [stack.LISTED_BYTES, 0])
@pytest.mark.parametrize("x_grad,frozen", [(True, ()), (False, ()), (False, (0,)), (True, (0, 1))])
def test_stack_of_layers_and_its_gradients(widths, x_grad, frozen, listed_bytes, monkeypatch):
    """Every order of products and maps next to one another, and gradients that stop at any of the layers,
    against float64 autograd over the dense adjacency; calls issued from a list and one by one."""
    monkeypatch.setattr(stack, "LISTED_BYTES", listed_bytes)
    n = 300
    gen = torch.Generator().manual_seed(sum(widths))
    a = torch.rand((n, n), generator=gen) < 0.03
    a = (a | a.t()).fill_diagonal_(True)
    edges = a.nonzero().t().contiguous()
    model = GCNModel(list(widths), alpha=2).cuda()
    for i in frozen:
        model.layers[i].lin.weight.requires_grad_(False)
    x = torch.randn((n, widths[0]), generator=gen).cuda().requires_grad_(x_grad)
    d = a.sum(1).double().rsqrt()
    adjacency = (d[:, None] * a.double() * d).cuda()
    h = x.double()
    for i, layer in enumerate(model.layers):
        h = adjacency @ h @ layer.lin.weight.double().t()
        h = h.relu() if i < len(model.layers) - 1 else h
    got = model(x, edges.cuda())
    g = torch.randn(got.shape, generator=gen).cuda()
    wrt = [w for w in model.parameters() if w.requires_grad] + ([x] if x_grad else [])
    torch.testing.assert_close(got, h.float(), atol=1e-5, rtol=1e-5)
    with torch.no_grad():
        assert torch.equal(model(x, edges.cuda()), got)
    for p, q in zip(torch.autograd.grad(got, wrt, g), torch.autograd.grad(h, wrt, g.double())):
        torch.testing.assert_close(p, q, atol=1e-4, rtol=1e-4)


def test_nan_passes_through_every_relu():
    """As through torch.relu and its backward: a NaN stays a NaN and lets the gradient through."""
    nan = float("nan")
    x, w, gy = _operand(140, 40, 0, 1), _operand(24, 40, 0, 2), _operand(140, 24, 0, 3)
    x[3, 5] = x[130, 39] = nan
    rows = x.isnan().any(1)
    for got in (dense.dense_forward(x, w, relu=True), dense.dense_forward(x, w, relu_in=True)):
        assert torch.equal(got.isnan(), rows[:, None].expand_as(got))
    gx = dense.dense_grad_input(gy, w)
    assert torch.equal(dense.dense_grad_input(gy, w, relu_output=x), torch.where(x <= 0, torch.zeros_like(gx), gx))
    for a, b in ((gy, x), (x, gy)):  # both orientations of the weight gradient
        assert torch.equal(dense.dense_grad_weight(a, b, relu_x=True).isnan(), (a.t() @ b.relu()).isnan())


@pytest.mark.parametrize("widths", [(6, 9, 20, 5), (20, 9, 6, 3), (20, 6, 9, 5), (6, 20, 5, 9)])
@pytest.mark.parametrize("listed_bytes", [stack.LISTED_BYTES, 0])
def test_nan_in_a_stack_of_layers(widths, listed_bytes, monkeypatch):
    """One NaN feature: outputs and gradients have their NaN where the layers called one by one have them."""
    monkeypatch.setattr(stack, "LISTED_BYTES", listed_bytes)
    n = 60
    gen = torch.Generator().manual_seed(3)
    a = torch.rand((n, n), generator=gen) < 0.02
    edges = (a | a.t()).fill_diagonal_(True).nonzero().t().contiguous().cuda()
    model = GCNModel(list(widths), alpha=2).cuda()
    x = torch.randn((n, widths[0]), generator=gen)
    x[7, 2] = float("nan")
    x = x.cuda().requires_grad_(True)
    wrt = [x, *model.parameters()]
    got = model(x, edges)
    want = x
    for i, layer in enumerate(model.layers):
        want = layer(want, edges)
        want = want.relu() if i < len(model.layers) - 1 else want
    assert 0 < int(want.isnan().any(1).sum()) < n
    torch.testing.assert_close(got, want, atol=1e-5, rtol=1e-5, equal_nan=True)
    g = torch.randn(got.shape, generator=gen).cuda()
    for p, q in zip(torch.autograd.grad(got, wrt, g), torch.autograd.grad(want, wrt, g)):
        torch.testing.assert_close(p, q, atol=1e-4, rtol=1e-4, equal_nan=True)


@pytest.mark.parametrize("listed_bytes", [stack.LISTED_BYTES, 0])
def test_saved_tensor_hooks_that_change_the_layout(listed_bytes, monkeypatch):
    monkeypatch.setattr(stack, "LISTED_BYTES", listed_bytes)
    edges = torch.arange(50).repeat(2, 1).cuda()
    model = GCNModel([20, 9, 6, 3], alpha=2).cuda()
    x = torch.randn(50, 20, device="cuda", requires_grad=True)
    g = torch.randn(50, 3, device="cuda")
    wrt = [x, *model.parameters()]
    want = torch.autograd.grad(model(x, edges), wrt, g)

    def turn(t):
        return t.t().contiguous() if t.dim() == 2 else torch.stack([t, t], 1)

    def turn_back(t):
        return t.t() if t.size(1) != 2 else t[:, 0]

    with torch.autograd.graph.saved_tensors_hooks(turn, turn_back):
        y = model(x, edges)
    for p, q in zip(torch.autograd.grad(y, wrt, g), want):
        assert torch.equal(p, q)


@pytest.mark.parametrize("listed_bytes", [stack.LISTED_BYTES, 0])
def test_forward_mode_is_refused(listed_bytes, monkeypatch):
    """No silent loss of a tangent, whether or not anything asks for a gradient."""
    import torch.autograd.forward_ad as forward_ad
    monkeypatch.setattr(stack, "LISTED_BYTES", listed_bytes)
    edges = torch.arange(50).repeat(2, 1).cuda()
    model = GCNModel([20, 9, 6, 3], alpha=2).cuda().requires_grad_(False)
    x = torch.randn(50, 20, device="cuda")
    want = model(x, edges)
    with forward_ad.dual_level():
        with pytest.raises(RuntimeError, match="jvp"):
            model(forward_ad.make_dual(x, torch.ones_like(x)), edges)
        with torch.no_grad(), pytest.raises(RuntimeError, match="jvp"):
            model(forward_ad.make_dual(x, torch.ones_like(x)), edges)
    for call in (lambda: torch.func.jvp(lambda t: model(t, edges), (x,), (x,)), lambda: torch.func.vmap(lambda t: model(t, edges))(x[None])):
        with pytest.raises(RuntimeError):
            call()
    with torch.no_grad():
        assert torch.equal(model(x, edges), want) and not want.requires_grad


def test_layers_are_called_where_someone_looks_at_them():
    """Hooks for all modules and a forward replaced on one layer see every call."""
    edges = torch.arange(50).repeat(2, 1).cuda()
    model = GCNModel([20, 9, 6, 3], alpha=2).cuda()
    x = torch.randn(50, 20, device="cuda")
    want, seen = model(x, edges), []
    hook = torch.nn.modules.module.register_module_forward_hook(lambda module, args, out: seen.append(type(module)))
    try:
        torch.testing.assert_close(model(x, edges), want)
    finally:
        hook.remove()
    assert seen == [type(model.layers[0])] * 3 + [GCNModel]
    layer = model.layers[1]
    layer.forward = lambda h, edge_index, relu=False: type(layer).forward(layer, h, edge_index, relu) * 0
    assert not model(x, edges).any()


@pytest.mark.parametrize("n,n_in,n_out,bound", [(4096, 64, 64, 7.0e-8), (20000, 128, 256, 7.7e-8), (20000, 256, 64, 9.5e-8)])
def test_error_of_the_maps_and_its_drift(n, n_in, n_out, bound):
    """2-norm error against float64 (measured: 6.3, 7.4 and 9.0e-8) and, what does not average out in the product behind
    a map, its mean towards zero (3.6e-8).  Accumulators of 64 columns, which the tensor cores cut off at
    every step, give 7.9, 7.9 and 8.5e-8, and a mean of 5e-8 and more; the bounds lie between."""
    x, w = _operand(n, n_in, 0, 1), _operand(n_out, n_in, 0, 2)
    gy = _operand(n, n_in, 0, 3)
    for got, want in ((dense.dense_forward(x, w), x.double() @ w.double().t()),
                      (dense.dense_grad_input(gy, w.t().contiguous()), gy.double() @ w.double().t())):
        off = got.double() - want
        assert float(off.norm() / want.norm()) < bound
        assert float((off * want.sign()).mean() / want.abs().mean()) > -4.6e-8


@pytest.mark.parametrize("listed_bytes", [stack.LISTED_BYTES, 0])
@pytest.mark.parametrize("width", [1, 2, 3, 4])
def test_narrow_products_are_contiguous(width, listed_bytes, monkeypatch):
    """A few classes at the end, or a few features in front, of a stack; views of them as of any contiguous tensor."""
    monkeypatch.setattr(stack, "LISTED_BYTES", listed_bytes)
    edges = torch.arange(50).repeat(2, 1).cuda()
    out = GCNModel([8, 6, width], alpha=2).cuda()(torch.randn(50, 8, device="cuda"), edges)
    assert out.is_contiguous() and out.view(-1).shape == (50 * width,)
    x = torch.randn(50, width, device="cuda", requires_grad=True)
    model = GCNModel([width, 8, 5], alpha=2).cuda()
    y = model(x, edges)
    gx, = torch.autograd.grad(y, x, torch.ones_like(y))
    assert gx.is_contiguous() and y.stride() == (8, 1)
    h = (x.double() @ model.layers[0].lin.weight.double().t()).relu()  # (the graph is the identity)
    want, = torch.autograd.grad(h @ model.layers[1].lin.weight.double().t(), x, torch.ones(50, 5, device="cuda").double())
    torch.testing.assert_close(gx, want, atol=1e-5, rtol=1e-5)
    assert model.layers[0].cached_a_t.matmul(x).is_contiguous()


@pytest.mark.parametrize("n,n_in,n_out", [(18944, 16, 4), (18945, 17, 33), (18975, 40, 47), (19000, 64, 48), (20001, 33, 64), (19071, 100, 100),
                                          (19072, 16, 112), (19073, 64, 200), (18816, 31, 256), (38000, 70, 96)])
@pytest.mark.parametrize("relu", [False, True])
def test_results_go_out_in_boxes_and_value_by_value_alike(n, n_in, n_out, relu):
    """From a tile for every SM on (148 x 128 rows) rows that are 16-byte aligned leave in boxes of 32 x 32 (cut off at the
    last row and column), others value by value: the same bits, and nothing beside the columns is written."""
    x, w = _operand(n, n_in, 0, 1), _operand(n_out, n_in, 0, 2)
    fn = _lib.lib().cbm_b200_dense_forward_relu if relu else _lib.lib().cbm_b200_dense_forward
    got = []
    for pitch in (-(-n_out // 4) * 4 + 4, -(-n_out // 4) * 4 + 1):
        room = torch.full((n + 1, pitch), 7.0, device="cuda")
        _lib.check(fn(x.data_ptr(), n_in, w.data_ptr(), n_in, room.data_ptr(), pitch, n, n_in, n_out,
                      torch.cuda.current_stream().cuda_stream))
        assert torch.all(room[:n, n_out:] == 7.0) and torch.all(room[n] == 7.0)
        got.append(room[:n, :n_out])
    assert torch.equal(*got)
    want, scale = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    want = want.clamp(min=0) if relu else want
    assert float(((got[0].double() - want).abs() / scale.clamp(min=1e-30)).max()) < 3e-7  # (as _close)
