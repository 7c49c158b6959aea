"""Performance cases of the CBM engine: the calls a user's program makes, over the range of sizes it makes them at.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes
what a program holds before the call (graph, structure, plan, operands, model), ``run`` is one pass through
the public entry points, ``work`` the bytes and operations that pass cannot do without and ``tolerance`` how
far another correct implementation at the same precision may be off.

Graphs are made on the GPU, from the seed alone, with the two shapes that ``cbm4gnn_b200/graphs.py`` uses for
the benchmark configurations (its generators walk node by node on the host, which is too slow to repeat):
"copy" is the vertex-copying model (heavy-tailed degrees, rows that resemble one another), "sbm" the
stochastic block model (communities of lognormal size, few links between them).
"""
from __future__ import annotations

import math

import torch

from cbm4gnn_b200.cbm import aligned_rows, cbm_matrix, csr_matrix_plan
from cbm4gnn_b200.gcn import GCNModel
from cbm4gnn_b200.utility import normalize_edge_index

DEGREE_CAP = 5000  # most links a node of the copy model receives, as in the second benchmark configuration


# ---------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # A few hundred nodes' worth of work: what a unit-test-sized or batched-subgraph caller sees, where
        # only latency counts.
        dict(name="product_tiny", kind="product", graph="copy", n=1000, p_copy=0.8, links=3, alpha=2,
             normalized=True, f=16, pitched=False),
        # First benchmark configuration: plain A X on a small graph with a wide operand.
        dict(name="product_small_plain", kind="product", graph="copy", n=4096, p_copy=0.8, links=3, alpha=0,
             normalized=False, f=500, pitched=False),
        # Second benchmark configuration, the headline: normalized product, operands pitched to whole lines.
        dict(name="product_wide", kind="product", graph="copy", n=100_000, p_copy=0.7, links=5, alpha=8,
             normalized=True, f=500, pitched=True),
        # Fourth benchmark configuration's kind of graph (rows of hundreds of entries, strongly compressed,
        # deep tree), at a size that is built in well under a second.
        dict(name="product_dense_rows", kind="product", graph="copy", n=40_000, p_copy=0.95, links=20, alpha=4,
             normalized=True, f=128, pitched=False),
        # Fifth benchmark configuration's last layer: community graph, 47 columns (odd width, rows that are
        # not 16-byte aligned), operand as the caller's plain tensor.
        dict(name="product_ragged", kind="product", graph="sbm", n=400_000, deg_in=20.0, deg_out=5.0, mu=3.5,
             sigma=1.0, alpha=2, normalized=True, f=47, pitched=False),
        # The reference's *_torch_csr_* methods: delta product, then the tree update in place.
        dict(name="two_step", kind="two_step", graph="copy", n=50_000, p_copy=0.7, links=5, alpha=8,
             normalized=True, f=64, pitched=False),
        # The uncompressed matrix through a CSR plan: the comparison the reference's benchmark makes.
        dict(name="csr_plan", kind="csr", graph="copy", n=100_000, p_copy=0.7, links=5, alpha=0, normalized=True,
             f=128, pitched=False),
        # Drop-in use: host tensors in, host tensors out, the call stages them through the GPU (page-locked,
        # as the benchmark's end-to-end figure has them).
        dict(name="host_operands", kind="host", graph="copy", n=100_000, p_copy=0.7, links=5, alpha=8,
             normalized=True, f=500, pinned=True),
        # Third benchmark configuration: training step of the 2-layer GCN, gradients of both weights and the
        # input features.
        dict(name="gcn_train", kind="train", graph="sbm", n=235_868, deg_in=8.0, deg_out=2.0, mu=4.5, sigma=0.8,
             alpha=2, normalized=True, widths="128,256,64", x_grad=True),
        # The same step on a small graph with a few classes: launches and host work count. Features carry no
        # gradient, the usual case in training.
        dict(name="gcn_train_small", kind="train", graph="copy", n=4096, p_copy=0.8, links=3, alpha=2,
             normalized=True, widths="500,64,7", x_grad=False),
        # Fifth benchmark configuration's forward pass (3 layers), on a graph of the same kind.
        dict(name="gcn_infer", kind="infer", graph="sbm", n=400_000, deg_in=20.0, deg_out=5.0, mu=3.5, sigma=1.0,
             alpha=2, normalized=True, widths="100,256,256,47"),
        # Building the structure for a new graph, candidate search on the GPU as the layers do it.
        dict(name="build", kind="build", graph="copy", n=100_000, p_copy=0.7, links=5, alpha=8, normalized=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "product", "two_step", "csr", "host", "train", "train", "infer", "build"])
    sbm = kind in ("train", "infer") and rng.random() < 0.7 or kind in ("product", "two_step", "csr") and rng.random() < 0.4
    case = dict(kind=kind, graph="sbm" if sbm else "copy")
    if sbm:
        case.update(n=_log(rng, 1000, 300_000), deg_in=round(rng.uniform(6.0, 20.0), 1), deg_out=round(rng.uniform(1.0, 5.0), 1),
                    mu=round(rng.uniform(3.5, 4.5), 2), sigma=round(rng.uniform(0.8, 1.0), 2), alpha=2)
    elif kind == "product" and rng.random() < 0.3:  # long rows
        case.update(n=_log(rng, 5000, 40_000), p_copy=0.95, links=20, alpha=rng.choice([0, 4, 16]))
    else:
        case.update(n=_log(rng, 500, 100_000), p_copy=round(rng.uniform(0.6, 0.8), 2), links=rng.randint(3, 5),
                    alpha=rng.choice([0, 2, 8]))
    case["normalized"] = True if kind in ("train", "infer", "csr") else rng.random() < 0.7
    room = 100_000 * 500  # operand elements of the largest listed product
    if kind in ("product", "two_step", "csr"):
        case.update(f=min(_log(rng, 1, 512), room // case["n"]), pitched=rng.random() < 0.3)
    elif kind == "host":
        case.update(f=_log(rng, 8, 500), pinned=rng.random() < 0.5)
    elif kind in ("train", "infer"):
        layers = 2 if kind == "train" else 3
        widths = [_log(rng, 16, 512)] + [_log(rng, 16, 256) for _ in range(layers - 1)] + [_log(rng, 4, 64)]
        while case["n"] * sum(widths) > 235_868 * 448:
            widths[widths.index(max(widths))] = max(widths) // 2
        case["widths"] = ",".join(map(str, widths))
        if kind == "train":
            case["x_grad"] = rng.random() < 0.5
    return case


# --------------------------------------------------------------------------------------------- graphs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _undirected(src, dst, n, self_loops):
    """Both directions, no duplicates, sorted by (row, column); self loops dropped, or one per node."""
    keep = src != dst
    src, dst = src[keep], dst[keep]
    keys = [src * n + dst, dst * n + src]
    if self_loops:
        keys.append(torch.arange(n, device=src.device) * (n + 1))
    key = torch.unique(torch.cat(keys))
    return torch.stack([key // n, key % n])


def _ragged(start, count):
    """Flat positions start[i] .. start[i] + count[i] - 1, and the i each belongs to."""
    owner = torch.repeat_interleave(torch.arange(count.numel(), device=count.device), count)
    first = torch.cumsum(count, 0) - count
    return start[owner] + torch.arange(owner.numel(), device=count.device) - first[owner], owner


def _copy_model(n, p_copy, links, gen):
    """Each new node repeats every link that an earlier node made when it joined with probability p_copy and
    adds ``links`` uniform ones; nodes join in batches of an eighth of those already there."""
    dev = gen.device
    flat = torch.zeros(0, dtype=torch.int64, device=dev)  # links in joining order
    start = torch.zeros(n, dtype=torch.int64, device=dev)
    count = torch.zeros(n, dtype=torch.int64, device=dev)
    degree = torch.zeros(n, dtype=torch.int64, device=dev)
    have = 1
    while have < n:
        k = min(max(1, have // 8), n - have)
        proto = torch.randint(0, have, (k,), generator=gen, device=dev)
        at, owner = _ragged(start[proto], count[proto])
        kept = torch.rand(at.numel(), generator=gen, device=dev) < p_copy
        extra = torch.randint(0, have, (k * links,), generator=gen, device=dev)
        own = torch.cat([owner[kept], torch.arange(k, device=dev).repeat_interleave(links)])
        to = torch.cat([flat[at[kept]], extra])
        free = degree[to] < DEGREE_CAP
        key = torch.unique(own[free] * n + to[free])
        own, to = key // n, key % n
        made = torch.bincount(own, minlength=k)
        start[have:have + k] = flat.numel() + torch.cumsum(made, 0) - made
        count[have:have + k] = made
        degree += torch.bincount(to, minlength=n)
        degree[have:have + k] += made
        flat = torch.cat([flat, to])
        have += k
    return torch.repeat_interleave(torch.arange(n, device=dev), count), flat


def _block_model(n, mu, sigma, deg_in, deg_out, gen):
    dev = gen.device
    n_comm = max(2, int(n / math.exp(mu + sigma * sigma / 2)))
    raw = torch.exp(mu + sigma * torch.randn(n_comm, generator=gen, device=dev, dtype=torch.float64))
    ends = (torch.cumsum(raw, 0) * (n / raw.sum())).round().to(torch.int64).clamp(max=n)
    ends[-1] = n
    begins = torch.cat([ends.new_zeros(1), ends[:-1]])
    m_in, m_out = int(n * deg_in / 2), int(n * deg_out / 2)
    src = torch.randint(0, n, (m_in,), generator=gen, device=dev)
    comm = torch.searchsorted(ends, src, right=True)
    size = ends[comm] - begins[comm]
    dst = begins[comm] + (torch.rand(m_in, generator=gen, device=dev, dtype=torch.float64) * size).to(torch.int64)
    far = torch.randint(0, n, (2, m_out), generator=gen, device=dev)
    label = torch.randperm(n, generator=gen, device=dev)  # communities are not contiguous in node id
    return label[torch.cat([src, far[0]])], label[torch.cat([dst, far[1]])]


def _edges(case, gen):
    n = case["n"]
    if case["graph"] == "copy":
        src, dst = _copy_model(n, case["p_copy"], case["links"], gen)
    else:
        src, dst = _block_model(n, case["mu"], case["sigma"], case["deg_in"], case["deg_out"], gen)
    return _undirected(src, dst, n, self_loops=case["normalized"])


def _structure(case, edges):
    m = cbm_matrix(edges.to(torch.int32), torch.ones(edges.size(1)), alpha=case["alpha"],
                   normalized=case["normalized"], build_device=torch.cuda.current_device())
    m.plan()
    return m


# ---------------------------------------------------------------------------------------- the interface
def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "build":
        # On the host, as the caller read the graph. One graph for each case under the seed's node numbers: the
        # arrays of the structure then come out equally long (their total is the optimum, whatever the numbering).
        label = torch.randperm(case["n"], generator=gen, device="cuda")
        edges = _undirected(*label[_edges(case, _gen(0))], case["n"], self_loops=case["normalized"])
        return dict(case=case, edges=edges.to(torch.int32).cpu(), values=torch.ones(edges.size(1)))
    edges = _edges(case, gen)
    if kind == "csr":
        n = case["n"]
        val = normalize_edge_index(edges, n)
        crow = torch.zeros(n + 1, dtype=torch.int64, device=edges.device)
        crow[1:] = torch.cumsum(torch.bincount(edges[0], minlength=n), 0)
        m = csr_matrix_plan(crow, edges[1], val, n)
        rows = n
    else:
        m = _structure(case, edges)
        rows = m.num_rows
    state = dict(case=case, matrix=m)
    if kind in ("train", "infer"):
        widths = [int(w) for w in case["widths"].split(",")]
        torch.manual_seed(seed)
        state["edges"] = edges
        state["model"] = GCNModel(widths, structure=m, alpha=case["alpha"]).cuda()
        state["x"] = torch.randn((rows, widths[0]), generator=gen, device="cuda")
        if kind == "train":
            state["x"].requires_grad_(case["x_grad"])
            state["gy"] = torch.randn((rows, widths[-1]), generator=gen, device="cuda")  # gradient of the loss
        return state
    x = torch.randn((rows, case["f"]), generator=gen, device="cuda")
    if kind == "host":
        state["x"] = torch.empty(x.shape, pin_memory=case["pinned"]).copy_(x)
        state["y"] = torch.empty(x.shape, pin_memory=case["pinned"])
        return state
    if case["pitched"]:
        state["x"], state["y"] = aligned_rows(rows, case["f"], "cuda"), aligned_rows(rows, case["f"], "cuda")
        state["x"].copy_(x)
    else:
        state["x"], state["y"] = x, torch.empty_like(x)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product" or kind == "host":
        x, y, m = state["x"], state["y"], state["matrix"]
        if case["normalized"]:
            m.omp_mkl_csr_fused_spmm_update(x, y)
        else:
            m.omp_mkl_csr_spmm_update(x, y)
        return y
    if kind == "two_step":
        m = state["matrix"]
        return m.omp_torch_csr_fused_matmul(state["x"]) if case["normalized"] else m.omp_torch_csr_matmul(state["x"])
    if kind == "csr":
        return state["matrix"].matmul(state["x"], out=state["y"])
    if kind == "train":
        model, x = state["model"], state["x"]
        out = model(x, state["edges"])
        wrt = list(model.parameters()) + ([x] if case["x_grad"] else [])
        return [out.detach(), *torch.autograd.grad(out, wrt, state["gy"])]
    if kind == "infer":
        with torch.no_grad():
            return state["model"](state["x"], state["edges"])
    m = cbm_matrix(state["edges"], state["values"], alpha=case["alpha"], normalized=case["normalized"],
                   build_device=torch.cuda.current_device())
    return [m.mst_row, m.mst_col, m.deltas.crow_indices(), m.deltas.col_indices(), m.deltas.values()]


def _entries(case):
    """Expected stored entries of the matrix."""
    n = case["n"]
    if case["graph"] == "sbm":
        d = case["deg_in"] + case["deg_out"]
    else:  # links per joining node: ``links`` new ones and p_copy times an earlier node's
        mean, have = 0.0, 1
        while have < n:
            k = min(max(1, have // 8), n - have)
            mean += (min(case["links"] + case["p_copy"] * mean, have) - mean) * k / (have + k)
            have += k
        d = 2 * mean
    return n * (d + (1 if case["normalized"] else 0))


def work(case):
    n, nnz, kind = case["n"], _entries(case), case["kind"]
    index = 8 * nnz + 24 * n  # column and value of each entry, row bounds, tree, multiplier
    if kind == "build":
        return {"bytes": 8 * nnz + index, "flops": nnz}
    if kind in ("train", "infer"):
        w = [int(v) for v in case["widths"].split(",")]
        maps = sum(2 * n * a * b for a, b in zip(w[:-1], w[1:]))
        products = sum(2 * nnz * min(a, b) for a, b in zip(w[:-1], w[1:]))
        if kind == "infer":
            return {"bytes": index + 4 * n * (w[0] + w[-1]) + 4 * sum(a * b for a, b in zip(w[:-1], w[1:])),
                    "flops": maps + products}
        # forward, weight gradients, gradients that flow back (down to the features where asked); the hidden
        # activations are kept from the forward to the backward pass
        first = 2 * n * w[0] * w[1]
        flops = 3 * maps - (0 if case["x_grad"] else first) + 2 * products
        bytes_ = index + 4 * n * (w[0] * (2 if case["x_grad"] else 1) + 2 * w[-1] + 2 * sum(w[1:-1]))
        return {"bytes": bytes_ + 8 * sum(a * b for a, b in zip(w[:-1], w[1:])), "flops": flops}
    return {"bytes": index + 8 * n * case["f"], "flops": 2 * nnz * case["f"]}


def tolerance(case):
    if case["kind"] == "build":
        return "exact"
    if case["kind"] == "train":
        # The mask of the ReLU between the layers follows the sign of a 32-bit sum. Of the values that lie within
        # rounding of zero (about 1e-7 of them) the mask, hence that value's whole gradient, may go either way:
        # sqrt(2e-7) = 5e-4 of the 2-norm of the gradients, and a single value of them by a good part of its size.
        return {"rel": 1e-3, "max": 0.5}
    return {"rel": 1e-5, "max": 1e-4}
