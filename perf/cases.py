"""The calls this framework is timed on: hierarchical Tucker (HT) decomposition
of dense tensors, the operations on a tensor held in HT format, and the HT
tensor layer, each through the package's public entry points.

``listed()`` are fixed cases, ``draw(rng)`` gives one more of the same ranges.
``prepare`` makes the inputs on the GPU from the seed, ``run`` is one call as a
user's program makes it, ``work`` the bytes and operations the call cannot do
without, ``exact`` the same outputs in 64 bits where they have such values
(leaf bases and transfer tensors are determined up to the signs of their
columns, so only the relative error of a decomposition has one).

A decomposed tensor is a signal of as many orthogonal components as the tree's
rank, of weights that fall linearly, plus 1e-2 relative Gaussian noise, so that
the bases are determined by the data.
"""
import numpy as np
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

NOISE = 1e-2


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one small tensor, as in a sweep over many of them: latency and launches
        _d3("d3_small_bf16", (48, 40, 56), 8, "bf16", "reference", True),
        # an ordinary tensor on the other root split, with the error reported
        _d3("d3_256_bf16", (256, 256, 256), 16, "bf16", "left_first", True),
        # ragged sizes on the plain FP32 path (the precision of the layer's initialisation)
        _d3("d3_ragged_fp32", (301, 260, 397), 24, "fp32", "reference", True),
        # the largest resident tensor of the benchmark
        _d3("d3_1024_bf16", (1024, 1024, 1024), 32, "bf16", "reference", False),
        # a long first mode, where the range finder replaces the mode Grams
        _d3("d3_sketch_bf16", (2560, 160, 144), 16, "bf16", "reference", False, leaf="sketch"),
        # the benchmark's 4th-order tensor, balanced tree
        _d4("d4_128_bf16", (128, 128, 128, 128), 24, 48, "bf16", False),
        # the benchmark's batch of small uneven tensors
        _batch("batch_512_bf16", 512, 32, 160, 31, "bf16"),
        # training step of a small fully connected layer, default precision
        _layer("layer_1024_fp32_b128", (8, 8, 16), (8, 8, 16), 16, 128, "fp32"),
        # the same layer at a large batch
        _layer("layer_1024_fp32_b8192", (8, 8, 16), (8, 8, 16), 16, 8192, "fp32"),
        # training step of a large classifier layer on BF16 operands
        _layer("layer_6400_bf16_b4096", (16, 16, 25), (16, 16, 16), 16, 4096, "bf16"),
        # the full tensor back from its HT format
        _recon("reconstruct_1024", (1024, 1024, 1024), 32),
        # single entries of a tensor in HT format
        _entries("entries_1m_1024", (1024, 1024, 1024), 32, 1 << 20),
    ]


def _d3(name, dims, rank, precision, tree, error, leaf="gram"):
    c = {"kind": "d3", "n1": dims[0], "n2": dims[1], "n3": dims[2], "rank": rank, "precision": precision,
         "tree": tree, "error": error, "leaf": leaf}
    return dict(c, name=name) if name else c


def _d4(name, dims, rank, inner, precision, error):
    c = {"kind": "d4", "n1": dims[0], "n2": dims[1], "n3": dims[2], "n4": dims[3], "rank": rank, "inner": inner,
         "precision": precision, "error": error}
    return dict(c, name=name) if name else c


def _batch(name, count, lo, hi, family, precision):
    c = {"kind": "batch", "count": count, "lo": lo, "hi": hi, "family": family, "precision": precision}
    return dict(c, name=name) if name else c


def _layer(name, n, m, rank, batch, precision):
    c = {"kind": "layer", "N0": n[0], "N1": n[1], "N2": n[2], "M0": m[0], "M1": m[1], "M2": m[2], "rank": rank,
         "batch": batch, "precision": precision}
    return dict(c, name=name) if name else c


def _recon(name, dims, rank):
    c = {"kind": "reconstruct", "n1": dims[0], "n2": dims[1], "n3": dims[2], "rank": rank}
    return dict(c, name=name) if name else c


def _entries(name, dims, rank, count):
    c = {"kind": "entries", "n1": dims[0], "n2": dims[1], "n3": dims[2], "rank": rank, "count": count}
    return dict(c, name=name) if name else c


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["d3", "d3", "d3", "d3", "d4", "batch", "layer", "layer", "reconstruct", "entries"])
    if kind == "d3":
        precision = rng.choice(["bf16", "bf16", "fp32"])
        # edges around a common size; the volume of the FP32 path's tensors is smaller
        edge = _log(rng, 40, 320 if precision == "fp32" else 720)
        dims = [max(36, int(edge * rng.uniform(0.7, 1.35))) for _ in range(3)]
        if rng.random() < 0.5:
            dims = [(d + 7) // 8 * 8 for d in dims]
        rank = min(rng.randint(6, 32), min(dims) // 2)
        return _d3("", dims, rank, precision, rng.choice(["reference", "reference", "left_first", "middle"]),
                   rng.random() < 0.5, "sketch" if precision == "bf16" and rng.random() < 0.15 else "gram")
    if kind == "d4":
        dims = [_log(rng, 24, 112) for _ in range(4)]
        if rng.random() < 0.5:
            dims = [(d + 7) // 8 * 8 for d in dims]
        rank = rng.randint(5, min(24, min(dims) // 2))
        return _d4("", dims, rank, min(2 * rank, 48), rng.choice(["bf16", "bf16", "fp32"]), rng.random() < 0.3)
    if kind == "batch":
        lo = rng.randint(32, 64)
        return _batch("", _log(rng, 8, 384), lo, rng.randint(lo + 16, 160), rng.randint(1, 1 << 20),
                      rng.choice(["bf16", "bf16", "fp32"]))
    if kind == "layer":
        n = (rng.choice([4, 8, 12, 16]), rng.choice([8, 10, 16]), rng.choice([8, 16, 25]))
        m = (rng.choice([4, 8, 10, 16]), rng.choice([8, 12, 16]), rng.choice([8, 10, 16]))
        return _layer("", n, m, rng.randint(4, 24), _log(rng, 32, 8192), rng.choice(["fp32", "bf16"]))
    if kind == "reconstruct":
        edge = _log(rng, 100, 900)
        return _recon("", [max(48, int(edge * rng.uniform(0.75, 1.3))) for _ in range(3)], rng.randint(6, 40))
    edge = _log(rng, 100, 1400)
    return _entries("", [max(48, int(edge * rng.uniform(0.75, 1.3))) for _ in range(3)], rng.randint(6, 40),
                    _log(rng, 1 << 12, 1 << 20))


# ------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _basis(g, n, k):
    return torch.linalg.qr(_randn(g, n, k))[0]


def _weights(k):
    return 1.0 - 0.75 * torch.arange(k, device="cuda", dtype=torch.float32) / k


def _add_noise(x, g):
    rms = x.square().mean().sqrt()
    for part in x:   # slice by slice: a whole tensor of noise would be another copy of x
        part.add_(_randn(g, *part.shape) * (NOISE * rms))
    return x


def _tensor3(dims, rank, seed):
    """Contiguous (n3, n2, n1): the memory of the column-major n1 x n2 x n3 tensor."""
    g = _generator(seed)
    a, b, c = (_basis(g, n, rank) for n in dims)
    left = ((c * _weights(rank))[:, None, :] * b[None, :, :]).reshape(-1, rank)
    return _add_noise((left @ a.T).reshape(dims[2], dims[1], dims[0]), g)


def _inner_basis(g, k, inner):
    """(k, k, inner): orthonormal columns whose energy falls along both leaf indices."""
    w = _weights(k)
    return torch.linalg.qr((_randn(g, k, k, inner) * w[:, None, None] * w[None, :, None]).reshape(k * k, inner))[0] \
        .reshape(k, k, inner)


def _tensor4(dims, rank, inner, seed):
    g = _generator(seed)
    u = [_basis(g, n, rank) for n in dims]
    b12, b34 = _inner_basis(g, rank, inner), _inner_basis(g, rank, inner)
    left = torch.einsum("ia,jb,abk->jik", u[0], u[1], b12).reshape(-1, inner)     # rows j, i
    right = torch.einsum("ia,jb,abk->jik", u[2], u[3], b34).reshape(-1, inner)    # rows n4, n3
    x = ((right * _weights(inner)) @ left.T).reshape(dims[3], dims[2], dims[1], dims[0])
    return _add_noise(x, g)


def _dims(case):
    return tuple(case[k] for k in ("n1", "n2", "n3", "n4") if k in case)


def _tree3(kind, rank):
    return {"reference": ht.reference_tree_3d, "left_first": ht.left_first_tree_3d,
            "middle": ht.middle_tree_3d}[kind]([1, rank, rank, rank, rank])


def _batch_shapes(case):
    r = np.random.default_rng(case["family"])
    shapes = [tuple(int(v) for v in r.integers(case["lo"], case["hi"] + 1, size=3)) for _ in range(case["count"])]
    return shapes, [int(v) for v in r.integers(8, 17, size=case["count"])]


def _factors(dims, rank, seed):
    """Column-major factors of the reference tree, as a decomposition returns them."""
    g = _generator(seed)
    cm = lambda t: t.permute(*reversed(range(t.dim()))).contiguous().permute(*reversed(range(t.dim())))
    U = {t: cm(_basis(g, dims[m], rank)) for t, m in ((2, 2), (3, 0), (4, 1))}
    core = torch.linalg.qr(_randn(g, rank * rank, rank))[0].reshape(rank, rank, rank)
    B = {1: cm(core), 0: cm(torch.diag(_weights(rank)).reshape(rank, rank, 1))}
    return U, B


def _layer_tensors(case, seed):
    g = _generator(seed)
    n = [case[k] for k in ("N0", "N1", "N2")]
    m = [case[k] for k in ("M0", "M1", "M2")]
    r = case["rank"]
    f = [_randn(g, n[j], m[j], r) / r ** 0.5 for j in range(3)]
    f += [_randn(g, r, r, r) / r, _randn(g, r, r) / r ** 0.5]
    nin, nout = n[0] * n[1] * n[2], m[0] * m[1] * m[2]
    x = _randn(g, case["batch"], nin).relu_()   # activations of the layer before
    dy = _randn(g, case["batch"], nout) / case["batch"]
    return x, f, _randn(g, *m) * 0.1, dy


def prepare(case, seed):
    kind = case["kind"]
    if kind == "d3":
        dims = _dims(case)
        return {"kind": "one", "x": _tensor3(dims, case["rank"], seed), "tree": _tree3(case["tree"], case["rank"]),
                "kw": {"precision": case["precision"], "compute_error": case["error"], "leaf_method": case["leaf"]}}
    if kind == "d4":
        r, s = case["rank"], case["inner"]
        return {"kind": "one", "x": _tensor4(_dims(case), r, s, seed),
                "tree": ht.balanced_tree_4d([1, s, s, r, r, r, r]),
                "kw": {"precision": case["precision"], "compute_error": case["error"]}}
    if kind == "batch":
        shapes, ranks = _batch_shapes(case)
        trees = [_tree3("reference", r) for r in ranks]
        bd = ht.BatchDecomposer(trees, shapes, precision=case["precision"], compute_error=True)
        xs = [_tensor3(d, r, seed * 100003 + i) for i, (d, r) in enumerate(zip(shapes, ranks))]
        sizes = [a.numel() for U, B in zip(bd.U, bd.B) for a in list(U.values()) + list(B.values())]
        flat = torch.empty(sum(sizes), device="cuda")
        # the buffer the program keeps the whole batch's factors in
        parts = []
        for v, a in zip(flat.split(sizes), (a for U, B in zip(bd.U, bd.B) for a in list(U.values()) + list(B.values()))):
            parts.append(v.view(*reversed(a.shape)).permute(*reversed(range(a.dim()))))
        return {"kind": "batch", "bd": bd, "xs": xs, "flat": flat, "parts": parts}
    if kind == "layer":
        x, f, bias, dy = _layer_tensors(case, seed)
        layer = htlayer.HTLinear([case["N0"], case["N1"], case["N2"]], [case["M0"], case["M1"], case["M2"]],
                                 case["rank"], precision=case["precision"])
        with torch.no_grad():
            for p, v in zip((layer.u1, layer.u2, layer.u3, layer.b2, layer.b1, layer.bias), f + [bias]):
                p.copy_(v)
        return {"kind": "layer", "layer": layer, "x": x.requires_grad_(True), "dy": dy}
    dims = _dims(case)
    U, B = _factors(dims, case["rank"], seed)
    state = {"kind": kind, "tree": _tree3("reference", case["rank"]), "U": U, "B": B, "dims": dims}
    if kind == "entries":
        state["idx"] = _indices(case, seed)
    return state


def _indices(case, seed):
    g = _generator(seed + 77)
    return torch.stack([torch.randint(0, n, (case["count"],), generator=g, device="cuda") for n in _dims(case)], 1) \
        .contiguous()


# ---------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "one":
        res = ht.decompose(state["x"], state["tree"], **state["kw"])
        out = {"U": {str(t): v for t, v in res.U.items()}, "B": {str(t): v for t, v in res.B.items()}}
        if state["kw"]["compute_error"]:
            out["rel_err"] = res.report["rel_err"]
        return out
    if kind == "batch":
        results, _ = state["bd"](state["xs"])
        torch._foreach_copy_(state["parts"], [a for r in results for a in list(r.U.values()) + list(r.B.values())])
        return {"factors": state["flat"],
                "rel_err": np.array([r.report["rel_err"] for r in results], dtype=np.float32)}
    if kind == "layer":
        layer, x = state["layer"], state["x"]
        y = layer(x)
        par = (layer.u1, layer.u2, layer.u3, layer.b2, layer.b1, layer.bias)
        return [y.detach(), *torch.autograd.grad(y, (x, *par), state["dy"])]
    if kind == "reconstruct":
        return ht.reconstruct(state["tree"], state["U"], state["B"], state["dims"])
    return ht.evaluate(state["tree"], state["U"], state["B"], state["dims"], state["idx"])


# --------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind in ("d3", "d4"):
        dims, r = _dims(case), case["rank"]
        total = float(np.prod([float(d) for d in dims]))
        factors = sum(dims) * r + (r ** 3 + r * r if kind == "d3" else 2 * r * r * case["inner"] + case["inner"] ** 2)
        # each mode Gram (half of a symmetric product) or, with the range finder, two products per leaf block
        leaf = total * sum(dims) if case.get("leaf", "gram") == "gram" else 3 * 8 * total * (r + 16)
        core = 2 * total * (r if kind == "d3" else 4 * (case["inner"] + 16))
        return {"bytes": 4 * (total + factors), "flops": leaf + core}
    if kind == "batch":
        shapes, ranks = _batch_shapes(case)
        b = f = 0.0
        for d, r in zip(shapes, ranks):
            total = float(d[0] * d[1] * d[2])
            b += 4 * (total + sum(d) * r + r ** 3 + r * r)
            f += total * (sum(d) + 2 * r + 2 * r)
        return {"bytes": b, "flops": f}
    if kind == "layer":
        nin, nout = case["N0"] * case["N1"] * case["N2"], case["M0"] * case["M1"] * case["M2"]
        b, r = float(case["batch"]), case["rank"]
        factors = (case["N0"] * case["M0"] + case["N1"] * case["M1"] + case["N2"] * case["M2"]) * r + r ** 3 + r * r
        return {"bytes": 4 * (2 * b * (nin + nout) + 2 * factors), "flops": 6 * b * nin * nout}
    dims, r = _dims(case), case["rank"]
    factors = 4 * (sum(dims) * r + r ** 3 + r * r)
    if kind == "reconstruct":
        total = float(dims[0]) * dims[1] * dims[2]
        return {"bytes": 4 * total + factors, "flops": 2 * total * r}
    n = float(case["count"])
    return {"bytes": 28 * n + factors, "flops": n * (2 * r * r + 2 * r)}


# -------------------------------------------------------------------- exact
def _unfold(x, m):
    """Rows over mode m (0-based) of the column-major tensor held as dims[::-1]."""
    return x.movedim(x.dim() - 1 - m, 0).reshape(x.shape[x.dim() - 1 - m], -1)


def _top(x, m, k):
    a = _unfold(x, m)
    return torch.linalg.eigh(a @ a.T)[1][:, -k:]


def _error3(x, rank):
    """With one rank at every node the HT truncation is the projection of x on its three leaf bases."""
    x = x.double()
    core = x
    for m in range(3):
        u = _top(x, m, rank)
        core = torch.tensordot(core, u, dims=([core.dim() - 1 - m], [0])).movedim(-1, core.dim() - 1 - m)
    return float(torch.sqrt((1 - core.square().sum() / x.square().sum()).clamp_min(0)))


def _error4(x, rank, inner):
    """Leaf projections of the best rank-`inner` approximation of the unfolding {1,2}."""
    x = x.double()
    a = x.reshape(x.shape[0] * x.shape[1], -1)           # rows (n4, n3), columns (n2, n1)
    q = torch.linalg.qr(torch.randn(a.shape[1], min(inner + 16, a.shape[1]), dtype=torch.float64, device="cuda"))[0]
    for _ in range(8):
        q = torch.linalg.qr(a.T @ (a @ q))[0]
    s, v = torch.linalg.eigh((a @ q).T @ (a @ q))
    v = q @ v[:, -inner:]
    best = ((a @ v) @ v.T).reshape(x.shape)
    p = best
    for m in range(4):
        u = _top(x, m, rank)
        p = torch.tensordot(torch.tensordot(p, u, dims=([3 - m], [0])), u, dims=([-1], [1])).movedim(-1, 3 - m)
    return float((x - p).norm() / x.norm())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("d3", "d4"):
        if not case["error"]:
            return None
        dims, r = _dims(case), case["rank"]
        e = _error3(_tensor3(dims, r, seed), r) if kind == "d3" else \
            _error4(_tensor4(dims, r, case["inner"], seed), r, case["inner"])
        return {"U": None, "B": None, "rel_err": e}
    if kind == "batch":
        shapes, ranks = _batch_shapes(case)
        return {"factors": None, "rel_err": np.array([_error3(_tensor3(d, r, seed * 100003 + i), r)
                                                      for i, (d, r) in enumerate(zip(shapes, ranks))])}
    if kind == "layer":
        x, f, bias, dy = _layer_tensors(case, seed)
        x, dy = x.double().requires_grad_(True), dy.double()
        par = [p.double().requires_grad_(True) for p in f + [bias]]
        u1, u2, u3, b2, b1, b = par
        t = torch.einsum("iar,rst->iast", u1, b2)
        t = torch.einsum("iast,jbs->iajbt", t, u2)
        t = torch.einsum("iajbt,tv,kcv->abcijk", t, b1, u3)
        w = t.reshape(t.shape[0] * t.shape[1] * t.shape[2], -1)
        y = x @ w.T + b.reshape(-1)
        return [y.detach(), *torch.autograd.grad(y, (x, *par), dy)]
    U, B = _factors(_dims(case), case["rank"], seed)
    u, b = {t: v.double() for t, v in U.items()}, {t: v.double() for t, v in B.items()}
    core = torch.einsum("abk,kc->abc", b[1], b[0][:, :, 0])
    if kind == "reconstruct":
        t = torch.einsum("ia,abc->ibc", u[3], core)
        t = torch.einsum("jb,ibc->jic", u[4], t).reshape(-1, core.shape[2])
        return (u[2] @ t.T).reshape(u[2].shape[0], u[4].shape[0], u[3].shape[0])
    out = []
    for i in _indices(case, seed).split(1 << 16):
        t = torch.einsum("abc,nc->nab", core, u[2][i[:, 2]])
        out.append(torch.einsum("nab,na,nb->n", t, u[3][i[:, 0]], u[4][i[:, 1]]))
    return torch.cat(out)
