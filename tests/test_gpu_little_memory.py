"""Calls that find no room for the operands' planes or the sort's records: the same
results from the smaller plan, call after call, and the larger plan again when
there is room.  A layer call recorded in a graph takes what the workspace holds.

(All but a little device memory is held by a tensor meanwhile; nothing touches it.)
"""
import contextlib

import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu
MB = 1 << 20


def rel(a, b):
    """In pieces: there is no room for copies in 64 bits."""
    n = d = 0.0
    for p, q in zip(a.reshape(-1).split(1 << 20), b.reshape(-1).split(1 << 20)):
        q = q.double()
        n += float((p.double() - q).square().sum())
        d += float(q.square().sum())
    return (n / d) ** 0.5


def randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def cm(t):
    rev = list(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


@contextlib.contextmanager
def room(nbytes):
    """About nbytes of device memory left, the workspaces given back first."""
    ht.release_workspace()
    htlayer.release()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = []
    while free - nbytes > 8 * MB:   # in pieces: one block of everything need not exist
        hold.append(torch.empty(min(free - nbytes, 32 << 30), dtype=torch.uint8, device="cuda"))
        free = torch.cuda.mem_get_info()[0]
    try:
        yield
    finally:
        hold.clear()
        torch.cuda.empty_cache()


def calls(run, nbytes, same, *, plan_bytes):
    want = run()     # (also leaves the outputs' memory in the allocator's cache)
    torch.cuda.synchronize()
    first = run()
    assert same(first, want)
    del first
    with room(nbytes):
        left = []
        for _ in range(3):
            assert same(run(), want)
            torch.cuda.synchronize()
            left.append(torch.cuda.mem_get_info()[0])
        assert left[0] == left[1] == left[2]
    free = torch.cuda.mem_get_info()[0]
    assert same(run(), want)   # with room again: the larger plan
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] > plan_bytes


def test_decompose():
    g = torch.Generator(device="cuda").manual_seed(1)
    dims, r = (512, 512, 256), 16
    U = [torch.linalg.qr(randn(g, n, r))[0] for n in dims]
    w = torch.linspace(1, 0.3, r, device="cuda")
    x = torch.einsum("ia,ja,ka,a->kji", U[0], U[1], U[2], w).contiguous()
    x += 1e-2 * x.square().mean().sqrt() * randn(g, *x.shape)
    tr = ht.reference_tree_3d([1, r, r, r, r])
    run = lambda: ht.decompose(x, tr, precision="fp32", compute_error=True).report["rel_err"]
    calls(run, 240 * MB, lambda a, b: abs(a - b) < 1e-6, plan_bytes=100 * MB)


def test_reconstruct():
    g = torch.Generator(device="cuda").manual_seed(2)
    dims, r = (1024, 1024, 64), 32
    tr = ht.reference_tree_3d([1, r, r, r, r])
    U = {t: cm(randn(g, dims[tr.modes[t][0]], r)) for t in tr.leaves()}
    B = {t: cm(randn(g, r, r, 1 if t == 0 else r)) for t in [0] + tr.interior()}
    calls(lambda: ht.reconstruct(tr, U, B, dims), 240 * MB, lambda a, b: rel(a, b) < 2e-6, plan_bytes=100 * MB)


def test_evaluate():
    g = torch.Generator(device="cuda").manual_seed(3)
    dims, r = (300, 300, 300), 16
    tr = ht.reference_tree_3d([1, r, r, r, r])
    U = {t: cm(randn(g, dims[tr.modes[t][0]], r)) for t in tr.leaves()}
    B = {t: cm(randn(g, r, r, 1 if t == 0 else r)) for t in [0] + tr.interior()}
    idx = torch.randint(0, 300, (1 << 22, 3), generator=g, device="cuda")
    calls(lambda: ht.evaluate(tr, U, B, dims, idx), 40 * MB, lambda a, b: rel(a, b) < 2e-6, plan_bytes=30 * MB)


def test_layer():
    g = torch.Generator(device="cuda").manual_seed(4)
    n, m, r = (8, 8, 16), (8, 8, 16), 16
    f = [randn(g, n[j], m[j], r) / 4 for j in range(3)] + [randn(g, r, r, r) / r, randn(g, r, r) / 4]
    x = randn(g, 40000, 1024)
    calls(lambda: htlayer.layer_forward(x, *f), 100 * MB, lambda a, b: rel(a, b) < 2e-6, plan_bytes=100 * MB)


def test_capture_with_a_workspace_too_small_for_the_planes():
    """A BF16 call made the workspace; the FP32 one being recorded fits it without planes."""
    g = torch.Generator(device="cuda").manual_seed(5)
    n, m, r = (8, 8, 16), (8, 8, 16), 16
    f = [randn(g, n[j], m[j], r) / 4 for j in range(3)] + [randn(g, r, r, r) / r, randn(g, r, r) / 4]
    x = randn(g, 8192, 1024)
    want = htlayer.layer_forward(x, *f)
    htlayer.release()
    htlayer.layer_forward(x, *f, precision="bf16")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = htlayer.layer_forward(x, *f)
    graph.replay()
    torch.cuda.synchronize()
    assert rel(out, want) < 2e-6
    htlayer.release()
