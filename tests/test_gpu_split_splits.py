"""Products from planes on both sides of the rule that splits K among the SMs (16 K
blocks to a split, four where the SMs would stay idle) and of the one that leaves
tiny forward products to the CUDA cores.

A layer of ranks 1 with n = (1, 1, N), m = (1, 1, M) has any N x M matrix as its
weight.  Tolerance: 4 * 2^-23 of a K block's truncating sums, rounded sums over
blocks and splits on top: 6e-7.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu
TOL = 6e-7


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


# K of 1, 4, 5, 8, 9, 16, 17 and 65 blocks; tiny: N <= 64, or N <= 128 and batch <= 64
@pytest.mark.parametrize("N,M", [(64, 64), (256, 48), (264, 40), (512, 24), (520, 16), (1024, 8), (1032, 8), (4104, 2)])
@pytest.mark.parametrize("batch", [1, 64, 65, 200])
def test_forward_and_gradient(N, M, batch):
    g = torch.Generator(device="cuda").manual_seed(N + batch)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, w, dy, b = rn(batch, N), rn(M, N), rn(batch, M), rn(M)
    one = torch.ones(1, 1, 1, device="cuda")
    f = (one, one, w.t().contiguous().unsqueeze(2), one, one[0])
    want = x.double() @ w.double().t() + b.double()
    assert rel(htlayer.layer_forward(x, *f, bias=b), want) < TOL
    assert rel(htlayer.layer_forward(x, *f, bias=b, relu=True), want.clamp_min(0)) < TOL
    got = htlayer.layer_backward(x, dy, *f)
    assert rel(got[0], dy.double() @ w.double()) < TOL
    assert rel(got[3][:, :, 0], x.double().t() @ dy.double()) < TOL


# Grams of one to a few tiles and 1 to 150 K blocks
@pytest.mark.parametrize("dims", [(8, 8, 8), (20, 20, 20), (24, 25, 24), (33, 31, 40), (64, 64, 64), (8, 300, 8), (130, 70, 9)])
def test_decomposition_error(dims):
    g = torch.Generator(device="cuda").manual_seed(9)
    r = 3
    U = [torch.linalg.qr(torch.randn(n, r, generator=g, device="cuda"))[0].double() for n in dims]
    w = torch.tensor([1.0, 0.7, 0.5], device="cuda").double()
    x = torch.einsum("ia,ja,ka,a->kji", U[0], U[1], U[2], w)
    x = (x + 1e-3 * x.square().mean().sqrt() * torch.randn(*x.shape, generator=g, device="cuda").double()).float()
    res = ht.decompose(x.contiguous(), ht.reference_tree_3d([1, r, r, r, r]), precision="fp32", compute_error=True)
    core = xd = x.double()
    for m in range(3):
        a = xd.movedim(2 - m, 0).reshape(dims[m], -1)
        u = torch.linalg.eigh(a @ a.T)[1][:, -r:]
        core = torch.tensordot(core, u, dims=([2 - m], [0])).movedim(-1, 2 - m)
    want = float(torch.sqrt(1 - core.square().sum() / xd.square().sum()))
    assert abs(res.report["rel_err"] - want) < 1e-6 + 1e-3 * want   # the bases' own error is of second order
