"""FP32 products from three BF16 planes per operand (csrc/tc3_gemm.cu): every
plane by itself, FP32's whole range of magnitudes, and errors against 64 bits
tight enough that no plane product can be missing.

A layer of ranks 1 with n = (1, 1, N), m = (1, 1, M) has any N x M matrix as its
weight, so a forward or backward call is a dense product.

Tolerance of a product, relative to its norm: the four h h' steps of a K block
truncate by at most 2^-23 of the running sum each, 4 * 2^-23 = 4.8e-7; the steps
before them run on sums 2^-7 as large, and what is left out is below 2^-24 of a
term with random signs (6e-9 of a sum).  Without one of the six products the
error is 2.4e-6 or more.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu
TOL = 5e-7


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def dense(w):
    """Factors of the layer whose weight is w (M x N)."""
    one = torch.ones(1, 1, 1, device="cuda")
    return one, one, w.t().contiguous().unsqueeze(2), one, one[0]


def mantissas(g, n):
    """FP32 numbers in [1, 2) with all 24 bits in use."""
    return (torch.randint(1 << 22, 1 << 23, (n,), generator=g, device="cuda") * 2 + 1).float() * 2.0 ** -23


# exponents of x: where planes are normal numbers, where the lower ones would be
# subnormal in FP32's own scale (-110), the last exact one (-124), FP32's smallest
# normal and subnormal numbers
@pytest.mark.parametrize("e", [100, 0, -60, -109, -110, -112, -117, -122, -124, -126, -130, -140])
@pytest.mark.parametrize("batch", [70, 128])
def test_one_term_per_sum(e, batch):
    """x has one entry a row and w powers of two: the product is exact, plane by plane."""
    g = gen(batch - e)
    N, M = 96, 128
    up = 2.0 ** (60 if e < -60 else 0)
    i = torch.randint(0, N, (batch,), generator=g, device="cuda")
    v = (mantissas(g, batch).double() * 2.0 ** e).float()   # (rounded where FP32 holds fewer bits)
    x = torch.zeros(batch, N, device="cuda")
    x[torch.arange(batch, device="cuda"), i] = v
    w = torch.randint(0, 4, (M, N), generator=g, device="cuda").float().exp2() * up
    want = v.double()[:, None] * w.double()[:, i].t()
    slack = 0.0 if e >= -124 else 2.0 ** -148
    y = htlayer.layer_forward(x, *dense(w)).double()
    assert ((y - want).abs() <= slack * w.double()[:, i].t()).all()
    # the same numbers as the weight: its planes are formed by the weight's own kernel
    y = htlayer.layer_forward(w, *dense(x)).double()
    assert ((y.t() - want).abs() <= slack * w.double()[:, i].t()).all()
    # and as dy
    dx = htlayer.layer_backward(x.new_zeros(batch, M), x, *dense(w.t().contiguous()), need_dbias=False)[0].double()
    assert ((dx - want).abs() <= slack * w.double()[:, i].t()).all()


@pytest.mark.parametrize("batch", [33, 300])
def test_product_of_full_mantissas(batch):
    """One term a sum again, both factors with 24 bits: 5 truncating sums and what is left out."""
    g = gen(batch)
    N, M = 64, 128
    i = torch.randint(0, N, (batch,), generator=g, device="cuda")
    x = torch.zeros(batch, N, device="cuda")
    x[torch.arange(batch, device="cuda"), i] = mantissas(g, batch)
    w = mantissas(g, M * N).view(M, N)
    want = x.double() @ w.double().t()
    y = htlayer.layer_forward(x, *dense(w)).double()
    assert ((y - want).abs() / want).max() < 5 * 2.0 ** -23 + 2.0 ** -24


@pytest.mark.parametrize("N,M,batch", [(64, 64, 64), (64, 192, 300), (8, 1024, 257), (1024, 8, 130), (640, 16, 1000),
                                       (104, 112, 2000)])
@pytest.mark.parametrize("ex,ew", [(0, 0), (-110, 60), (-118, 100), (60, -110), (-50, -40), (-62, -50), (62, 56)])
def test_gaussian_products(N, M, batch, ex, ew):
    g = gen(N + batch)
    x, w, dy = randn(g, batch, N) * 2.0 ** ex, randn(g, M, N) * 2.0 ** ew, randn(g, batch, M) * 2.0 ** ex
    f = dense(w)
    assert rel(htlayer.layer_forward(x, *f), x.double() @ w.double().t()) < TOL
    assert rel(htlayer.layer_backward(x, dy, *f)[0], dy.double() @ w.double()) < TOL


@pytest.mark.parametrize("value", [1e-40, 3e-36, 1e-33, 3.4e38, 1e30])
def test_row_with_one_extreme_entry(value):
    """The row that holds it, against 64 bits, relative to the sum of the terms' magnitudes."""
    g = gen(4)
    x, w = randn(g, 70, 64), randn(g, 96, 64)
    x[17, 5] = value
    y = htlayer.layer_forward(x, *dense(w)).double()
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    over = want.abs() > 3.4028235e38
    assert torch.isinf(y[over]).all()
    # FP32 chains of 64 terms where the call goes to the CUDA cores (3.4e38 has no planes)
    assert ((y - want).abs()[~over] / size[~over]).max() < 64 * 2.0 ** -24


def cm(t):
    rev = list(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


def expansion(tr, U, B):
    i = tr.interior()[0]
    p, q = tr.left[i], tr.right[i]
    c = [t for t in tr.leaves() if t not in (p, q)][0]
    root = B[0][:, :, 0].double()
    W = torch.einsum("ia,jb,abk,kc->ijc", U[p].double(), U[q].double(), B[i].double(),
                     root if tr.left[0] == i else root.T)
    want = torch.einsum("ijc,lc->ijl", W, U[c].double())
    order = [tr.modes[t][0] for t in (p, q, c)]
    return want.permute(*[order.index(m) for m in range(3)])


# 1.4e9 multiply-adds take planes: two tensors above, one below
@pytest.mark.parametrize("dims,r", [((301, 260, 397), 64), ((640, 321, 420), 17), ((40, 33, 65), 9)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
@pytest.mark.parametrize("e", [0, -116])
def test_reconstruct(dims, r, make, e):
    g = gen(3)
    tr = make([1, r, r, r, r])
    U = {t: cm(randn(g, dims[tr.modes[t][0]], r)) for t in tr.leaves()}
    B = {t: cm(randn(g, r, r, 1 if t == 0 else r)) for t in [0] + tr.interior()}
    i = tr.interior()[0]
    c = [t for t in tr.leaves() if t not in (tr.left[i], tr.right[i])][0]
    U[c] *= 2.0 ** e        # the last product's planes
    U[tr.left[i]] *= 2.0 ** (-e // 2)
    X = ht.reconstruct(tr, U, B, dims).permute(2, 1, 0)
    assert rel(X, expansion(tr, U, B)) < 3 * TOL   # core, both expansion steps, the product


# (1.5e8 multiply-adds take planes)
@pytest.mark.parametrize("dims", [(256, 200, 300), (301, 263, 203)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
def test_small_error_of_a_decomposition(dims, make):
    """An error of 1e-5, which an error delta of the expansion moves by delta^2 / 2e-5:
    5e-8 at delta = 1e-6 (two products), 3e-7 and more without a plane."""
    g = gen(5)
    r = 12
    tr = make([1, r, r, r, r])
    U = {t: cm(torch.linalg.qr(randn(g, dims[tr.modes[t][0]], r))[0]) for t in tr.leaves()}
    B = {t: cm(randn(g, r, r, 1 if t == 0 else r)) for t in [0] + tr.interior()}
    x = expansion(tr, U, B)
    x = x + 1e-5 * x.square().mean().sqrt() * randn(g, *x.shape).double()
    x = x.float().permute(2, 1, 0).contiguous()
    res = ht.decompose(x, tr, precision="fp32", compute_error=True)
    d = x.double().permute(2, 1, 0) - expansion(tr, res.U, res.B)
    want = float(d.norm() / x.double().norm())
    assert abs(res.report["rel_err"] - want) < 1e-7
