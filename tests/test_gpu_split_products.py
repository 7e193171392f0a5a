"""FP32 products formed from three BF16 planes per operand (csrc/tc3_gemm.cu)
against 64 bits, at the edges of its tiles, K blocks and dispatch rules.

Tolerance of a product: the planes hold every operand bit, the plane products
left out are below 3 * 2^-26 of a term, and a K block's 24 accumulations in the
tensor core truncate by at most 2^-23 of the running sum each, 24 * 2^-23 =
2.9e-6 if every sum had one sign; the blocks' sums are rounded to nearest.
"""
import numpy as np
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht
from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu
TOL = 3e-6


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def layer(n, m, r, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    f = [rn(n[j], m[j], r) / r ** 0.5 for j in range(3)] + [rn(r, r, r) / r, rn(r, r) / r ** 0.5]
    return f, rn


# nin, nout: multiples of 8 (planes) and not (CUDA cores); batches around the
# tile's 64, 128 and 256 columns; K blocks of 64 with remainders
@pytest.mark.parametrize("n,m", [((2, 4, 8), (4, 4, 8)), ((3, 5, 8), (2, 7, 12)), ((8, 8, 16), (8, 8, 16)),
                                 ((3, 5, 7), (4, 3, 5))])
@pytest.mark.parametrize("batch", [1, 8, 63, 64, 65, 129, 257, 700])
def test_layer_products(n, m, batch):
    f, rn = layer(n, m, 6)
    nin, nout = int(np.prod(n)), int(np.prod(m))
    x, dy, b = rn(batch, nin), rn(batch, nout), rn(nout)
    w = htlayer.layer_weight(*f).double()
    for relu in (False, True):
        y = htlayer.layer_forward(x, *f, bias=b, relu=relu)
        want = x.double() @ w.T + b.double()
        assert rel(y, want.clamp_min(0) if relu else want) < TOL
    dx, du1 = htlayer.layer_backward(x, dy, *f)[:2]
    assert rel(dx, dy.double() @ w) < TOL
    p = [t.double().requires_grad_(True) for t in f]
    t = torch.einsum("iar,rst,jbs->iajbt", p[0], p[3], p[1])
    wd = torch.einsum("iajbt,tv,kcv->abcijk", t, p[4], p[2]).reshape(nout, nin)
    want = torch.autograd.grad((x.double() @ wd.T * dy.double()).sum(), p[0])[0]
    assert rel(du1, want) < 2e-5   # dW through FP32 sums over every mode


def test_layer_long_batch_splits_k():
    f, rn = layer((4, 4, 8), (4, 4, 8), 5)
    x, dy = rn(9000, 128), rn(9000, 128)
    w = htlayer.layer_weight(*f).double()
    assert rel(htlayer.layer_forward(x, *f), x.double() @ w.T) < TOL
    assert rel(htlayer.layer_backward(x, dy, *f)[0], dy.double() @ w) < TOL


def test_unaligned_rows_of_a_batch():
    """x and dy that start 4 bytes off a 16-byte boundary."""
    f, rn = layer((2, 4, 8), (4, 4, 8), 4)
    x, dy = rn(33 * 64 + 1)[1:].view(33, 64), rn(33 * 128 + 1)[1:].view(33, 128)
    w = htlayer.layer_weight(*f).double()
    assert rel(htlayer.layer_forward(x, *f), x.double() @ w.T) < TOL
    assert rel(htlayer.layer_backward(x, dy, *f)[0], dy.double() @ w) < TOL


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38, 1e-40])
def test_entries_without_planes(value):
    """Infinities, NaN and the largest magnitudes give what FP32 arithmetic gives."""
    f, rn = layer((2, 4, 8), (4, 4, 8), 4)
    x = rn(70, 64)
    x[17, 5] = value
    w = htlayer.layer_weight(*f)
    w[:, 5] = 0
    y = htlayer.layer_forward(x, *f).double()
    want = x.double() @ htlayer.layer_weight(*f).double().T
    over = want.abs() > 3.4028235e38
    want[over] = want[over].sign() * float("inf")
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    assert torch.equal(torch.isinf(y), torch.isinf(want))
    fin = torch.isfinite(want)
    assert torch.equal(y[~fin & ~torch.isnan(want)].sign(), want[~fin & ~torch.isnan(want)].sign())
    rows = torch.ones(70, dtype=torch.bool, device="cuda")
    rows[17] = False
    assert rel(y[rows], want[rows]) < TOL
    # and the next call, on finite data, is unaffected
    x[17, 5] = 1.0
    assert rel(htlayer.layer_forward(x, *f), x.double() @ htlayer.layer_weight(*f).double().T) < TOL


def cm(t):
    rev = list(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


# sizes on both sides of the rule that takes the planes (2e8 multiply-adds),
# ragged rows, K of 1, 16, 17 and 64, every place of the complementary mode
@pytest.mark.parametrize("dims,r", [((301, 260, 397), 17), ((515, 129, 1027), 5), ((96, 2050, 120), 16),
                                    ((200, 150, 257), 64), ((640, 640, 640), 1), ((40, 33, 65), 9)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
def test_reconstruct(dims, r, make):
    g = torch.Generator(device="cuda").manual_seed(3)
    tr = make([1, r, r, r, r])
    U = {t: cm(torch.randn(dims[tr.modes[t][0]], r, generator=g, device="cuda")) for t in tr.leaves()}
    B = {t: cm(torch.randn(r, r, 1 if t == 0 else r, generator=g, device="cuda")) for t in [0] + tr.interior()}
    X = ht.reconstruct(tr, U, B, dims).permute(2, 1, 0)
    i = tr.interior()[0]
    p, q = tr.left[i], tr.right[i]
    c = [t for t in tr.leaves() if t not in (p, q)][0]
    root = B[0][:, :, 0].double()
    W = torch.einsum("ia,jb,abk,kc->ijc", U[p].double(), U[q].double(), B[i].double(),
                     root if tr.left[0] == i else root.T)
    want = torch.einsum("ijc,lc->ijl", W, U[c].double())
    order = [tr.modes[t][0] for t in (p, q, c)]
    want = want.permute(*[order.index(m) for m in range(3)])
    assert rel(X, want) < 3 * TOL   # core, both expansion steps, the product


@pytest.mark.parametrize("dims", [(256, 200, 96), (181, 150, 203), (300, 40, 500)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_error_pass_of_a_decomposition(dims, make, precision):
    """The error a decomposition reports (planes at these sizes) against the
    CUDA-core error pass over its factors."""
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(*reversed(dims), generator=g, device="cuda")
    tr = make([1, 12, 12, 12, 12])
    res = ht.decompose(x, tr, precision=precision, compute_error=True)
    want = ht.reconstruct_error(x, tr, res.U, res.B)
    assert abs(res.report["rel_err"] - want) < 1e-6


def test_error_pass_4th_order():
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn(41, 60, 52, 44, generator=g, device="cuda")
    tr = ht.balanced_tree_4d([1, 16, 16, 8, 8, 8, 8])
    res = ht.decompose(x, tr, precision="fp32", compute_error=True)
    assert abs(res.report["rel_err"] - ht.reconstruct_error(x, tr, res.U, res.B)) < 1e-6
