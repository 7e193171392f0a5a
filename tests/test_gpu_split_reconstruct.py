"""Reconstructions and error passes on both sides of the sizes from which their
products run from planes: 1.4e9 multiply-adds (2.5e9 below 12 terms), 6e8 for an
expansion step, 1.5e8 for the error pass; ragged rows, every place of the
complementary mode, sums of 12 to 64 terms.

Tolerance: a product's 5e-7 (four truncating steps of 2^-23), three in a row.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht

pytestmark = pytest.mark.gpu
TOL = 5e-7


def rel(a, b):
    n = d = 0.0
    for p, q in zip(a.reshape(-1).split(1 << 24), b.reshape(-1).split(1 << 24)):
        n += float((p.double() - q).square().sum())
        d += float(q.square().sum())
    return (n / d) ** 0.5


def cm(t):
    rev = list(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


def factors(tr, dims, r, g):
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    U = {t: cm(rn(dims[tr.modes[t][0]], r)) for t in tr.leaves()}
    return U, {t: cm(rn(r, r, 1 if t == 0 else r)) for t in [0] + tr.interior()}


def expansion(tr, U, B):
    i = tr.interior()[0]
    p, q = tr.left[i], tr.right[i]
    c = [t for t in tr.leaves() if t not in (p, q)][0]
    root = B[0][:, :, 0].double()
    core = torch.einsum("abk,kc->abc", B[i].double(), root if tr.left[0] == i else root.T)
    W = torch.einsum("ia,abc->ibc", U[p].double(), core)
    W = torch.einsum("jb,ibc->ijc", U[q].double(), W)
    want = torch.einsum("ijc,lc->ijl", W, U[c].double())
    order = [tr.modes[t][0] for t in (p, q, c)]
    return want.permute(*[order.index(m) for m in range(3)])


@pytest.mark.parametrize("dims,r", [((700, 601, 301), 12), ((515, 129, 1300), 17), ((301, 260, 397), 64),
                                    ((96, 2050, 220), 33), ((350, 350, 350), 32), ((700, 601, 301), 11),
                                    ((780, 690, 700), 7)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
def test_third_order(dims, r, make):
    g = torch.Generator(device="cuda").manual_seed(r)
    tr = make([1, r, r, r, r])
    U, B = factors(tr, dims, r, g)
    X = ht.reconstruct(tr, U, B, dims).permute(2, 1, 0)
    assert rel(X, expansion(tr, U, B)) < 3 * TOL


def test_fourth_order():
    dims, r, s = (120, 95, 101, 77), 16, 24
    g = torch.Generator(device="cuda").manual_seed(4)
    tr = ht.balanced_tree_4d([1, s, s, r, r, r, r])
    rn = lambda *q: torch.randn(*q, generator=g, device="cuda")
    U = {t: cm(rn(dims[tr.modes[t][0]], r)) for t in tr.leaves()}
    B = {t: cm(rn(s, s, 1) if t == 0 else rn(r, r, s)) for t in [0] + tr.interior()}
    X = ht.reconstruct(tr, U, B, dims).permute(3, 2, 1, 0)
    half = lambda t: torch.einsum("ia,jb,abk->ijk", U[tr.left[t]].double(), U[tr.right[t]].double(), B[t].double())
    a, b = half(tr.left[0]), half(tr.right[0])
    want = torch.einsum("ijk,kl,mnl->ijmn", a, B[0][:, :, 0].double(), b)
    modes = [tr.modes[t][0] for t in (tr.left[tr.left[0]], tr.right[tr.left[0]], tr.left[tr.right[0]], tr.right[tr.right[0]])]
    assert rel(X, want.permute(*[modes.index(m) for m in range(4)])) < 4 * TOL


@pytest.mark.parametrize("dims,r", [((230, 231, 233), 12), ((229, 230, 232), 12), ((100, 2001, 60), 13), ((2001, 100, 60), 13)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
def test_error_pass(dims, r, make):
    """A relative error of 1e-3 against 64 bits over the decomposition's own factors."""
    g = torch.Generator(device="cuda").manual_seed(6)
    tr = make([1, r, r, r, r])
    U, B = factors(tr, dims, r, g)
    x = expansion(tr, U, B)
    x = (x + 1e-3 * x.square().mean().sqrt() * torch.randn(*x.shape, generator=g, device="cuda").double()).float()
    x = x.permute(2, 1, 0).contiguous()
    res = ht.decompose(x, tr, precision="fp32", compute_error=True)
    d = x.double().permute(2, 1, 0) - expansion(tr, res.U, res.B)
    want = float(d.norm() / x.double().norm())
    assert abs(res.report["rel_err"] - want) < 2e-8 + 1e-6 * want   # an error of 1e-6 of X across 1e-3: 5e-10
