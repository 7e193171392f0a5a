"""Reconstruction on both sides of the rule that gives the second step of an HT
expansion to a thread per output (sums of at most 10 terms, at most 1.5e6
multiply-adds), for every tree and a 4th-order tensor.

Tolerance: four FP32 chains of at most 11 terms with random signs, 11 2^-24 each.
"""
import pytest
import torch

import ht_tensor_learning_using_gpu_tensor_cores_gb300 as ht

pytestmark = pytest.mark.gpu


def cm(t):
    rev = list(reversed(range(t.dim())))
    return t.permute(*rev).contiguous().permute(*rev)


def factors(tr, dims, ranks, g):
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    U = {t: cm(rn(dims[tr.modes[t][0]], ranks[t])) for t in tr.leaves()}
    B = {t: cm(rn(ranks[tr.left[t]], ranks[tr.right[t]], ranks[t])) for t in [0] + tr.interior()}
    return U, B


def full(tr, U, B, t):
    """Node t's basis in 64 bits, modes in the tree's order, rank last."""
    if t in U:
        return U[t].double()
    a, b = full(tr, U, B, tr.left[t]), full(tr, U, B, tr.right[t])
    return torch.tensordot(torch.tensordot(a, B[t].double(), dims=([-1], [0])).movedim(-2, -1), b.movedim(-1, 0),
                           dims=([-1], [0])).movedim(a.dim() - 1, -1)


@pytest.mark.parametrize("dims,r", [((5, 3, 4), 1), ((80, 81, 82), 8), ((136, 137, 33), 8), ((137, 138, 33), 8),
                                    ((122, 123, 20), 10), ((122, 123, 20), 11), ((3000, 7, 9), 6)])
@pytest.mark.parametrize("make", [ht.reference_tree_3d, ht.left_first_tree_3d, ht.middle_tree_3d])
def test_third_order(dims, r, make):
    r = min(r, min(dims))
    tr = make([1, r, r, r, r])
    U, B = factors(tr, dims, [1, r, r, r, r], torch.Generator(device="cuda").manual_seed(r))
    X = ht.reconstruct(tr, U, B, dims).permute(2, 1, 0).double()
    want = full(tr, U, B, 0)[..., 0]
    leaf_order = []
    walk = lambda t: leaf_order.append(tr.modes[t][0]) if t in U else (walk(tr.left[t]), walk(tr.right[t]))
    walk(0)
    want = want.permute(*[leaf_order.index(m) for m in range(3)])
    assert float((X - want).norm() / want.norm()) < 4 * 11 * 2.0 ** -24


def test_fourth_order():
    dims, r, s = (48, 20, 31, 17), 10, 12
    tr = ht.balanced_tree_4d([1, s, s, r, r, r, r])
    U, B = factors(tr, dims, [1, s, s, r, r, r, r], torch.Generator(device="cuda").manual_seed(1))
    X = ht.reconstruct(tr, U, B, dims).permute(3, 2, 1, 0).double()
    want = full(tr, U, B, 0)[..., 0]
    leaf_order = []
    walk = lambda t: leaf_order.append(tr.modes[t][0]) if t in U else (walk(tr.left[t]), walk(tr.right[t]))
    walk(0)
    want = want.permute(*[leaf_order.index(m) for m in range(4)])
    assert float((X - want).norm() / want.norm()) < 4 * 12 * 2.0 ** -24
