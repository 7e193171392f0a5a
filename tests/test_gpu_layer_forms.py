"""Layer shapes on both sides of the rules that choose the weight's and the factor
gradients' kernels (csrc/layer.cu): padded rows that fit shared memory or do not,
few and many pairs, ranks that are and are not multiples of four.

Tolerance: FP32 chains over at most N0 N1 N2 or M0 M1 M2 batch terms with random
signs; 2e-5 as for the layer's other gradients.
"""
import numpy as np
import pytest
import torch

from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu

SHAPES = [
    ((4, 4, 128), (8, 8, 64), 5),     # dP/dQ: only the packed form fits
    ((4, 4, 128), (8, 8, 64), 6),     # neither
    ((4, 4, 128), (8, 8, 32), 9),     # both, few pairs
    ((8, 16, 64), (8, 8, 64), 9),     # only packed, 128 pairs
    ((2, 3, 8), (4, 4, 32), 7),       # both, six pairs
    ((6, 8, 16), (4, 4, 8), 10),      # 48 pairs
    ((7, 7, 16), (4, 4, 24), 10),     # 49 pairs
    ((8, 12, 8), (4, 4, 8), 33),      # 96 pairs, blocks of one row
    ((16, 16, 25), (4, 4, 16), 16),   # 256 pairs
    ((3, 5, 7), (2, 3, 5), 3),        # nothing a multiple of anything
    ((12, 64, 32), (2, 4, 32), 33),   # weight: only the packed form fits
    ((12, 64, 32), (1, 2, 19), 48),   # and a remainder of its groups of m2
    ((30, 30, 8), (4, 4, 8), 40),     # an entry a thread
    ((40, 40, 4), (8, 8, 8), 18),     # packed, blocks enough for planes
    ((16, 16, 16), (4, 4, 16), 12),   # tiled
]


@pytest.mark.parametrize("n,m,r", SHAPES)
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_forms(n, m, r, precision):
    nin, nout = int(np.prod(n)), int(np.prod(m))
    if precision == "bf16" and (nin % 8 or nout % 8):
        pytest.skip("BF16 layers take multiples of 8")
    g = torch.Generator(device="cuda").manual_seed(r)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    f = [rn(n[j], m[j], r) / r ** 0.5 for j in range(3)] + [rn(r, r, r) / r, rn(r, r) / r ** 0.5]
    x, dy = rn(24, nin), rn(24, nout)
    p = [t.double().requires_grad_(True) for t in f]
    t = torch.einsum("iar,rst,jbs->iajbt", p[0], p[3], p[1])
    w = torch.einsum("iajbt,tv,kcv->abcijk", t, p[4], p[2]).reshape(nout, nin)
    xd, dyd = x.double(), dy.double()
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    if precision == "fp32":
        assert rel(htlayer.layer_weight(*f), w.detach()) < 2e-6
        assert rel(htlayer.layer_forward(x, *f), xd @ w.detach().T) < 3e-6
    tol = 2e-5 if precision == "fp32" else 8e-3   # BF16 operands: 2^-8 each, random signs
    got = htlayer.layer_backward(x, dy, *f, precision=precision)
    want = torch.autograd.grad((xd @ w.T * dyd).sum(), p)
    assert rel(got[0], dyd @ w.detach()) < tol
    for a, b in zip(got[1:6], want):
        assert rel(a, b) < tol
    # the sums have a fixed order
    for a, b in zip(got, htlayer.layer_backward(x, dy, *f, precision=precision)):
        assert torch.equal(a, b)
