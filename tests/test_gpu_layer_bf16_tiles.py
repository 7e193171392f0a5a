"""BF16 layers whose products have fewer 128-row tiles than SMs (K in one piece or
split), as many, and more, and ranks on both sides of 16 and 32 in the factor
gradients.

Tolerance: operands rounded to BF16, 2^-8 each with random signs: 8e-3.
"""
import numpy as np
import pytest
import torch

from ht_tensor_learning_using_gpu_tensor_cores_gb300 import htlayer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,r,batch", [((16, 16, 16), (8, 8, 16), 16, 256), ((16, 16, 16), (8, 8, 16), 17, 1024),
                                         ((16, 16, 16), (8, 16, 16), 3, 4096), ((16, 16, 16), (16, 16, 16), 2, 1024),
                                         ((8, 8, 8), (8, 8, 8), 32, 8200), ((8, 10, 8), (10, 8, 12), 33, 777),
                                         ((4, 8, 8), (4, 8, 8), 24, 300)])
def test_layer(n, m, r, batch):
    nin, nout = int(np.prod(n)), int(np.prod(m))
    g = torch.Generator(device="cuda").manual_seed(r)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    f = [rn(n[j], m[j], r) / r ** 0.5 for j in range(3)] + [rn(r, r, r) / r, rn(r, r) / r ** 0.5]
    x, dy, b = rn(batch, nin), rn(batch, nout), rn(nout)
    rel = lambda p, q: float((p.double() - q).norm() / q.norm())
    w = htlayer.layer_weight(*f).double()
    want = x.double() @ w.T + b.double()
    assert rel(htlayer.layer_forward(x, *f, bias=b, precision="bf16"), want) < 8e-3
    assert rel(htlayer.layer_forward(x, *f, bias=b, relu=True, precision="bf16"), want.clamp_min(0)) < 8e-3
    got = htlayer.layer_backward(x, dy, *f, precision="bf16")
    assert rel(got[0], dy.double() @ w) < 8e-3
    p = [t.double().requires_grad_(True) for t in f]
    t = torch.einsum("iar,rst,jbs->iajbt", p[0], p[3], p[1])
    wd = torch.einsum("iajbt,tv,kcv->abcijk", t, p[4], p[2]).reshape(nout, nin)
    dw = dy.double().T @ x.double()
    for a, q in zip(got[1:6], torch.autograd.grad((wd * dw).sum(), p)):
        assert rel(a, q) < 8e-3
    assert rel(got[6], dy.double().sum(0)) < 1e-5
