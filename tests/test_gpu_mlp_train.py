"""The training launches (csrc/mlp_train.cu)
against the layer-by-layer entry points (poyd_gemm_bf16 and its companions)
at the edges of the 32-row chain blocks, the 16-row chunks of a gradient
split and the 8 ranks that share a gradient.

Tolerances: two fp32 sums of at most 256 products in different orders differ
by far less than a bf16 ulp, so a hidden activation may round to the
neighbouring bf16 value and no further; such a step is 2^-8 of one of a row's
256 terms and rare (a fraction of about 2^-24 * 256 / 2^-8 = 2^-8 at most), so
predictions agree to 2^-8 * 2^-4 = 2^-12 of their norm, and gradients, sums
over rows of products of two such values, to 2^-10."""
import ctypes as C

import numpy as np
import pytest
import torch

from poyd_gb300 import mlp, native

pytestmark = pytest.mark.gpu
DIMS = mlp.DIMS


def rel(a, b):
    a, b = a.double(), b.double()
    n = b.norm().item()
    return (a - b).norm().item() / n if n else a.norm().item()


def layers(net, X16, target):
    """forward + backward through the layer-by-layer entry points."""
    L, p = net.L, lambda t: None if t is None else C.c_void_p(t.data_ptr())
    st, B, dev = C.c_void_p(torch.cuda.current_stream().cuda_stream), X16.shape[0], X16.device
    bf = lambda *s: torch.empty(s, dtype=torch.bfloat16, device=dev)

    def gemm(A, tA, lda, W, tB, ldb, M, N, K, bias=None, relu=0, c32=None, c16=None):
        native.check(L.poyd_gemm_bf16(p(A), lda, tA, p(W), ldb, tB, M, N, K, p(bias), relu,
                                      p(c32), p(c16), N, 0, st))

    H, a = [], X16
    for i in range(3):
        H.append(bf(B, DIMS[i + 1]))
        gemm(a, 0, DIMS[i], net.W16[i], 0, DIMS[i + 1], B, DIMS[i + 1], DIMS[i], net.b[i], 1,
             c16=H[i])
        a = H[i]
    y = torch.empty(B, device=dev)
    native.check(L.poyd_mlp_head_forward(p(a), p(net.W16[3]), p(net.b[3]), B, DIMS[3], p(y), st))
    gW = [torch.empty_like(w) for w in net.W]
    gb = [torch.empty_like(b) for b in net.b]
    loss, dZ = torch.zeros(1, device=dev), bf(B, DIMS[3])
    native.check(L.poyd_mlp_head_backward(p(H[2]), p(net.W16[3]), p(y), p(target), B, DIMS[3],
                                          p(dZ), p(gW[3]), p(gb[3]), p(loss), st))
    for i in (2, 1, 0):
        K, N = DIMS[i], DIMS[i + 1]
        gemm(X16 if i == 0 else H[i - 1], 1, K, dZ, 0, N, K, N, B, c32=gW[i])
        native.check(L.poyd_colsum_bf16(p(dZ), B, N, p(gb[i]), st))
        if i:
            dH, dZn = bf(B, K), bf(B, K)
            gemm(dZ, 0, N, net.W16[i], 1, N, B, K, N, c16=dH)
            native.check(L.poyd_relu_grad_bf16(p(dH), p(H[i - 1]), p(dZn), dH.numel(), st))
            dZ = dZn
    return H, y, loss, gW, gb


@pytest.mark.parametrize("rows", [1, 15, 16, 17, 33, 127, 128, 129, 1000, 19457])
def test_fused_training_equals_layers(rows):
    net = mlp.MLP(seed=rows)
    g = torch.Generator(device="cpu").manual_seed(rows)
    X = torch.randn((rows, 32), generator=g).cuda().to(torch.bfloat16)
    t = torch.randn(rows, generator=g).cuda()
    for b in net.b:
        b.copy_(0.1 * torch.randn(b.shape, generator=g).cuda())
    H, y, loss, gW, gb = layers(net, X, t)
    y1 = net.forward(X)
    loss1, gW1, gb1 = net.backward(t)
    for i in range(3):
        ulp = (net.H[i].view(torch.int16).int() - H[i].view(torch.int16).int()).abs().max()
        assert int(ulp) <= 1, i
    assert rel(y1, y) < 2 ** -12
    assert rel(loss1, loss) < 2 ** -12
    for i in range(4):
        assert rel(gW1[i], gW[i]) < 2 ** -10, i
        assert rel(gb1[i], gb[i]) < 2 ** -10, i


def test_adam_step_equals_single_tensor_entries():
    net, ref = mlp.MLP(seed=2), mlp.MLP(seed=2)
    g = torch.Generator(device="cpu").manual_seed(7)
    p = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for step in (1, 2, 3):
        gW = [torch.randn(w.shape, generator=g).cuda() for w in net.W]
        gb = [torch.randn(b.shape, generator=g).cuda() for b in net.b]
        net.step(gW, gb)
        for w, w16, gr, m, v in zip(ref.W + ref.b, ref.W16 + [None] * 4, gW + gb,
                                    ref.mW + ref.mb, ref.vW + ref.vb):
            native.check(ref.L.poyd_adam_step(p(w), p(w16), p(gr), p(m), p(v), w.numel(), 1e-3,
                                              0.9, 0.999, 1e-8, step, st))
    for a, b in zip(net.W + net.b + net.W16, ref.W + ref.b + ref.W16):
        assert torch.equal(a, b)
