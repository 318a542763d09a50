"""The fused tcgen05 forward (csrc/mlp_forward.cu) against the layer-by-layer
entry points (poyd_gemm_bf16, poyd_mlp_head_forward) at the edges of its
128-row tiles.

Tolerance: two fp32 sums of at most 256 products in different orders differ
by far less than a bf16 ulp, so a hidden activation may round to the
neighbouring bf16 value and no further; such a step is 2^-8 of one of a row's
256 terms and rare (a fraction of about 2^-24 * 256 / 2^-8 = 2^-8 at most), so
predictions agree to 2^-8 * 2^-4 = 2^-12 of their norm."""
import ctypes as C

import pytest
import torch

from poyd_gb300 import mlp, native

pytestmark = pytest.mark.gpu
DIMS = mlp.DIMS


def rel(a, b):
    a, b = a.double(), b.double()
    n = b.norm().item()
    return (a - b).norm().item() / n if n else a.norm().item()


def layers(net, X16):
    """The forward through the layer-by-layer entry points."""
    p = lambda t: C.c_void_p(t.data_ptr())
    st, B, H = C.c_void_p(torch.cuda.current_stream().cuda_stream), X16.shape[0], [X16]
    for i in range(3):
        K, N = DIMS[i], DIMS[i + 1]
        H.append(torch.empty((B, N), dtype=torch.bfloat16, device=X16.device))
        native.check(net.L.poyd_gemm_bf16(p(H[i]), K, 0, p(net.W16[i]), N, 0, B, N, K,
                                          p(net.b[i]), 1, None, p(H[i + 1]), N, 0, st))
    y = torch.empty(B, device=X16.device)
    native.check(net.L.poyd_mlp_head_forward(p(H[3]), p(net.W16[3]), p(net.b[3]), B, DIMS[3],
                                             p(y), st))
    return H[1:], y


@pytest.mark.parametrize("rows", [1, 15, 127, 128, 129, 1000, 19457])
def test_fused_forward_equals_layers(rows):
    net = mlp.MLP(seed=rows)
    g = torch.Generator(device="cpu").manual_seed(rows)
    X = torch.randn((rows, 32), generator=g).cuda().to(torch.bfloat16)
    for b in net.b:
        b.copy_(0.1 * torch.randn(b.shape, generator=g).cuda())
    H, y = layers(net, X)
    y1 = net.forward(X)
    for i in range(3):
        ulp = (net.H[i].view(torch.int16).int() - H[i].view(torch.int16).int()).abs().max()
        assert int(ulp) <= 1, i
    assert rel(y1, y) < 2 ** -12


def test_unaligned_rows_are_taken():
    net = mlp.MLP(seed=4)
    flat = torch.randn(65 * 32 + 1, generator=torch.Generator().manual_seed(3)).cuda()
    X = flat[1:].view(65, 32)  # starts 4 bytes off
    assert torch.equal(net.predict(X), net.predict(X.clone()))
    X16 = torch.cat([X.new_zeros(1, dtype=torch.bfloat16), X.to(torch.bfloat16).flatten()])[1:]
    assert torch.equal(net.forward(X16.view(65, 32)), net.predict(X))
