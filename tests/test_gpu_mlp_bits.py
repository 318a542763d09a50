"""The fused forward (csrc/mlp_forward.cu) against the layer-by-layer kernels
(poyd_gemm_bf16, poyd_mlp_head_forward), which accumulate k in the same chunks of 16 and
sum the head in the same tree: predictions and hidden activations are the same bits, for
both entry points (weights as rows of inputs or of outputs), bf16 and fp32 inputs, weights
on 16- and on 4-byte boundaries, and weights and biases that training has moved."""
import ctypes as C

import pytest
import torch

from poyd_gb300 import mlp, native
from tests.test_gpu_mlp_fused import layers

pytestmark = pytest.mark.gpu


def shifted(t, elements):
    """A copy of t that starts `elements` past a 16-byte boundary."""
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=t.device)
    return flat[elements:elements + t.numel()].view(t.shape).copy_(t)


@pytest.mark.parametrize("rows", [1, 31, 127, 128, 129, 1000, 19457])
@pytest.mark.parametrize("shift", [0, 2])
def test_same_bits_as_the_layers(rows, shift):
    net = mlp.MLP(seed=rows)
    g = torch.Generator(device="cpu").manual_seed(rows)
    for b in net.b:
        b.copy_(0.1 * torch.randn(b.shape, generator=g).cuda())
    X = torch.randn((max(rows, 512), 32), generator=g).cuda()
    net.fit(X, torch.randn(X.shape[0], generator=g).cuda(), epochs=3, batch=512, lr=1e-2)
    X = X[:rows].contiguous()
    X16 = X.to(torch.bfloat16)
    H, want = layers(net, X16)

    W = [shifted(w, shift) for w in net.W16[:3]]
    Wt = [shifted(w.t().contiguous(), shift) for w in net.W16[:3]]
    w4, b = net.W16[3], net.b
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    L = net.L
    L.poyd_mlp_forward.argtypes = [C.c_void_p, C.c_int32] + [C.c_void_p] * 10
    pairs = lambda ws: [p for w, bb in zip(ws, b) for p in (w.data_ptr(), bb.data_ptr())]
    y = lambda: torch.full((rows,), float("nan"), device="cuda")
    got = [y() for _ in range(4)]
    kept = [torch.full_like(h, float("nan")) for h in H]
    native.check(L.poyd_mlp_forward(X16.data_ptr(), rows, *pairs(Wt), w4.data_ptr(), b[3].data_ptr(),
                                    got[0].data_ptr(), st))
    for k, (x, fp32, hs) in enumerate(((X16, 0, None), (X, 1, None), (X16, 0, kept)), 1):
        native.check(L.poyd_mlp_forward_rows(
            x.data_ptr(), fp32, rows, *pairs(W), w4.data_ptr(), b[3].data_ptr(),
            *([h.data_ptr() for h in hs] if hs else [None] * 3), got[k].data_ptr(), st))
    for k, p in enumerate(got):
        assert torch.equal(p, want), k
    for i, (h, r) in enumerate(zip(kept, H)):
        assert torch.equal(h, r), i


def test_some_activations_only():
    net = mlp.MLP(seed=8)
    X16 = torch.randn((200, 32), generator=torch.Generator().manual_seed(8)).cuda().to(torch.bfloat16)
    H, want = layers(net, X16)
    w, b = net.W16, net.b
    for i in range(3):
        h = torch.full_like(H[i], float("nan"))
        y = torch.empty(200, device="cuda")
        at = [h.data_ptr() if i == j else None for j in range(3)]
        native.check(net.L.poyd_mlp_forward_rows(
            X16.data_ptr(), 0, 200, w[0].data_ptr(), b[0].data_ptr(), w[1].data_ptr(), b[1].data_ptr(),
            w[2].data_ptr(), b[2].data_ptr(), w[3].data_ptr(), b[3].data_ptr(), *at, y.data_ptr(),
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert torch.equal(h, H[i]) and torch.equal(y, want), i
