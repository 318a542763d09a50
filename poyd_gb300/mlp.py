"""The join-proposal MLP (32-256-256-128-1, ReLU) on the project's own BF16
tensor-core kernels (csrc/mlp_forward.cu, csrc/mlp_train.cu): forward, backward and Adam, with FP32
master weights and FP32 accumulation.  No reference counterpart: this is
the learned proposal that orders the candidate joins of a search pass."""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import native

DIMS = (32, 256, 256, 128, 1)


def _lib():
    L = native.lib()
    vp, i32, i64, f32 = C.c_void_p, C.c_int32, C.c_int64, C.c_float
    L.poyd_gemm_bf16.argtypes = [vp, i32, i32, vp, i32, i32, i32, i32, i32, vp, i32, vp, vp,
                                 i32, i32, vp]
    L.poyd_relu_grad_bf16.argtypes = [vp, vp, vp, i64, vp]
    L.poyd_colsum_bf16.argtypes = [vp, i32, i32, vp, vp]
    L.poyd_mlp_head_forward.argtypes = [vp, vp, vp, i32, i32, vp, vp]
    L.poyd_mlp_head_backward.argtypes = [vp, vp, vp, vp, i32, i32, vp, vp, vp, vp, vp]
    L.poyd_adam_step.argtypes = [vp, vp, vp, vp, vp, i64, f32, f32, f32, f32, i32, vp]
    L.poyd_to_bf16.argtypes = [vp, vp, i64, vp]
    L.poyd_mlp_forward_rows.argtypes = [vp, i32, i32] + [vp] * 13
    L.poyd_mlp_backward.argtypes = [vp, i32] + [vp] * 13
    L.poyd_adam_step_all.argtypes = [i32] + [vp] * 6 + [f32, f32, f32, f32, i32, vp]
    return L


def _aligned(t):
    """t, or a copy when its rows do not start on 16 bytes (the kernels' loads)."""
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _ptrs(ts):
    return (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


def _st():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


class MLP:
    """Parameters: W_l [in, out] row-major (fp32 master + bf16 copy), b_l fp32."""

    def __init__(self, seed: int = 0, device="cuda"):
        self.dev = torch.device(device)
        rng = np.random.default_rng(seed)
        self.W, self.W16, self.b = [], [], []
        for i in range(4):
            fan_in, fan_out = DIMS[i], DIMS[i + 1]
            w = rng.normal(0, np.sqrt(2.0 / fan_in), size=(fan_in, fan_out)).astype(np.float32)
            self.W.append(torch.from_numpy(w).to(self.dev))
            self.b.append(torch.zeros(fan_out, dtype=torch.float32, device=self.dev))
        self.W16 = [w.to(torch.bfloat16) for w in self.W]
        self.mW = [torch.zeros_like(w) for w in self.W]
        self.vW = [torch.zeros_like(w) for w in self.W]
        self.mb = [torch.zeros_like(b) for b in self.b]
        self.vb = [torch.zeros_like(b) for b in self.b]
        self.steps = 0
        self.L = _lib()

    def state(self):
        return {"W": [w.cpu().numpy() for w in self.W], "b": [b.cpu().numpy() for b in self.b]}

    def _forward(self, X, fp32, H, y):
        W, b = self.W16, self.b
        native.check(self.L.poyd_mlp_forward_rows(
            X.data_ptr(), fp32, X.shape[0], W[0].data_ptr(), b[0].data_ptr(), W[1].data_ptr(),
            b[1].data_ptr(), W[2].data_ptr(), b[2].data_ptr(), W[3].data_ptr(), b[3].data_ptr(),
            *[h.data_ptr() if h is not None else None for h in H], y.data_ptr(), _st()))

    def forward(self, X16: torch.Tensor):
        """X16 [B, 32] bf16 -> predictions [B] fp32 (activations kept)."""
        B = X16.shape[0]
        self.X16 = X16
        self.H = [torch.empty((B, DIMS[i + 1]), dtype=torch.bfloat16, device=self.dev)
                  for i in range(3)]
        self.y = torch.empty(B, dtype=torch.float32, device=self.dev)
        self._forward(_aligned(X16), 0, self.H, self.y)
        return self.y

    def backward(self, target: torch.Tensor):
        """Gradients of mean squared error; returns (loss, gW list, gb list)."""
        B = self.X16.shape[0]
        gW = [torch.empty_like(w) for w in self.W]
        gb = [torch.empty_like(b) for b in self.b]
        loss = torch.empty(1, dtype=torch.float32, device=self.dev)
        dZ = torch.empty(B * sum(DIMS[1:4]), dtype=torch.bfloat16, device=self.dev)
        X = _aligned(self.X16)
        native.check(self.L.poyd_mlp_backward(
            X.data_ptr(), B, *[h.data_ptr() for h in self.H], self.W16[1].data_ptr(),
            self.W16[2].data_ptr(), self.W16[3].data_ptr(), self.y.data_ptr(), target.data_ptr(),
            dZ.data_ptr(), _ptrs(gW), _ptrs(gb), loss.data_ptr(), _st()))
        return loss, gW, gb

    def step(self, gW, gb, lr=1e-3, b1=0.9, b2=0.999, eps=1e-8):
        self.steps += 1
        w = self.W + self.b
        w16 = (C.c_void_p * 8)(*[x.data_ptr() for x in self.W16], None, None, None, None)
        sizes = (C.c_int64 * 8)(*[x.numel() for x in w])
        native.check(self.L.poyd_adam_step_all(
            8, _ptrs(w), w16, _ptrs(list(gW) + list(gb)), _ptrs(self.mW + self.mb),
            _ptrs(self.vW + self.vb), sizes, lr, b1, b2, eps, self.steps, _st()))

    def fit(self, X: torch.Tensor, y: torch.Tensor, epochs=3, batch=4096, lr=1e-3, seed=0):
        """Mini-batch Adam on (X fp32 [n, 32], y fp32 [n]); returns losses."""
        g = torch.Generator(device="cpu").manual_seed(seed)
        n = X.shape[0]
        X16 = X.to(torch.bfloat16)
        losses = []
        for _ in range(epochs):
            perm = torch.randperm(n, generator=g).to(self.dev)
            for s in range(0, n - batch + 1, batch):
                idx = perm[s:s + batch]
                self.forward(X16[idx].contiguous())
                loss, gW, gb = self.backward(y[idx].contiguous())
                self.step(gW, gb, lr=lr)
                losses.append(loss)
        return [float(l.item()) for l in losses[-10:]]

    def predict(self, X: torch.Tensor) -> torch.Tensor:
        """Predictions for the rows of X (fp32 [n, 32]) in one fused launch
        (``poyd_mlp_forward_rows``), equal to ``forward``'s."""
        y = torch.empty(X.shape[0], dtype=torch.float32, device=self.dev)
        if X.shape[0] == 0:
            return y
        if X.dtype == torch.float32 and X.is_contiguous() and X.device == y.device:
            self._forward(_aligned(X), 1, (None, None, None), y)  # rounded to bf16 on the way in
        else:
            self._forward(_aligned(X.to(torch.bfloat16).contiguous()), 0, (None, None, None), y)
        return y
