"""The fused forward (csrc/mlp_forward.cu) of the most rows that its 32-bit count
holds: the last tile of 128 ends past 2^31."""
import ctypes as C

import pytest
import torch

from poyd_gb300 import mlp, native

pytestmark = pytest.mark.gpu


def test_last_rows_of_31_bits():
    rows = 2 ** 31 - 1
    if torch.cuda.mem_get_info()[0] < (170 << 30):
        pytest.skip("needs 170 GB of device memory")
    net = mlp.MLP(seed=2)
    g = torch.Generator(device="cpu").manual_seed(2)
    ends = torch.randn((300, 32), generator=g).cuda().to(torch.bfloat16)
    want = net.predict(ends)
    X, y = None, None
    try:
        X = torch.zeros((rows, 32), dtype=torch.bfloat16, device="cuda")
        y = torch.empty(rows, dtype=torch.float32, device="cuda")
        X[:300], X[-300:] = ends, ends
        w, b = net.W16, net.b
        native.check(net.L.poyd_mlp_forward_rows(
            X.data_ptr(), 0, rows, w[0].data_ptr(), b[0].data_ptr(), w[1].data_ptr(), b[1].data_ptr(),
            w[2].data_ptr(), b[2].data_ptr(), w[3].data_ptr(), b[3].data_ptr(), None, None, None,
            y.data_ptr(), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert torch.equal(y[:300], want) and torch.equal(y[-300:], want)
        assert bool((y[300:-300] == y[300]).all())
    finally:
        X = y = None
        torch.cuda.empty_cache()
