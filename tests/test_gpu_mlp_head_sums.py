"""The output bias's gradient and the loss of poyd_mlp_backward are summed row
after row like poyd_mlp_head_backward's: the same bits, at the edges of the
1,024-row turns (csrc/mlp_train.cu)."""
import ctypes as C

import pytest
import torch

from poyd_gb300 import mlp, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 1023, 1024, 1025, 2048, 5001])
def test_the_layerwise_sums(rows):
    net = mlp.MLP(seed=rows)
    g = torch.Generator(device="cpu").manual_seed(rows)
    X = torch.randn((rows, 32), generator=g).cuda().to(torch.bfloat16)  # as forward takes it
    t = torch.randn(rows, generator=g).cuda()
    y = net.forward(X)
    loss, gW, gb = net.backward(t)
    p = lambda x: C.c_void_p(x.data_ptr())
    dZ = torch.empty((rows, 128), dtype=torch.bfloat16, device="cuda")
    dw, db, l = torch.empty(128, device="cuda"), torch.empty(1, device="cuda"), torch.empty(1, device="cuda")
    native.check(net.L.poyd_mlp_head_backward(p(net.H[2]), p(net.W16[3]), p(y), p(t), rows, 128, p(dZ),
                                              p(dw), p(db), p(l),
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(gb[3].view(-1), db) and torch.equal(loss.view(-1), l)
