"""Fitch distances at the edges of a lane's vectors (16 characters), a warp's row
of vectors (512) and its four rows in flight (2,048), with non-zero bytes past the
rows' ends, against a count on the CPU."""
import ctypes as C

import numpy as np
import pytest
import torch

from poyd_gb300 import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 15, 16, 17, 511, 512, 513, 1535, 2047, 2048, 2049, 4500])
def test_distances_at_vector_and_batch_edges(length):
    rng = np.random.default_rng(length)
    stride, nodes, n = (length + 15) // 16 * 16 + 16, 9, 70
    rows = rng.choice(np.array([1, 2, 4, 8, 0x81, 0xFF, 0x80], np.uint8), (nodes, stride))
    a, b = rng.integers(0, nodes, n).astype(np.int32), rng.integers(0, nodes, n).astype(np.int32)
    t = [torch.from_numpy(x).cuda() for x in (rows, a, b)]
    dist = torch.empty(n, dtype=torch.int64, device="cuda")
    p = lambda x: C.c_void_p(x.data_ptr())
    L = native.lib()
    L.poyd_nonadd8_distance_batch.argtypes = [C.c_void_p, C.c_int64, C.c_int32, C.c_int32] + [C.c_void_p] * 4
    native.check(L.poyd_nonadd8_distance_batch(p(t[0]), stride, length, n, p(t[1]), p(t[2]), p(dist),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    want = ((rows[a, :length] & rows[b, :length]) == 0).sum(1)
    assert dist.cpu().tolist() == want.tolist()
