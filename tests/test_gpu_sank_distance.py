"""Sankoff distances and medians (csrc/fitch_sankoff.cu) over every state count,
infinite and negative costs, rows on 4-, 8- and 16-byte boundaries and character
counts around a warp's 32: the distance equals the sum of min c - min a - min b
of a 64-bit restatement of elt_median with its saturating infinity, and the
median's c that restatement's."""
import ctypes as C

import numpy as np
import pytest
import torch

from poyd_gb300 import native

pytestmark = pytest.mark.gpu
INF = native.SANK_INF


def sadd(a, b):
    return np.where((a >= INF) | (b >= INF), INF, a + b)


def reference(tcm, a, b):
    """(c [n, ch, k], distance [n]) of rows a, b [n, ch, k]."""
    t = tcm.astype(np.int64)
    half = lambda s: np.minimum(sadd(t[None, None], s[:, :, None, :]).min(-1), INF)
    c = sadd(half(a), half(b))
    m = lambda x: np.minimum(x.min(-1), INF)
    return c, (m(c) - m(a) - m(b)).sum(-1)


@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("shift", [0, 1, 2])  # rows start 4 * shift bytes off a 16-byte boundary
def test_distances_and_medians(k, shift):
    rng = np.random.default_rng(10 * k + shift)
    p = lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for nchar, forbid, low in [(1, 0, 0), (31, 1, 0), (32, 0, 0), (33, 1, 1), (200, 1, 0)]:
        nn, n = 30, 77
        nodes = rng.integers(0, 60, (nn, nchar, k)).astype(np.int32)
        nodes[rng.random(nodes.shape) < 0.3] = INF
        nodes[0] = INF                       # a row with no finite state
        nodes[1] = INF - 3                   # sums past the infinity
        if low:
            nodes[2, 0] = -5
        tcm = rng.integers(0, 9, (k, k)).astype(np.int32)
        if forbid:
            tcm[0, k - 1] = INF
        ai, bi = (rng.integers(0, nn, n).astype(np.int32) for _ in range(2))
        flat = torch.zeros(nodes.size + 4, dtype=torch.int32, device="cuda")
        dn = flat[shift:shift + nodes.size]
        dn.copy_(torch.from_numpy(nodes.ravel()))
        dt, da, db = (torch.from_numpy(x).cuda() for x in (tcm, ai, bi))
        dist = torch.empty(n, dtype=torch.int64, device="cuda")
        s = torch.empty((n, nchar, k), dtype=torch.int32, device="cuda")
        L = native.lib()
        native.check(L.poyd_sank_distance_batch(p(dn), nchar, k, p(dt), n, p(da), p(db), p(dist), st))
        native.check(L.poyd_sank_median_batch(p(dn), nchar, k, p(dt), n, p(da), p(db), p(s), None,
                                              None, st))
        x = nodes.astype(np.int64)
        c, d = reference(tcm, x[ai], x[bi])
        assert np.array_equal(s.cpu().numpy(), c.astype(np.int32)), (nchar, forbid, low)
        assert np.array_equal(dist.cpu().numpy(), d), (nchar, forbid, low)
