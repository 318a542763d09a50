"""Packing of more than 4,096 results, four pairs a block: lengths around a warp's bytes
(128), its vectors and what the block copies together (16,384), mixed within a block, at
every alignment, and the ends of the last block; slots and results as poyd_pack_slots and
poyd_pack_alignments take them.  Every byte is that of a copy by tensor operations."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align

pytestmark = pytest.mark.gpu
LENS = [0, 1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 130, 500, 2048, 2049]


@pytest.mark.parametrize("n", [4097, 4098, 4099, 4100, 70001])
def test_blocks_of_four_pairs(n):
    rng = np.random.default_rng(n)
    na = rng.choice(LENS, n)
    nm = np.maximum(na - rng.integers(0, 3, n), 0)
    if n < 5000:
        na[[0, 5, 6, n - 1]], nm[[0, 5, 6, n - 1]] = [16384, 16385, 40000, 16385], [16384, 3, 39999, 16385]
    cap = (na + rng.integers(0, 9, n) + 3) // 4 * 4
    off = np.zeros(n, np.int64)
    off[1:] = np.cumsum(4 * cap)[:-1]
    out = torch.randint(0, 255, (int(off[-1] + 4 * cap[-1]),), dtype=torch.uint8, device="cuda")
    d = lambda x, t: torch.from_numpy(np.ascontiguousarray(x)).to("cuda", t)
    ln = np.stack([na, nm], 1).reshape(-1)
    r = align.AlignResult(torch.zeros(n, dtype=torch.int32, device="cuda"), out, d(off, torch.int64),
                          d(ln, torch.int32), d(cap, torch.int64), None)
    got = r.pack().packed
    r.cap = r.cap.to(torch.int32)  # the tensor operations' path
    again = r.pack().packed
    # where each packed byte comes from: sequence k of pair i ends at off + (k + 1) cap
    sizes = np.stack([na, na, na, nm], 1).reshape(-1)
    ends = (off[:, None] + cap[:, None] * np.arange(1, 5)).reshape(-1)
    at = np.cumsum(sizes)
    src = np.repeat(ends - at, sizes) + np.arange(at[-1])
    want = out[torch.from_numpy(src).cuda()]
    assert torch.equal(got, want) and torch.equal(again, want)
