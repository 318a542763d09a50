"""Packing of alignment results (k_pack_alignments): lengths around the 16-byte
stores, slots whose sequences start at every byte of a word, against a byte copy."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align

pytestmark = pytest.mark.gpu


def test_every_length_and_offset():
    rng = np.random.default_rng(4)
    lens = [(n, m) for n in (0, 1, 2, 15, 16, 17, 31, 32, 33, 47, 300, 2051) for m in (0, 1, 15, 16, 21, n)]
    cap = np.array([(max(n, m) + 2 + 3) // 4 * 4 + 4 * (i % 3) for i, (n, m) in enumerate(lens)], np.int64)
    off = np.cumsum(4 * cap + 4) - (4 * cap + 4)
    out = rng.integers(0, 256, int(off[-1] + 4 * cap[-1]), dtype=np.uint8)
    want = []
    for (n, m), c, o in zip(lens, cap, off):
        for k, ln in enumerate((n, n, n, m)):
            want.append(out[o + (k + 1) * c - ln:o + (k + 1) * c])
    t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()
    r = align.AlignResult(torch.zeros(len(lens), dtype=torch.int32).cuda(), t(out), t(off),
                          t(np.array(lens, np.int32).ravel()), t(cap), None)
    assert np.array_equal(r.pack().packed.cpu().numpy(), np.concatenate(want))
