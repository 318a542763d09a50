"""The plan's counts over a pair's codes (k_lin_plan: single bytes up to the first
16-byte boundary and after the last, 16 bytes a load between): bands from the
gap-bearing codes at every alignment and length around those edges, and the
refusal of a code above 31 wherever it stands."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, native

pytestmark = pytest.mark.gpu


def band_cells(a, b):
    l1, l2 = max(len(a), len(b)), min(len(a), len(b))
    gaps = max(int((a & 16 != 0).sum()), int((b & 16 != 0).sum()))
    dif, lower = l1 - l2, int(l1 * 0.10)
    dw = gaps + (lower // 2 if dif < lower else 2)
    width, height = min(50 + dw, l2), min(dif + 50 + dw, l1)
    full = np.float32(1.5) * np.float32(l2) <= np.float32(l1) or (2 * height >= l1 and 8 >= l1 - height)
    delta = 1 if not full and 2 * height < l1 else 0
    dlo, dhi = (-(l1 - 1), l2 - 1) if full else (delta - height, width - 1)
    r = np.arange(l1)
    return int(np.maximum(0, np.minimum(dhi, l2 - 1 - r) - np.maximum(dlo, -r) + 1).sum())


@pytest.mark.parametrize("shift", [0, 1, 7, 15])
def test_bands_at_every_alignment(shift):
    rng = np.random.default_rng(shift)
    lens = list(range(1, 36)) + [47, 48, 49, 63, 64, 65, 255, 256, 257, 511, 529, 1000]
    seqs = []
    for n in lens * 2:
        s = rng.choice(np.array([1, 2, 4, 8], np.uint8), n)
        s[0] = 16
        s[rng.random(n) < 0.2] |= 16
        seqs.append(s)
    buf = np.concatenate([np.full(shift, 255, np.uint8)] + seqs + [np.full(64, 255, np.uint8)])
    off = shift + np.concatenate([[0], np.cumsum([len(s) for s in seqs])])[:-1]
    ia = rng.permutation(len(seqs))
    ib = rng.permutation(len(seqs))
    t = lambda x, d: torch.from_numpy(np.asarray(x, d)).cuda()
    ln = np.array([len(s) for s in seqs])
    b = align.PairBatch(t(buf, np.uint8), t(off[ia], np.int64), t(ln[ia], np.int32),
                        t(off[ib], np.int64), t(ln[ib], np.int32))
    cm = align.CostMatrix.default()
    cells = align.cost_2(b, cm, band_cells=True)[1].cpu().numpy()
    assert cells.tolist() == [band_cells(seqs[x], seqs[y]) for x, y in zip(ia, ib)]
    # a code above 31 anywhere in a sequence of the batch
    x = len(lens) - 1  # 1,000 codes
    for p in (1, 2, 14, 15, 16, 17, 31, 500, 983, 984, 998, 999):
        bad = b.seq.clone()
        bad[int(off[x]) + p] = 33
        with pytest.raises(native.PoydError):
            align.cost_2(align.PairBatch(bad, b.a_off, b.a_len, b.b_off, b.b_len), cm)
