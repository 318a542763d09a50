"""An affine batch of more than 2^27 pairs, whose plan and traceback take a warp a
pair: 2^32 threads are not enough.  The pairs share two short sequences; the last
ones differ from the others and have the oracle's costs and alignments."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from poyd_gb300 import align, native

pytestmark = pytest.mark.gpu


def test_more_pairs_than_warps_in_32_bits():
    n, odd = (1 << 27) + 5, 7
    if torch.cuda.mem_get_info()[0] < (120 << 30):
        pytest.skip("needs 120 GB of device memory")
    s = [np.array(x, np.uint8) for x in ([16, 1, 2], [16, 4, 8])]
    seq = torch.from_numpy(np.concatenate(s + [np.zeros(64, np.uint8)])).cuda()
    a_off = torch.zeros(n, dtype=torch.int64, device="cuda")
    b_off = torch.zeros_like(a_off)
    b_off[-odd:] = 3
    ln = torch.full((n,), 3, dtype=torch.int32, device="cuda")
    batch = align.PairBatch(seq, a_off, ln, b_off, ln)
    cm, om = align.CostMatrix.dna(1, 2, 3), O.cm_dna(1, 2, 3)
    r = None
    try:
        r = align.align_2(batch, cm, dos_empty=True)
        for i, b in ((0, s[0]), (n - odd - 1, s[0]), (n - odd, s[1]), (n - 1, s[1])):
            c, med, ra, rb, _ = O.dos_median(s[0], b, om)
            k, o = int(r.cap[i]), int(r.out_off[i])
            la, lm = r.out_len.view(-1, 2)[i].tolist()
            at = lambda q, m: r.out[o + q * k - m:o + q * k].cpu().numpy()
            assert int(r.cost[i]) == c, i
            assert np.array_equal(at(1, la), ra) and np.array_equal(at(2, la), rb), i
            assert np.array_equal(at(4, lm), med), i
        for t in (r.cost, r.out_len.view(-1, 2)[:, 0], r.out_len.view(-1, 2)[:, 1]):
            assert bool((t[:-odd] == t[0]).all()) and bool((t[-odd:] == t[-1]).all())
        del t
    finally:
        r = None
        native.check(native.lib().poyd_workspace_release())
        torch.cuda.empty_cache()
