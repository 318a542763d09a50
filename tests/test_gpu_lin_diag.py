"""The antidiagonal kernel of large linear batches (csrc/linear_diag.cu): each
of its classes (8, 16 or 32 lanes, by the batch's size; 8 to 24 diagonals a lane,
by the band), both kinds of band offset, sequences of a few characters, all-gap
ones and bands that none of its classes holds.  Costs, aligned sequences and
medians equal the warp-per-pair kernel's (a tuned variant keeps that one) and, for
a sample, the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from poyd_gb300 import align, native, synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def warp_per_pair():
    def on():
        for al in (0, 1):
            for lg in range(0, 15):
                for w in range(0, 16):
                    native.check(native.lib().poyd_autotune_set(torch.cuda.current_device(), al, lg, w,
                                                                1, 0, -1))
    yield on
    native.check(native.lib().poyd_autotune_clear())


def pairs(rng, n):
    A, B = [], []
    for i in range(n):
        kind = i % 8
        hi = (4, 20, 60, 120, 200, 400, 900, 1300)[kind]
        la = int(rng.integers(1, hi + 1))
        lb = max(1, int(la * rng.uniform(0.4, 1.0) if kind == 3 else la * rng.uniform(0.93, 1.07)))
        if i in (11, 12):
            la, lb = 1400, 700 - 100 * (i - 11)  # the whole matrix
        a = synth.random_dna(rng, max(la, lb), 0.05)
        b = synth.mutate(rng, a, 0.15, 0.03)[:lb - 1]
        b = np.concatenate([b, synth.random_dna(rng, lb - 1 - len(b))])
        a = a[:la - 1].copy()
        a[rng.random(len(a)) < rng.choice([0.0, 0.05, 0.1])] |= 16  # a median's optional positions
        A.append(synth.with_gap(a))
        B.append(synth.with_gap(b))
    A[5] = np.array([16, 16, 16], np.uint8)
    return A, B


@pytest.mark.parametrize("sub,indel", [(1, 2), (7, 3)])
@pytest.mark.parametrize("size", [0.6, 1.3, 2.2])  # of the resident warps: 32, 16 and 8 lanes at least
def test_matches_the_warp_per_pair_kernel(warp_per_pair, size, sub, indel):
    n = int(size * 16 * torch.cuda.get_device_properties(0).multi_processor_count) + 1
    A, B = pairs(np.random.default_rng(n + sub), n)
    cm, om = align.CostMatrix.dna(sub, indel), O.cm_dna(sub, indel, -1)
    b = align.PairBatch.from_host(A, B)

    def all_results():
        r = align.align_2(b, cm, dos_empty=True)
        bad = align.align_2(b, cm)
        return [r.cost, r.out_len, r.pack().packed, bad.cost, bad.out_len] + \
               [align.cost_2(b, cm, d)[0] for d in (None, "dos")], r

    got, res = all_results()
    warp_per_pair()
    for k, (x, y) in enumerate(zip(got, all_results()[0])):
        assert torch.equal(x, y), k
    host = res.to_host()
    for i in (0, 1, 2, 3, 5, 6, 11):
        c, med, ra, rb, wg = O.dos_median(A[i], B[i], om)
        x = host[i]
        assert x["cost"] == c and np.array_equal(x["median"], med), i
        assert np.array_equal(x["a"], ra) and np.array_equal(x["b"], rb), i
