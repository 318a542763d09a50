"""Large affine batches with many pairs of few rows and many columns, which go to the
rows kernels once there are enough of them (csrc/affine.cu), beside even ones, which
do not: costs, aligned sequences and medians are those of a small batch of the same
pairs, which the antidiagonal kernel takes, and of the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from poyd_gb300 import align, synth

pytestmark = pytest.mark.gpu

SHAPES = [(0, 41), (1, 60), (1, 200), (5, 100), (8, 439), (10, 440), (20, 300), (3, 470), (3, 480),
          (80, 400), (100, 300), (60, 60), (7, 7), (300, 310), (0, 0), (440, 10), (60, 2)]


@pytest.mark.parametrize("codes", [0.0, 0.05])
@pytest.mark.parametrize("reps", [400, 1500])
def test_uneven_pairs_among_even_ones(reps, codes):
    rng = np.random.default_rng(int(reps + 100 * codes))
    A, B = [], []
    for la, lb in SHAPES:
        a, b = synth.random_dna(rng, la, 0.05), synth.random_dna(rng, lb, 0.05)
        k = min(la, lb)
        b[lb // 3:lb // 3 + k] = a[:len(b[lb // 3:lb // 3 + k])]
        for s in (a, b):
            s[rng.random(len(s)) < codes] |= 16
        A.append(synth.with_gap(a))
        B.append(synth.with_gap(b))
    cm, om = align.CostMatrix.dna(1, 2, 3), O.cm_dna(1, 2, 3)
    one = align.PairBatch.from_host(A, B)
    many = align.PairBatch(one.seq, *[t.repeat(reps) for t in (one.a_off, one.a_len, one.b_off, one.b_len)])
    want, got = align.align_2(one, cm, dos_empty=True), align.align_2(many, cm, dos_empty=True)
    assert torch.equal(got.cost, want.cost.repeat(reps))
    assert torch.equal(got.out_len, want.out_len.repeat(reps))
    assert torch.equal(got.pack().packed, want.pack().packed.repeat(reps))
    assert torch.equal(align.cost_2(many, cm)[0], align.cost_2(one, cm)[0].repeat(reps))
    for i, r in enumerate(want.to_host()):
        c, med, ra, rb, _ = O.dos_median(A[i], B[i], om)
        assert r["cost"] == c and np.array_equal(r["median"], med), i
        assert np.array_equal(r["a"], ra) and np.array_equal(r["b"], rb), i
