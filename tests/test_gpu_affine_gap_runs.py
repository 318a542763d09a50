"""Long gaps in affine alignments, whose columns k_aff_walk (csrc/affine_diag.cu) takes
32 at a time: gaps of lengths around that in either sequence, inside the band and at
its edges, one after another and with gap-bearing codes, against the 32-bit rows
kernel's walk and, for a sample, the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from poyd_gb300 import align, synth

pytestmark = pytest.mark.gpu
RUNS = [1, 2, 31, 32, 33, 34, 63, 64, 65, 66, 97, 130, 200, 300, 429]


@pytest.mark.parametrize("codes", [0.0, 0.05])
@pytest.mark.parametrize("model,reps", [((1, 2, 3), 1), ((1, 2, 3), 4), ((2, 1, 9), 1)])
def test_runs_of_every_length(monkeypatch, model, reps, codes):
    rng = np.random.default_rng(int(model[2] + 100 * codes))
    A, B = [], []
    for run in RUNS:
        for at in (0, 1, 20, 60):
            b = synth.random_dna(rng, 60 + run)
            a = np.concatenate([b[:at], b[at + run:]])        # one gap
            c = np.concatenate([a[:30], a[50:]])              # and another in the other one
            d = a.copy()
            d[rng.random(len(d)) < codes] |= 16
            for x, y in ((a, b), (b, a), (c, b), (d, b), (b[:at + 3], b), (b, b[-3:])):
                A.append(synth.with_gap(x))
                B.append(synth.with_gap(y))
    cm, om = align.CostMatrix.dna(*model), O.cm_dna(*model)
    batch = align.PairBatch.from_host(A * reps, B * reps)  # four times: the large batches' classes
    got = align.align_2(batch, cm, dos_empty=True).to_host()
    monkeypatch.setenv("POYD_AFF_PACKED", "0")
    want = align.align_2(batch, cm, dos_empty=True).to_host()
    for i, (x, y) in enumerate(zip(got, want)):
        assert x["cost"] == y["cost"], i
        for k in ("a", "b", "median", "median_wg"):
            assert np.array_equal(x[k], y[k]), (i, k)
    for i in range(0, len(A), 17):
        c, med, ra, rb, wg = O.dos_median(A[i], B[i], om)
        assert got[i]["cost"] == c and np.array_equal(got[i]["median"], med), i
        assert np.array_equal(got[i]["a"], ra) and np.array_equal(got[i]["b"], rb), i
