"""Small affine batches with directions take 16 lanes a pair (8 diagonals each
where the band allows), larger ones 8 (csrc/affine_diag.cuh): both sides of the
line against the 32-bit rows kernel, at band widths around each class's end."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gaps", [0.0, 0.04])
@pytest.mark.parametrize("times", [1, 30])
def test_both_spreads_match_the_rows_kernel(monkeypatch, times, gaps):
    rng = np.random.default_rng(times)
    A, B = [], []
    for dif in (0, 5, 46, 47, 78, 79, 80, 110, 143, 144, 207, 208):  # e0 = dif + 8
        for n in (2, 61, 300):
            a = synth.random_dna(rng, n, 0.05)
            b = np.concatenate([synth.mutate(rng, a, 0.15, 0.03), synth.random_dna(rng, 400)])[:n + dif]
            for s in (a, b):
                s[rng.random(len(s)) < gaps] |= 16
            A.append(synth.with_gap(a))
            B.append(synth.with_gap(b))
    A.append(np.array([16, 16], np.uint8))
    B.append(synth.with_gap(synth.random_dna(rng, 30)))
    n = len(A)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert n <= 8 * sms < 30 * n + 8 * sms
    reps = 1 if times == 1 else 8 * sms // n + 1  # the first size past the line, or well before it
    cm = align.CostMatrix.dna(1, 2, 3)
    one = align.PairBatch.from_host(A, B)
    many = align.PairBatch(one.seq, *(t.repeat(reps) for t in (one.a_off, one.a_len, one.b_off, one.b_len)))
    got = align.align_2(many, cm, dos_empty=True)
    packed = got.pack().packed
    monkeypatch.setenv("POYD_AFF_PACKED", "0")
    want = align.align_2(one, cm, dos_empty=True)
    assert torch.equal(got.cost, want.cost.repeat(reps))
    assert torch.equal(got.out_len, want.out_len.repeat(reps))
    assert torch.equal(packed, want.pack().packed.repeat(reps))
