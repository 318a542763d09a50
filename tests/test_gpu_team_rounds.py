"""Two to three pairs an SM, where k_lin_team (csrc/linear_team.cu) takes the batch by how
much of its 512 or 1,024 diagonals the widest band fills: costs and alignments on both
sides of those bands equal the warp-per-pair kernel's (a tuned variant keeps that one)."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [2200, 3700, 4700, 6200])  # bands of about 320, 470, 570 and 720
@pytest.mark.parametrize("per_sm", [2.1, 3.0])
def test_bands_around_the_limits(length, per_sm):
    n = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count)
    rng = np.random.default_rng(length)
    A, B = [], []
    for _ in range(6):
        a = synth.random_dna(rng, length)
        b = a.copy()
        b[rng.random(length) < 0.2] = 1
        A.append(synth.with_gap(a[:length - int(rng.integers(0, 30))]))
        B.append(synth.with_gap(b[:length - int(rng.integers(0, 30))]))
    one = align.PairBatch.from_host(A, B)
    pick = torch.arange(n, device="cuda") % 6
    batch = align.PairBatch(one.seq, *[t[pick] for t in (one.a_off, one.a_len, one.b_off, one.b_len)])
    cm = align.CostMatrix.dna(1, 1)

    def all_results():
        r = align.align_2(batch, cm)
        return [align.cost_2(batch, cm)[0], r.cost, r.out_len, r.pack().packed]

    got = all_results()
    for al in (0, 1):
        for w in range(16):
            native.check(native.lib().poyd_autotune_set(torch.cuda.current_device(), al,
                                                        n.bit_length() - 1, w, 1, 0, -1))
    try:
        want = all_results()
    finally:
        native.check(native.lib().poyd_autotune_clear())
    for x, y in zip(got, want):
        assert torch.equal(x, y)
