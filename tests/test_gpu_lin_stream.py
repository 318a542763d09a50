"""poyd_align_2_host on batches that k_lin_diag runs, in one, two and four parts (by
the bytes of the results) and with a pair that sends the batch to the streamed
warp-per-pair kernel: every pair's results equal the device-resident batch's."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi,wide", [(20, 60, False), (800, 1200, False), (5000, 5700, False),
                                        (800, 1200, True)])
def test_streamed_parts_match_the_device_batch(lo, hi, wide):
    rng = np.random.default_rng(hi)
    n = 14 * torch.cuda.get_device_properties(0).multi_processor_count + 7
    A, B = [], []
    for i in range(n):
        a = synth.random_dna(rng, int(rng.integers(lo, hi)), 0.05)
        A.append(synth.with_gap(a))
        B.append(synth.with_gap(synth.mutate(rng, a, 0.1, 0.02)))
    if wide:
        A[7] = synth.with_gap(synth.random_dna(rng, 1200))
        B[7] = A[7][:601].copy()
    A[5] = np.array([16, 16], np.uint8)
    cm = align.CostMatrix.dna(1, 2)
    parts = align.PairBatch.pack_host(A, B, pin=True)
    dev = align.align_2(align.PairBatch.from_host(A, B), cm, dos_empty=True).to_host()
    host = align.align_2_host(parts, cm, dos_empty=True)
    for i, (d, h) in enumerate(zip(dev, host.to_host())):
        assert d["cost"] == h["cost"], i
        for k in ("a", "b", "median_wg", "median"):
            assert np.array_equal(d[k], h[k]), (i, k)
