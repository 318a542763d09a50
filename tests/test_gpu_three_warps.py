"""Warps per triple of the zero-opening three-sequence kernel (csrc/three.cu): a
large batch whose one long triple asks for eight warps, with short ones that leave
most of them idle, against the 32-bit kernel."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, synth, three

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [130, 300])  # four and eight warps
def test_one_long_triple_among_short_ones(monkeypatch, longest):
    rng = np.random.default_rng(longest)
    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 5
    items = []
    for i in range(n):
        base = synth.random_dna(rng, longest - 1 if i == 3 else int(rng.integers(1, 12)))
        a, b, c = (synth.mutate(rng, base, 0.1, 0.03) for _ in range(3))
        items.append((synth.with_gap(a), synth.with_gap(b), synth.with_gap(c)))
    cm = align.CostMatrix.dna(1, 2)
    b = three.TripleBatch.from_host(items)
    got = three.align_3_powell(b, 1, 0, 2, cm).to_host()
    monkeypatch.setenv("POYD_P3_PACKED", "0")
    for i, (x, y) in enumerate(zip(got, three.align_3_powell(b, 1, 0, 2, cm).to_host())):
        assert x["cost"] == y["cost"], i
        for k in ("a", "b", "c", "median"):
            assert np.array_equal(x[k], y[k]), (i, k)
