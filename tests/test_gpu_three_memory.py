"""A triple whose choices the 16-bit kernel with openings (csrc/three_open.cu) has no
memory for, since its strips of 32 are mostly padding beside a short sequence, while
the 32-bit kernel's cube fits: it is aligned all the same."""
import numpy as np
import pytest
import torch

from poyd_gb300 import native, synth, three

pytestmark = pytest.mark.gpu


def test_short_sequence_beside_long_ones_in_little_memory(monkeypatch):
    # 0.6 GB of strips; a cube of 0.04
    rng = np.random.default_rng(1)
    T = [synth.with_gap(synth.random_dna(rng, n)) for n in (1500, 1, 1500)]
    b = three.TripleBatch.from_host([tuple(T)])
    res = lambda: three.align_3_powell(b, 1, 3, 2).to_host()[0]
    monkeypatch.setenv("POYD_P3_PACKED", "0")
    want = res()
    monkeypatch.delenv("POYD_P3_PACKED")
    native.check(native.lib().poyd_workspace_release())
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (320 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = res()
    finally:
        del held
        torch.cuda.empty_cache()
    again = res()  # in memory enough
    for x in (got, again):
        assert x["cost"] == want["cost"]
        for k in "abc":
            assert np.array_equal(x[k], want[k]), k
