"""Explicit band widths (``cost_2 ~deltaw``) so negative that the band holds
neither the first nor the final cell.  The reference reads cells that it never
filled there, so no cost is right, but the call stays defined: it is the
warp-per-pair kernel's (a tuned variant keeps that one), whatever the batch's
size.  k_lin_team places its tables by the final cell's diagonal, which lies
outside them for such a band."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, native, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", ["a block per pair", "by antidiagonals"])
@pytest.mark.parametrize("deltaw", [-60, -100000])
def test_band_that_holds_no_path(size, deltaw):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 5 if size == "a block per pair" else 8 * sms + 1
    rng = np.random.default_rng(5)
    A = [synth.with_gap(synth.random_dna(rng, 399)) for _ in range(n)]
    B = [synth.with_gap(synth.random_dna(rng, 299)) for _ in range(n)]
    batch = align.PairBatch.from_host(A, B)
    cm = align.CostMatrix.default()
    # one pair alone: the others' costs are what they are without it
    dw = torch.zeros(n, dtype=torch.int32, device="cuda")
    dw[n // 2] = deltaw
    got = align.cost_2(batch, cm, deltaw=dw)[0]
    usual = align.cost_2(batch, cm, deltaw=torch.zeros_like(dw))[0]
    for w in range(16):
        native.check(native.lib().poyd_autotune_set(torch.cuda.current_device(), 0,
                                                    n.bit_length() - 1, w, 1, 0, -1))
    try:
        want = align.cost_2(batch, cm, deltaw=dw)[0]
    finally:
        native.check(native.lib().poyd_autotune_clear())
    assert torch.equal(got, want)
    others = torch.arange(n, device="cuda") != n // 2
    assert torch.equal(got[others], usual[others])
