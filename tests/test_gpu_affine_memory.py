"""Affine alignments of short sequences with much longer ones, in memory that holds
the rows kernels' direction matrix but not the antidiagonal kernel's, fourteen times
as large: they are not refused, and their results are those of ample memory."""
import pytest
import torch

from poyd_gb300 import align, native, synth

pytestmark = pytest.mark.gpu


def test_uneven_pairs_in_little_memory():
    A, _ = synth.pair_batch(1, 4000, lmin=8, lmax=10)
    _, B = synth.pair_batch(2, 4000, lmin=430, lmax=440)
    b = align.PairBatch.from_host(A, B)
    cm = align.CostMatrix.dna(1, 2, 3)

    def res():
        r = align.align_2(b, cm, dos_empty=True)
        return [r.cost, r.out_len, r.pack().packed]

    want = res()  # 460 MB of direction words
    native.check(native.lib().poyd_workspace_release())
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (320 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = res()
    finally:
        del held
        torch.cuda.empty_cache()
    for x, y in zip(got, want):
        assert torch.equal(x, y)
