"""k_lin_diag's alignments (csrc/linear_diag.cu) by their lanes: 16 at least and, for
bands that 16 lanes do not hold, 32 just past the size from which the kernel takes
alignments, 8 in larger batches.  That it took them shows in the walk's own launch,
which the warp-per-pair kernel has none of; results equal that kernel's."""
import numpy as np
import pytest
import torch

from poyd_gb300 import align, native, synth

pytestmark = pytest.mark.gpu


def walks(f):
    """f()'s value and the launches of the antidiagonal kernel's walk."""
    lib = native.lib()
    native.profile_read(clear=True)
    lib.poyd_profile_enable(1)
    try:
        r = f()
        torch.cuda.synchronize()
        return r, native.profile_read("lin_traceback", clear=True)[1]
    finally:
        lib.poyd_profile_enable(0)


@pytest.mark.parametrize("per_sm", [12.5, 25.0])
@pytest.mark.parametrize("lengths", [(30, 200), (900, 1100), (4300, 4400)])  # bands to 130, 250, 560
def test_alignments_past_the_threshold(per_sm, lengths):
    n = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count)
    A, B = synth.pair_batch(int(per_sm) + lengths[0], 40, lmin=lengths[0], lmax=lengths[1])
    one = align.PairBatch.from_host(A, B)
    pick = torch.from_numpy(np.random.default_rng(n).permutation(np.arange(n) % 40)).cuda()
    batch = align.PairBatch(one.seq, *[t[pick] for t in (one.a_off, one.a_len, one.b_off, one.b_len)])
    cm = align.CostMatrix.dna(1, 1)
    got, launches = walks(lambda: align.align_2(batch, cm))
    assert launches == 1
    small, none = walks(lambda: align.align_2(one, cm))
    assert none == 0
    assert torch.equal(got.cost, small.cost[pick])
    assert torch.equal(got.out_len.view(-1, 2), small.out_len.view(-1, 2)[pick])
    w, g = small.to_host(), got.to_host()
    for i, p in enumerate(pick.tolist()):
        for k in ("a", "b", "median", "median_wg"):
            assert np.array_equal(g[i][k], w[p][k]), (i, k)
