"""The block-per-pair kernel of small batches (csrc/linear_team.cu) at the edges
of its 8-double-step chunks, 8 / 16 / 32 diagonals per lane, band parities and
sequence ends: costs, aligned sequences and medians equal the warp-per-pair
kernel's (a tuned variant keeps that one) and, for a sample, the oracle's."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from poyd_gb300 import align, native, synth

pytestmark = pytest.mark.gpu


@pytest.fixture
def warp_per_pair():
    """Makes the warp-per-pair kernel the variant of every class below."""
    def on():
        for al in (0, 1):
            for lg in range(0, 11):
                for w in range(0, 16):
                    native.check(native.lib().poyd_autotune_set(torch.cuda.current_device(), al, lg, w,
                                                                1, 0, -1))
    yield on
    native.check(native.lib().poyd_autotune_clear())


def pairs(rng, n, lo, hi, ratio):
    out = []
    for _ in range(n):
        la = int(rng.integers(lo, hi + 1))
        lb = max(1, int(la * rng.uniform(1 / ratio, ratio)))
        a = synth.random_dna(rng, max(la, lb), 0.05)
        b = synth.mutate(rng, a, 0.15, 0.03)[:lb - 1]
        b = np.concatenate([b, synth.random_dna(rng, lb - 1 - len(b))])
        a = a[:la - 1].copy()
        a[rng.random(len(a)) < 0.02] |= 16  # a median's optional positions
        out.append((synth.with_gap(a), synth.with_gap(b)))
    return [p[0] for p in out], [p[1] for p in out]


# lengths and length ratios: bands of 1 to 1,023 diagonals (8, 16, 32 a lane)
SHAPES = [(1, 3, 1.0), (1, 20, 2.0), (14, 19, 1.0), (60, 130, 1.1), (120, 300, 1.6),
          (300, 420, 1.02), (900, 1100, 1.05), (1400, 1700, 1.1), (400, 480, 2.5)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sub,indel", [(1, 2), (1, 1), (3, 2)])
def test_matches_the_warp_per_pair_kernel(warp_per_pair, shape, sub, indel):
    rng = np.random.default_rng(int(shape[1] * 7 + sub))
    A, B = pairs(rng, 24, *shape)
    cm, om = align.CostMatrix.dna(sub, indel), O.cm_dna(sub, indel, -1)
    b = align.PairBatch.from_host(A, B)
    got = align.align_2(b, cm, dos_empty=True).to_host()
    costs = [align.cost_2(b, cm, d)[0].cpu().numpy() for d in (None, "dos")]
    warp_per_pair()
    want = align.align_2(b, cm, dos_empty=True).to_host()
    for c, d in zip(costs, (None, "dos")):
        assert np.array_equal(c, align.cost_2(b, cm, d)[0].cpu().numpy()), d
    for i, (x, y) in enumerate(zip(got, want)):
        assert x["cost"] == y["cost"], i
        for k in ("a", "b", "median_wg", "median"):
            assert np.array_equal(x[k], y[k]), (i, k)
        if i < 6:
            c, med, ra, rb, wg = O.dos_median(A[i], B[i], om)
            assert x["cost"] == c and np.array_equal(x["median"], med), i
            assert np.array_equal(x["a"], ra) and np.array_equal(x["b"], rb), i


def test_batches_around_the_limit(warp_per_pair):
    # the last size that takes a block per pair, the first that does not, and
    # a pair with an all-gap sequence among them
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(8)
    cm = align.CostMatrix.default()
    for n in (1, 3 * sms, 3 * sms + 1):
        A, B = pairs(rng, n, 20, 90, 1.2)
        A[0] = np.array([16, 16, 16], np.uint8)
        b = align.PairBatch.from_host(A, B)
        got = align.align_2(b, cm, dos_empty=True).to_host()
        cost = align.cost_2(b, cm, "dos")[0].cpu().numpy()
        warp_per_pair()
        want = align.align_2(b, cm, dos_empty=True).to_host()
        assert np.array_equal(cost, align.cost_2(b, cm, "dos")[0].cpu().numpy())
        native.check(native.lib().poyd_autotune_clear())
        for x, y in zip(got, want):
            assert x["cost"] == y["cost"]
            for k in ("a", "b", "median_wg", "median"):
                assert np.array_equal(x[k], y[k])
