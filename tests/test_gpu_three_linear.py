"""The zero-opening three-sequence kernel (csrc/three_linear.cu) at the edges
of its 4 x 4 tiles, 32-tile strips, 8-step chunks and axis orders: costs,
aligned rows, medians and flags equal the 32-bit 16-state kernel's byte for
byte, and the oracle's where the cube is small."""
import itertools

import numpy as np
import pytest

from oracle import oracle as O
from poyd_gb300 import align, synth, three

pytestmark = pytest.mark.gpu


def triple(rng, lens):
    """Three relatives of the given lengths (leading gap included)."""
    base = synth.random_dna(rng, max(lens) + 8)
    out = []
    for n in lens:
        s = synth.mutate(rng, base, 0.1, 0.03)[:n - 1]
        out.append(synth.with_gap(np.concatenate([s, synth.random_dna(rng, n - 1 - len(s))])))
    return tuple(out)


SIZES = [(1, 1, 1), (1, 1, 2), (1, 2, 70), (3, 4, 5), (4, 8, 9), (5, 64, 65), (17, 68, 69),
         (8, 40, 41), (24, 31, 7), (33, 33, 33), (16, 97, 130), (64, 66, 68)]


def same(x, y, i):
    assert x["cost"] == y["cost"], i
    for k in ("a", "b", "c", "median"):
        assert np.array_equal(x[k], y[k]), (i, k)


@pytest.mark.parametrize("mm,ge", [(1, 2), (3, 1)])
def test_small_cubes_match_oracle_and_the_32_bit_kernel(monkeypatch, mm, ge):
    rng = np.random.default_rng(mm)
    T = [triple(rng, p) for s in SIZES for p in sorted(set(itertools.permutations(s)))]
    b = three.TripleBatch.from_host(T)
    cm = align.CostMatrix.dna(mm, ge)
    got = three.align_3_powell(b, mm, 0, ge, cm).to_host()
    monkeypatch.setenv("POYD_P3_PACKED", "0")
    want = three.align_3_powell(b, mm, 0, ge, cm).to_host()
    for i, (x, y) in enumerate(zip(got, want)):
        same(x, y, i)
        if np.prod([len(s) for s in T[i]]) < 100_000:
            c, *rows = O.powell_3d(*T[i], mm, 0, ge)
            assert c == x["cost"], i
            for r, k in zip(rows, "abc"):
                assert np.array_equal(r, x[k]), (i, k)


@pytest.mark.parametrize("n", [1, 7, 400])
def test_batches_of_every_block_shape(monkeypatch, n):
    # one triple (many warps a block) to a batch that fills the SMs
    rng = np.random.default_rng(n)
    lo, hi = (200, 330) if n < 10 else (2, 120)
    T = [triple(rng, rng.integers(lo, hi, 3).tolist()) for _ in range(n)]
    items = [(a, b, a.copy() if i % 3 else b.copy(), p) for i, (a, b, p) in enumerate(T)]
    cm = align.CostMatrix.dna(1, 2)
    b = three.TripleBatch.from_host(items)
    got = three.readjust_3d(b, cm).to_host()
    monkeypatch.setenv("POYD_P3_PACKED", "0")
    want = three.readjust_3d(b, cm).to_host()
    for i, (x, y) in enumerate(zip(got, want)):
        same(x, y, i)
        assert x["changed"] == y["changed"], i
