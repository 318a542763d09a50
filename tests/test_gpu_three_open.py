"""The 16-bit three-sequence kernel with gap openings (csrc/three_open.cu) at
the edges of its row pairs, 32-lane strips, 8-step chunks and panels: costs,
aligned rows, medians and flags equal the 32-bit kernel's byte for byte (one
block or a cluster per triple), and the oracle's where the cube is small."""
import itertools

import numpy as np
import pytest

from oracle import oracle as O
from poyd_gb300 import align, three
from tests.test_gpu_three_linear import same, triple

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (1, 1, 2), (1, 2, 70), (3, 4, 5), (4, 8, 9), (5, 32, 33), (17, 64, 65),
         (8, 40, 41), (24, 31, 7), (33, 33, 33), (16, 97, 130)]


# the last two cut values off at infinity before a column cost is added
@pytest.mark.parametrize("mm,go,ge", [(1, 3, 2), (2, 1, 1), (1, 300, 100), (120, 40, 300)])
def test_small_cubes_match_oracle_and_the_32_bit_kernel(monkeypatch, mm, go, ge):
    rng = np.random.default_rng(mm)
    T = [triple(rng, p) for s in SIZES for p in sorted(set(itertools.permutations(s)))]
    b = three.TripleBatch.from_host(T)
    cm = align.CostMatrix.dna(1, 2)
    got = three.align_3_powell(b, mm, go, ge, cm).to_host()
    monkeypatch.setenv("POYD_P3_PACKED", "0")
    want = three.align_3_powell(b, mm, go, ge, cm).to_host()
    for i, (x, y) in enumerate(zip(got, want)):
        same(x, y, i)
        if np.prod([len(s) for s in T[i]]) < 100_000:
            c, *rows = O.powell_3d(*T[i], mm, go, ge)
            assert c == x["cost"], i
            for r, k in zip(rows, "abc"):
                assert np.array_equal(r, x[k]), (i, k)


@pytest.mark.parametrize("n,lens", [(1, (120, 200)), (20, (60, 90)), (300, (2, 60)),
                                    (3, (270, 300))])
@pytest.mark.parametrize("cluster", ["1", "0"])
def test_batches_of_every_block_shape(monkeypatch, n, lens, cluster):
    # clusters of 1 to 8 blocks; the last runs a long b in panels of 8 strips
    rng = np.random.default_rng(n)
    T = [triple(rng, rng.integers(*lens, 3).tolist()) for _ in range(n)]
    items = [(a, b, a.copy() if i % 3 else b.copy(), p) for i, (a, b, p) in enumerate(T)]
    cm = align.CostMatrix.dna(1, 2, 3)
    b = three.TripleBatch.from_host(items)
    monkeypatch.setenv("POYD_P3_CLUSTER", cluster)
    got = three.readjust_3d(b, cm).to_host()
    monkeypatch.setenv("POYD_P3_PACKED", "0")
    want = three.readjust_3d(b, cm).to_host()
    for i, (x, y) in enumerate(zip(got, want)):
        same(x, y, i)
        assert x["changed"] == y["changed"], i
