"""The antidiagonal affine kernel (csrc/affine_diag.cu) and its walk against the
32-bit rows kernel (POYD_AFF_PACKED=0) over every class it takes: 8, 16 and 32
lanes of 12 and 16 diagonals and wider bands that stay in rows, with and without
gap-bearing codes, cost and align, ends of the band (rows and columns shorter
than it), ragged tasks, all-gap and length-1 sequences; a sample against the
oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from poyd_gb300 import align, synth

pytestmark = pytest.mark.gpu


def pairs(seed, gaps):
    rng = np.random.default_rng(seed)
    A, B = [], []

    def add(la, lb, related=True):
        a = synth.random_dna(rng, la, 0.05)
        b = synth.mutate(rng, a, 0.15, 0.03) if related else synth.random_dna(rng, lb, 0.05)
        b = np.concatenate([b, synth.random_dna(rng, max(0, lb - len(b)), 0.05)])[:lb]
        if gaps:
            for s in (a, b):
                s[rng.random(len(s)) < 0.04] |= 16
                if len(s) > 30 and rng.random() < 0.3:
                    s[10:10 + int(rng.integers(1, 12))] = 16
        A.append(synth.with_gap(a))
        B.append(synth.with_gap(b))

    for la, lb in [(0, 0), (0, 1), (1, 0), (0, 9), (9, 0), (1, 1), (39, 41), (41, 39), (40, 40),
                   (45, 200), (200, 45), (64, 1), (3, 80), (120, 121)]:
        add(la, lb)
    for _ in range(30):
        n = int(rng.integers(30, 900))
        add(n, n + int(rng.integers(-20, 20)))
    for dif in (31, 33, 47, 48, 79, 80, 143, 144, 207, 208, 335, 336, 463, 464):  # e0 = dif + 8
        n = int(rng.integers(100, 700))
        add(n, n + dif)
        add(n + dif, n, related=False)
    A.append(np.array([16, 16, 16], np.uint8))
    B.append(synth.with_gap(synth.random_dna(rng, 30)))
    A.append(synth.with_gap(synth.random_dna(rng, 30)))
    B.append(np.array([16], np.uint8))
    return A, B


@pytest.mark.parametrize("gaps", [False, True])
@pytest.mark.parametrize("model", [(1, 2, 3), (2, 1, 1), (3, 1, 5), (1, 1, 0), (1, 2, 60)])
def test_classes_match_the_rows_kernel_and_the_oracle(monkeypatch, model, gaps):
    A, B = pairs(3 + model[2], gaps)
    cm, om = align.CostMatrix.dna(*model), O.cm_dna(*model)
    b = align.PairBatch.from_host(A, B)
    for empty in (True, False):
        monkeypatch.delenv("POYD_AFF_PACKED", raising=False)
        got = align.align_2(b, cm, dos_empty=empty).to_host()
        cost, cells = align.cost_2(b, cm, band_cells=True)
        monkeypatch.setenv("POYD_AFF_PACKED", "0")
        want = align.align_2(b, cm, dos_empty=empty).to_host()
        assert torch.equal(cost, align.cost_2(b, cm)[0])
        for i, (x, y) in enumerate(zip(got, want)):
            assert x["cost"] == y["cost"], i
            for k in ("a", "b", "median_wg", "median"):
                assert np.array_equal(x[k], y[k]), (i, k)
    for i in range(0, len(A), 7):
        assert cost[i] == O.cost_affine_3(A[i], B[i], om), i
        assert cells[i] == O.band_cells_affine(len(A[i]), len(B[i])), i
        c, med, mwg, ri, rj = O.align_affine_3(A[i], B[i], om)
        assert c == got[i]["cost"] and np.array_equal(med, got[i]["median"]), i
        assert np.array_equal(ri, got[i]["a"]) and np.array_equal(rj, got[i]["b"]), i


def test_values_past_16_bits_stay_in_rows(monkeypatch):
    # unrelated long pairs under large costs next to short ones: some tasks'
    # values fit, the others run in rows, in one call
    rng = np.random.default_rng(2)
    A = [synth.with_gap(synth.random_dna(rng, n)) for n in (60, 3000, 200, 5000, 40)]
    B = [synth.with_gap(synth.random_dna(rng, n)) for n in (70, 2990, 210, 4980, 40)]
    cm = align.CostMatrix.dna(9, 6, 20)
    b = align.PairBatch.from_host(A, B)
    got = align.align_2(b, cm).to_host()
    cost = align.cost_2(b, cm)[0]
    monkeypatch.setenv("POYD_AFF_PACKED", "0")
    want = align.align_2(b, cm).to_host()
    assert torch.equal(cost, align.cost_2(b, cm)[0])
    for x, y in zip(got, want):
        assert x["cost"] == y["cost"]
        for k in ("a", "b", "median_wg", "median"):
            assert np.array_equal(x[k], y[k])
