"""Calls of several host threads, each with a stream of its own, while torch's
current stream stays the default one: the layouts of their results, which run on
the current stream, do not see each other's totals, and a batch of short triples
does not take from a batch of long ones the shared memory that it asked for."""
import threading

import numpy as np
import pytest
import torch

from poyd_gb300 import align, synth, three

pytestmark = pytest.mark.gpu


def run_threads(work):
    """work(k) in a thread each; the first exception is raised here."""
    errors = []

    def call(f):
        try:
            torch.cuda.set_device(0)
            f()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=call, args=(f,)) for f in work]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]


def test_slot_layouts_overlap():
    lens = [torch.full((n,), 100 + n, dtype=torch.int32, device="cuda") for n in (3, 40, 500, 6000)]

    def worker(x):
        n, cap = x.numel(), (2 * (100 + x.numel()) + 2 + 3) // 4 * 4
        def f():
            for _ in range(400):
                assert align.slot_layout((x, x), 2)[1] == 4 * cap * n
        return f

    run_threads([worker(x) for x in lens])


def test_alignments_and_packs_overlap():
    cm = align.CostMatrix.default()
    sets = [synth.pair_batch(n, n, lmin=20, lmax=40 + n) for n in (2, 11, 60, 300)]
    batches = [align.PairBatch.from_host(*s) for s in sets]
    want = [align.align_2(b, cm).pack().packed.clone() for b in batches]
    torch.cuda.synchronize()

    def worker(b, w):
        s = torch.cuda.Stream()
        def f():
            for _ in range(60):
                r = align.align_2(b, cm, stream=s)
                s.synchronize()
                assert torch.equal(r.pack().packed, w)
        return f

    run_threads([worker(b, w) for b, w in zip(batches, want)])


# with openings a block a triple; without, sixteen warps for both shapes
@pytest.mark.parametrize("go,shapes", [(3, ((2, 1, 2), (300, 1, 300))),
                                       (0, ((4, 600, 900), (4, 600, 1200)))])
def test_triples_of_different_lengths_overlap(monkeypatch, go, shapes):
    monkeypatch.setenv("POYD_P3_CLUSTER", "0")
    rng = np.random.default_rng(go)

    def worker(lens):
        T = [synth.with_gap(synth.random_dna(rng, n)) for n in lens]
        b = three.TripleBatch.from_host([tuple(T)])
        want = three.align_3_powell(b, 1, go, 2).cost.item()
        s = torch.cuda.Stream()
        def f():
            for _ in range(1500):
                r = three.align_3_powell(b, 1, go, 2, stream=s)
                s.synchronize()
            assert r.cost.item() == want
        return f

    run_threads([worker(n) for n in shapes for _ in range(2)])
