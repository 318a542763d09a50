"""A call that is given a stream sizes its results by what that stream has made of
the lengths, though the layout itself runs on the current stream.  The lengths
hold larger values at first (a layout that came too early would be too large, not
too small) and get their own behind a wait on the stream."""
import pytest
import torch

from poyd_gb300 import align, synth, three

pytestmark = pytest.mark.gpu
CYCLES = 200_000_000  # about 0.1 s


def later(stream, pairs):
    """The first tensor of each pair becomes the second on `stream`, after a while."""
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(CYCLES)
        for t, v in pairs:
            t.copy_(v)


@pytest.mark.parametrize("native", [True, False])  # the layout's kernel, tensor operations
def test_pack_follows_its_stream(native):
    A, B = synth.pair_batch(3, 40, lmin=20, lmax=200)
    r = align.align_2(align.PairBatch.from_host(A, B), align.CostMatrix.default())
    want = r.pack().packed
    if not native:
        r.cap = r.cap.to(torch.int32)
    assert torch.equal(r.pack().packed, want)  # loads the kernels, which waits for the device
    true_len = r.out_len.clone()
    r.out_len.add_(5)
    s = torch.cuda.Stream()
    later(s, [(r.out_len, true_len)])
    got = r.pack(stream=s).packed
    s.synchronize()
    assert torch.equal(got, want)


def test_alignment_slots_follow_their_stream():
    cm = align.CostMatrix.default()
    A, B = synth.pair_batch(4, 40, lmin=20, lmax=200)
    b = align.PairBatch.from_host(A, B)
    lens = [(t, t.clone()) for t in (b.a_len, b.b_len)]
    s = torch.cuda.Stream()
    for call in (align.align_2, align.closest):
        want = call(b, cm)
        for t, _ in lens:
            t.add_(8)
        later(s, lens)
        got = call(b, cm, stream=s)
        s.synchronize()
        assert torch.equal(got.cap, want.cap) and torch.equal(got.out_off, want.out_off)
        assert torch.equal(got.out_len, want.out_len)


def test_triple_slots_follow_their_stream():
    T = synth.triple_batch(5, 4, lmin=20, lmax=60)
    b = three.TripleBatch.from_host([(x, y, x.copy(), p) for x, y, p in T])
    cm = align.CostMatrix.dna(1, 2)
    lens = [(t, t.clone()) for t in b.lens]
    s = torch.cuda.Stream()
    want = three.readjust_3d(b, cm)
    for t, _ in lens:
        t.add_(8)
    later(s, lens)
    got = three.readjust_3d(b, cm, stream=s)
    s.synchronize()
    assert torch.equal(got.cap, want.cap) and torch.equal(got.cost, want.cost)
