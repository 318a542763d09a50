"""A call's stream may be any object with a ``cuda_stream`` handle, as before its
result layouts were ordered after it."""
import pytest
import torch

from poyd_gb300 import align, synth, three

pytestmark = pytest.mark.gpu


class Handle:
    def __init__(self, stream):
        self.cuda_stream = stream.cuda_stream


@pytest.mark.parametrize("own", [True, False])  # a stream of its own, the current one
def test_calls_take_a_bare_handle(own):
    s = torch.cuda.Stream() if own else torch.cuda.current_stream()
    h = Handle(s)
    A, B = synth.pair_batch(1, 30, lmin=20, lmax=60)
    b, cm = align.PairBatch.from_host(A, B), align.CostMatrix.default()
    want = align.align_2(b, cm)
    got = align.align_2(b, cm, stream=h)
    packed = got.pack(stream=h)
    got.cap = got.cap.to(torch.int32)  # sized by tensor operations
    again = got.pack(stream=h)
    s.synchronize()
    assert torch.equal(got.cost, want.cost)
    assert torch.equal(packed.packed, want.pack().packed) and torch.equal(again.packed, packed.packed)
    T = synth.triple_batch(5, 4, lmin=20, lmax=60)
    tb = three.TripleBatch.from_host([(x, y, x.copy(), p) for x, y, p in T])
    r = three.readjust_3d(tb, align.CostMatrix.dna(1, 2), stream=h)
    s.synchronize()
    assert torch.equal(r.cost, three.readjust_3d(tb, align.CostMatrix.dna(1, 2)).cost)
