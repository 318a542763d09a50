"""The first alignment of a small batch on a new stream allocates its direction
matrix once: a buffer that is allocated and then grown frees its first memory, which
waits for whatever the device's other streams are doing.  A batch whose matrix for a
block per pair is over the budget takes the warp-per-pair kernel, with the same
results."""
import pytest
import torch

from poyd_gb300 import align, synth

pytestmark = pytest.mark.gpu


def batch(n, length, longest):
    """n pairs of about one length and a longer one: a matrix for a block per pair
    has n + 1 times the longest pair's words."""
    A, B = synth.pair_batch(n, n, lmin=length, lmax=length + 20)
    A2, B2 = synth.pair_batch(n + 1, 1, lmin=longest, lmax=longest + 20)
    return align.PairBatch.from_host(A + A2, B + B2)


def results(b, stream=None):
    r = align.align_2(b, align.CostMatrix.default(), stream=stream)
    torch.cuda.synchronize()
    return [r.cost, r.out_len, r.pack().packed]


@pytest.mark.parametrize("n,length,longest", [(1, 60, 1000), (20, 40, 2000), (100, 300, 300)])
def test_first_call_does_not_wait_for_other_streams(n, length, longest):
    b, cm = batch(n, length, longest), align.CostMatrix.default()
    want = results(b)
    layout = b.out_layout()
    busy, own = torch.cuda.Stream(), torch.cuda.Stream()
    done = torch.cuda.Event()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(1_000_000_000)  # about half a second
        done.record()
    r = align.align_2(b, cm, stream=own, layout=layout)
    own.synchronize()
    assert not done.query()
    torch.cuda.synchronize()
    for x, y in zip([r.cost, r.out_len, r.pack().packed], want):
        assert torch.equal(x, y)


def test_matrix_over_the_budget(monkeypatch):
    b = batch(20, 40, 2000)
    want = results(b)
    monkeypatch.setenv("POYD_DM_BUDGET_BYTES", str(1 << 20))
    for x, y in zip(results(b, torch.cuda.Stream()), want):
        assert torch.equal(x, y)
