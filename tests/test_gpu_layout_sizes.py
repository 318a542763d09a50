"""Result layouts on both sides of the size from which tensor operations make them."""
import pytest
import torch

from poyd_gb300 import align

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65535, 65536, 65537, 300001])
def test_slots_and_packed_places(n):
    g = torch.Generator().manual_seed(n)
    lens = [torch.randint(1, 40, (n,), generator=g, dtype=torch.int32) for _ in range(2)]
    want = align.slot_layout(lens, 2)
    got = align.slot_layout([t.cuda() for t in lens], 2)
    assert torch.equal(got[0].cpu(), want[0]) and got[1] == want[1] and torch.equal(got[2].cpu(), want[2])
    r = align.AlignResult(torch.zeros(n, dtype=torch.int32, device="cuda"),
                          torch.arange(want[1], device="cuda").to(torch.uint8), got[0],
                          torch.stack(lens, 1).flatten().cuda(), got[2], None)
    # sequence k of pair i: bytes numbered from off + (k + 1) cap - length on
    sizes = torch.stack([lens[0]] * 3 + [lens[1]], 1).flatten().long()
    ends = (want[0][:, None] + want[2][:, None] * torch.arange(1, 5)).flatten()
    src = torch.repeat_interleave(ends - sizes.cumsum(0), sizes) + torch.arange(int(sizes.sum()))
    assert torch.equal(r.pack().packed.cpu(), src.to(torch.uint8))
