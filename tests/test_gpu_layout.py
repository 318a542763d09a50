"""Result layouts on the device (csrc/layout.cu) at the edges of the running
sum's rounds, against the same layouts from tensor operations on the CPU."""
import pytest
import torch

from poyd_gb300 import align, native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7, 8, 257, 8191, 8192, 8193, 70001])
def test_slot_and_pack_layouts(n):
    g = torch.Generator().manual_seed(n)
    lens = [torch.randint(1, 6000, (n,), generator=g, dtype=torch.int32) for _ in range(3)]
    for k, extra in ((2, 2), (3, 0)):
        want = align.slot_layout(lens[:k], extra)
        got = align.slot_layout([t.cuda() for t in lens[:k]], extra)
        # lengths that a kernel cannot read as they are
        odd = align.slot_layout([t.cuda().repeat_interleave(2)[::2] for t in lens[:k]], extra)
        for r in (got, odd):
            assert torch.equal(r[0].cpu(), want[0]) and r[1] == want[1] and torch.equal(r[2].cpu(), want[2])
    out_len = torch.randint(0, 100, (n, 2), generator=g, dtype=torch.int32)
    off, cap = torch.arange(n) * 416, torch.full((n,), 104)
    out = torch.randint(0, 255, (416 * n,), generator=g, dtype=torch.uint8)
    p = align.AlignResult(torch.zeros(n, dtype=torch.int32, device="cuda"), out.cuda(), off.cuda(),
                          out_len.flatten().cuda(), cap.cuda(), None).pack()
    parts = []
    for i in list(range(min(n, 40))) + [n - 1]:
        a, m = out_len[i].tolist()
        s = out[416 * i:416 * (i + 1)]
        parts.append(torch.cat([s[104 - a:104], s[208 - a:208], s[312 - a:312], s[416 - m:]]))
    first = torch.cat(parts[:-1])
    assert p.packed.numel() == int(3 * out_len[:, 0].sum() + out_len[:, 1].sum())
    assert torch.equal(p.packed[:first.numel()].cpu(), first)
    if parts[-1].numel():
        assert torch.equal(p.packed[-parts[-1].numel():].cpu(), parts[-1])


def test_a_failed_traceback_is_an_error():
    n = 9000
    out_len = torch.ones(2 * n, dtype=torch.int32, device="cuda")
    out_len[8500] = -1
    z = torch.zeros(n, dtype=torch.int64, device="cuda")
    r = align.AlignResult(torch.zeros(n, dtype=torch.int32, device="cuda"),
                          torch.zeros(64, dtype=torch.uint8, device="cuda"), z, out_len, z + 4, None)
    with pytest.raises(native.PoydError, match="4250"):
        r.pack()
