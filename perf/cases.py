"""The measured work of this framework: what a search over DO sequences,
non-additive and Sankoff characters has it do, through the entry points a
program calls.

Sizes are those of the repository's own workloads (the 20-taxon Wagner build,
the 200-taxon SPR pass, the 65,536-pair alignment batch, the 1,216-triple
readjustment, the join proposal's training and inference) and smaller and odd
ones between them.  Inputs are seeded and synthetic, made on the device.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from poyd_gb300 import align, learned, mlp, native, search, simulate, three

DIMS = mlp.DIMS


def listed():
    return [
        # The last step of a 20-taxon Wagner build: the distance of the new
        # taxon to every node of the tree.  The smallest cost call.
        {"name": "wagner_costs", "kind": "cost", "pairs": 39, "seqs": 40, "length": 300,
         "gap_open": -1},
        # Every candidate join of a 200-taxon SPR pass (DOS.distance).
        {"name": "spr_costs", "kind": "cost", "pairs": 154296, "seqs": 398, "length": 1500,
         "gap_open": -1},
        # The same for a 100-taxon pass under an affine model.
        {"name": "affine_costs", "kind": "cost", "pairs": 38001, "seqs": 198, "length": 1000,
         "gap_open": 3},
        # One DOS.median of two ~1,000 bp sequences: the smallest alignment.
        {"name": "align_one", "kind": "align", "pairs": 1, "lmin": 1000, "lmax": 1000,
         "gap_open": -1},
        # The 65,536-pair alignment batch, 100 to 5,000 bp, results packed.
        {"name": "align_batch", "kind": "align", "pairs": 65536, "lmin": 100, "lmax": 5000,
         "gap_open": -1},
        # A quarter of it under an affine model.
        {"name": "align_affine", "kind": "align", "pairs": 16384, "lmin": 100, "lmax": 5000,
         "gap_open": 3},
        # The non-DO characters of the 200-taxon pass: the Fitch and Sankoff
        # distances of its joins and the medians of a TBR round's re-rootings.
        {"name": "chars", "kind": "chars", "nodes": 400, "pairs": 154296, "medians": 4256,
         "fitch": 2000, "sank": 200},
        # The downpass of a whole 200-taxon tree with all three character
        # types: a list of dependent levels of medians.
        {"name": "downpass", "kind": "downpass", "taxa": 200, "length": 1500, "fitch": 2000,
         "sank": 200},
        # One level of an Iterative (ThreeD) adjustment under an affine model.
        {"name": "readjust_level", "kind": "readjust", "triples": 20, "lmin": 150, "lmax": 200,
         "gap_open": 3},
        # A large readjustment batch under the default linear model.
        {"name": "readjust_batch", "kind": "readjust", "triples": 1216, "lmin": 100, "lmax": 300,
         "gap_open": -1},
        # The join proposal: scoring every candidate of a 500-taxon pass ...
        {"name": "proposal_predict", "kind": "predict", "rows": 984102},
        # ... and one optimizer step of its training.
        {"name": "proposal_train", "kind": "train", "rows": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cost", "cost", "align", "align", "chars", "downpass", "readjust",
                       "predict", "train"])
    go = rng.choice([-1, -1, 3])
    if kind == "cost":
        return {"kind": kind, "pairs": _log(rng, 1, 154296), "seqs": _log(rng, 3, 398),
                "length": _log(rng, 100, 1500), "gap_open": go}
    if kind == "align":
        lmax = _log(rng, 100, 5000)
        return {"kind": kind, "pairs": _log(rng, 1, 65536), "lmin": rng.randint(50, lmax),
                "lmax": lmax, "gap_open": go}
    if kind == "chars":
        return {"kind": kind, "nodes": _log(rng, 16, 400), "pairs": _log(rng, 16, 154296),
                "medians": _log(rng, 1, 4256), "fitch": _log(rng, 20, 2000),
                "sank": _log(rng, 5, 200)}
    if kind == "downpass":
        return {"kind": kind, "taxa": _log(rng, 8, 200), "length": _log(rng, 100, 1500),
                "fitch": _log(rng, 10, 2000), "sank": _log(rng, 5, 200)}
    if kind == "readjust":
        lmax = _log(rng, 20, 500)
        most = min(1216, max(1, int(7e9 / lmax ** 3)))
        return {"kind": kind, "triples": _log(rng, 1, most), "lmin": rng.randint(10, lmax),
                "lmax": lmax, "gap_open": go}
    if kind == "predict":
        return {"kind": kind, "rows": _log(rng, 64, 984102)}
    return {"kind": kind, "rows": _log(rng, 64, 16384)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
GAP = 16


class _Dna:
    """Seeded DNA on the device: sequences are a concatenation of bases with
    the owner of every position."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.bases = torch.tensor([1, 2, 4, 8], dtype=torch.uint8, device="cuda")
        self.ambig = torch.tensor([v for v in range(1, 16) if v & (v - 1)], dtype=torch.uint8,
                                  device="cuda")

    def rand(self, n):
        return torch.rand(n, generator=self.g, device="cuda")

    def ints(self, lo, hi, n):
        return torch.randint(lo, hi, (n,), generator=self.g, device="cuda")

    def uniform(self, lo, hi, n):
        return lo + (hi - lo) * self.rand(n)

    def random(self, lens):
        n = int(lens.sum())
        owner = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), lens,
                                        output_size=n)
        return self.bases[self.ints(0, 4, n)], owner

    def evolve(self, base, owner, sub, indel):
        """Substitutions, insertions and deletions of geometric length (mean
        2, at most 8) at the owner's rates."""
        n = len(base)
        s = torch.where(self.rand(n) < sub[owner], self.bases[self.ints(0, 4, n)], base)
        ln = (torch.log2(self.rand(n).clamp(min=1e-6)).neg().floor().long() + 1).clamp(max=8)
        event, dele = self.rand(n) < indel[owner], self.rand(n) < 0.5
        keep = torch.ones(n, dtype=torch.bool, device="cuda")
        dlen = torch.where(event & dele, ln, 0)
        for d in range(min(8, n)):
            keep[d:] &= ~((dlen[:n - d] > d) & (owner[:n - d] == owner[d:]))
        ins = torch.where(event & ~dele, ln, 0)
        count = ins + keep
        src = torch.repeat_interleave(torch.arange(n, device="cuda"), count)
        rank = torch.arange(len(src), device="cuda") - (torch.cumsum(count, 0) - count)[src]
        out = torch.where(rank < ins[src], self.bases[self.ints(0, 4, len(src))], s[src])
        return out, owner[src]

    def masks(self, s, frac, gaps=0.0):
        """IUPAC ambiguity at a fraction of the positions; with `gaps`, the
        gap bit (as a median's optional positions carry it) at another."""
        s = torch.where(self.rand(len(s)) < frac,
                        self.ambig[self.ints(0, len(self.ambig), len(s))], s)
        return torch.where(self.rand(len(s)) < gaps, s | GAP, s) if gaps else s

    @staticmethod
    def pack(parts):
        """(bases, owner, count) parts into one byte buffer, every sequence
        behind its leading gap: (buffer, [(offsets, lengths)] per part)."""
        bufs, places, top = [], [], 0
        for s, owner, k in parts:
            ln = torch.bincount(owner, minlength=k) + 1
            off = torch.cumsum(ln, 0) - ln
            buf = torch.full((len(s) + k,), GAP, dtype=torch.uint8, device="cuda")
            buf[torch.arange(len(s), device="cuda") + owner + 1] = s
            bufs.append(buf)
            places.append((off + top, ln.to(torch.int32)))
            top += len(buf)
        bufs.append(torch.zeros(64, dtype=torch.uint8, device="cuda"))
        return torch.cat(bufs), places


def _buffer(size):
    """The program's own buffer for results of varying length."""
    return torch.zeros(int(size), dtype=torch.uint8, device="cuda")


def _cm(case):
    return align.CostMatrix.dna(1, 2, None if case["gap_open"] < 0 else case["gap_open"])


def _weights(seed):
    rng = np.random.default_rng(seed)
    W = [rng.normal(0, math.sqrt(2.0 / DIMS[i]), (DIMS[i], DIMS[i + 1])).astype(np.float32)
         for i in range(4)]
    b = [rng.normal(0, 0.05, DIMS[i + 1]).astype(np.float32) for i in range(4)]
    return W, b


def _rows(case, seed):
    """Standardised features and targets of `rows` candidates."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((case["rows"], DIMS[0]), generator=g, device="cuda")
    t = X[:, 0] * 0.8 - X[:, 1].clamp(min=0) + 0.3 * X[:, 2] * X[:, 3]
    return X, t + 0.1 * torch.randn(case["rows"], generator=g, device="cuda")


def _prepare_cost(case, seed):
    d = _Dna(seed)
    k, n, L = case["seqs"], case["pairs"], case["length"]
    root = d.bases[d.ints(0, 4, L)]
    owner = torch.arange(k, device="cuda").repeat_interleave(L)
    s, owner = d.evolve(root.repeat(k), owner, d.uniform(0.02, 0.15, k),
                        d.uniform(0.005, 0.03, k))
    buf, [(off, ln)] = d.pack([(d.masks(s, 0.05, 0.005), owner, k)])
    a = d.ints(0, k, n)
    b = (a + 1 + d.ints(0, k - 1, n)) % k
    batch = align.PairBatch(buf, off[a].contiguous(), ln[a].contiguous(), off[b].contiguous(),
                            ln[b].contiguous())
    return {"batch": batch, "cm": _cm(case)}


def _prepare_align(case, seed):
    d = _Dna(seed)
    n = case["pairs"]
    a, oa = d.random(d.ints(case["lmin"], case["lmax"] + 1, n))
    b, ob = d.evolve(a, oa, d.uniform(0.10, 0.30, n), d.uniform(0.02, 0.05, n))
    buf, [(ao, al), (bo, bl)] = d.pack([(d.masks(a, 0.05), oa, n), (d.masks(b, 0.05), ob, n)])
    mean = (case["lmin"] + case["lmax"]) / 2
    most = min(n * (1.5 * case["lmax"] + 64), 1.3 * n * mean + 8 * math.sqrt(n) * case["lmax"])
    return {"batch": align.PairBatch(buf, ao, al, bo, bl), "cm": _cm(case), "rows": _buffer(4 * most)}


def _prepare_chars(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ints = lambda lo, hi, *shape: torch.randint(lo, hi, shape, generator=g, device="cuda")
    nn, nf, ns, k = case["nodes"], case["fitch"], case["sank"], 4
    half = nn // 2
    stride = (nf + 15) // 16 * 16
    fitch = torch.zeros((nn, stride), dtype=torch.uint8, device="cuda")
    one = (1 << ints(0, 8, nn, nf)).to(torch.uint8)
    two = (1 << ints(0, 8, nn, nf)).to(torch.uint8)
    fitch[:, :nf] = one
    fitch[half:, :nf] |= two[half:]  # interior nodes hold sets of states
    sank = ints(0, 40, nn, ns, k).to(torch.int32)
    leaf = torch.full((half, ns, k), native.SANK_INF, dtype=torch.int32, device="cuda")
    leaf.scatter_(2, ints(0, k, half, ns, 1), 0)
    sank[:half] = leaf
    tcm = torch.triu(ints(1, 6, k, k), 1).to(torch.int32)
    idx = lambda n: ints(0, nn, n).to(torch.int32)
    n, m = case["pairs"], case["medians"]
    dev = dict(device="cuda")
    return {"fitch": fitch, "stride": stride, "nf": nf, "sank": sank, "ns": ns, "k": k,
            "tcm": (tcm + tcm.T).contiguous(), "a": idx(n), "b": idx(n), "ma": idx(m),
            "mb": idx(m), "fd": torch.empty(n, dtype=torch.int64, **dev),
            "sd": torch.empty(n, dtype=torch.int64, **dev),
            "fm": torch.zeros((m, stride), dtype=torch.uint8, **dev),
            "fc": torch.empty(m, dtype=torch.int64, **dev),
            "sm": [torch.empty((m, ns, k), dtype=torch.int32, **dev) for _ in range(3)]}


def _prepare_downpass(case, seed):
    n = case["taxa"]
    d = _Dna(seed)
    # sequences evolved down a random tree, level by level
    parent = simulate.yule_tree(np.random.default_rng(seed), n)
    depth = _depths(parent)
    seqs = {2 * n - 2: d.bases[d.ints(0, 4, case["length"])]}
    for lv in range(1, int(depth.max()) + 1):
        vs = np.flatnonzero(depth == lv)
        par = [seqs[int(parent[v])] for v in vs]
        owner = torch.repeat_interleave(
            torch.arange(len(vs), device="cuda"),
            torch.tensor([len(p) for p in par], device="cuda"))
        s, owner = d.evolve(torch.cat(par), owner, torch.full((len(vs),), 0.05, device="cuda"),
                            torch.full((len(vs),), 0.01, device="cuda"))
        for v, x in zip(vs, torch.split(s, torch.bincount(owner, minlength=len(vs)).tolist())):
            seqs[int(v)] = x
    rng = np.random.default_rng(seed)
    nf, ns, k = case["fitch"], case["sank"], 4
    fitch = (1 << rng.integers(0, rng.integers(2, 9, nf), (n, nf))).astype(np.uint8)
    tcm = np.triu(rng.integers(1, 6, (k, k)), 1)
    sank = np.full((n, ns, k), native.SANK_INF, np.int32)
    np.put_along_axis(sank, rng.integers(0, k, (n, ns, 1)), 0, 2)
    data = simulate.Dataset(
        names=["t%d" % i for i in range(n)],
        seqs=[np.concatenate([np.array([GAP], np.uint8), seqs[i].cpu().numpy()])
              for i in range(n)],
        fitch=fitch, fitch_states=np.full(nf, 8), sank=sank,
        sank_tcm=(tcm + tcm.T).astype(np.int32))
    be = search.GpuBackend(data, align.CostMatrix.default())
    # a random start tree, as the SPR passes of a search begin from
    return {"be": be, "tree": learned.random_tree(n, seed + 1),
            "medians": _buffer(8 * (n - 1) * (case["length"] + 64))}


def _depths(parent):
    kids = [[] for _ in parent]
    for v, p in enumerate(parent):
        if p >= 0:
            kids[p].append(v)
    depth = np.zeros(len(parent), np.int64)
    stack = [len(parent) - 1]
    while stack:
        v = stack.pop()
        for c in kids[v]:
            depth[c] = depth[v] + 1
            stack.append(c)
    return depth


def _prepare_readjust(case, seed):
    d = _Dna(seed)
    n = case["triples"]
    anc, owner = d.random(d.ints(case["lmin"], case["lmax"] + 1, n))
    parts = []
    for _ in range(4):  # the two children, the current median, the parent
        s, o = d.evolve(anc, owner, d.uniform(0.05, 0.20, n), d.uniform(0.01, 0.04, n))
        parts.append((d.masks(s, 0.02), o, n))
    buf, places = d.pack(parts)
    return {"batch": three.TripleBatch(buf, [p[0] for p in places], [p[1] for p in places]),
            "cm": _cm(case), "rows": _buffer(4 * n * (2 * case["lmax"] + 64))}


def _prepare_net(case, seed):
    net = mlp.MLP(seed=0)
    W, b = _weights(seed)
    for i in range(4):
        net.W[i].copy_(torch.from_numpy(W[i]))
        net.b[i].copy_(torch.from_numpy(b[i]))
        net.W16[i].copy_(net.W[i])
    X, t = _rows(case, seed)
    if case["kind"] == "train":
        return {"net": net, "X": X.to(torch.bfloat16), "t": t}
    return {"net": net, "X": X}


_PREPARE = {"cost": _prepare_cost, "align": _prepare_align, "chars": _prepare_chars,
            "downpass": _prepare_downpass, "readjust": _prepare_readjust,
            "predict": _prepare_net, "train": _prepare_net}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _run_chars(s):
    L, p = native.lib(), lambda t: C.c_void_p(t.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    n, m, stride = s["a"].numel(), s["ma"].numel(), C.c_int64(s["stride"])
    native.check(L.poyd_nonadd8_distance_batch(p(s["fitch"]), stride, s["nf"], n, p(s["a"]),
                                               p(s["b"]), p(s["fd"]), st))
    native.check(L.poyd_sank_distance_batch(p(s["sank"]), s["ns"], s["k"], p(s["tcm"]), n,
                                            p(s["a"]), p(s["b"]), p(s["sd"]), st))
    native.check(L.poyd_nonadd8_median_batch(p(s["fitch"]), stride, s["nf"], m, p(s["ma"]),
                                             p(s["mb"]), p(s["fm"]), p(s["fc"]), st))
    native.check(L.poyd_sank_median_batch(p(s["sank"]), s["ns"], s["k"], p(s["tcm"]), m,
                                          p(s["ma"]), p(s["mb"]), p(s["sm"][0]), p(s["sm"][1]),
                                          p(s["sm"][2]), st))
    return {"fitch_distance": s["fd"], "sank_distance": s["sd"],
            "fitch_median": s["fm"][:, :s["nf"]], "fitch_cost": s["fc"], "sank_median": s["sm"]}


def run(state):
    kind = state["kind"]
    if kind == "cost":
        return align.cost_2(state["batch"], state["cm"], deltaw="dos")[0]
    if kind == "align":
        p = align.align_2(state["batch"], state["cm"], dos_empty=True).pack()
        state["rows"][:p.packed.numel()].copy_(p.packed)
        return {"cost": p.cost, "rows": state["rows"], "out_len": p.out_len}
    if kind == "chars":
        return _run_chars(state)
    if kind == "downpass":
        be, tree = state["be"], state["tree"]
        d = search.downpass(tree, be)
        nodes = sorted(d.do_cost)
        medians = torch.cat([be.pool[int(be.off[v]):int(be.off[v]) + int(be.len[v])]
                             for v in nodes])
        state["medians"][:medians.numel()].copy_(medians)
        return {"total": d.total, "do": np.array([d.do_cost[v] for v in nodes]),
                "fitch": np.array([d.fitch_cost[v] for v in nodes]), "length": be.len.copy(),
                "medians": state["medians"], "fitch_rows": be.fitch, "sank_rows": be.sank}
    if kind == "readjust":
        r = three.readjust_3d(state["batch"], state["cm"])
        p = align.AlignResult(r.cost, r.out, r.out_off, r.out_len, r.cap, None).pack()
        state["rows"][:p.packed.numel()].copy_(p.packed)
        return {"cost": r.cost, "changed": r.changed, "out_len": r.out_len,
                "rows": state["rows"]}
    net = state["net"]
    if kind == "predict":
        return net.predict(state["X"])
    y = net.forward(state["X"])
    loss, gW, gb = net.backward(state["t"])
    net.step(gW, gb)
    return {"y": y, "loss": loss, "gW": gW, "gb": gb, "W": net.W, "b": net.b}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _pair_cells(mean, square, affine, dos):
    """Cells of the reference's band for one pair of ~`mean` elements: about
    102 diagonals and a tenth (DOS.distance: a fifth) of the length; 85 for
    the affine model."""
    return 85 * mean if affine else 102 * mean + (0.2 if dos else 0.1) * square


def work(case):
    kind = case["kind"]
    if kind in ("cost", "align"):
        n, affine = case["pairs"], case["gap_open"] >= 0
        if kind == "cost":
            L = case["length"]
            cells = n * _pair_cells(L, L * L, affine, True)
            bytes_ = case["seqs"] * L + n * (24 + 4)
        else:
            lo, hi = case["lmin"], case["lmax"]
            mean, square = (lo + hi) / 2, (lo * lo + lo * hi + hi * hi) / 3
            cells = n * _pair_cells(mean, square, affine, False)
            bytes_ = n * (2 * mean + 4.1 * mean + 24 + 12)
        return {"bytes": bytes_, "flops": cells * (24 if affine else 8)}
    if kind == "chars":
        n, m, nf, ns, k = case["pairs"], case["medians"], case["fitch"], case["sank"], 4
        return {"bytes": case["nodes"] * (nf + 4 * k * ns) + n * 24 + m * (nf + 16 + 12 * k * ns),
                "flops": (n + m) * (nf + ns * (4 * k * k + 4 * k))}
    if kind == "downpass":
        n, L, nf, ns, k = case["taxa"], case["length"], case["fitch"], case["sank"], 4
        cells = (n - 1) * _pair_cells(L, L * L, False, False)
        return {"bytes": n * (L + nf + 4 * k * ns) + (n - 1) * (5 * L + nf + 4 * k * ns),
                "flops": 8 * cells + (n - 1) * (nf + ns * 4 * k * k)}
    if kind == "readjust":
        lo, hi = case["lmin"], case["lmax"]
        mean = (lo + hi) / 2
        cube = (lo + hi) * (lo * lo + hi * hi) / 4
        # 7 neighbours a cell; with gap openings, 256 pairs of column states
        return {"bytes": case["triples"] * 8 * mean,
                "flops": case["triples"] * cube * (512 if case["gap_open"] > 0 else 14)}
    weights = sum(DIMS[i] * DIMS[i + 1] for i in range(4))
    n = case["rows"]
    if kind == "predict":
        return {"bytes": n * (4 * DIMS[0] + 4) + 2 * weights, "flops": 2 * n * weights}
    return {"bytes": n * (2 * DIMS[0] + 8) + 34 * weights, "flops": 6 * n * weights}


# ---------------------------------------------------------------------------
# The same in 64 bits (whole-number outputs have to be equal anyway)
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] not in ("predict", "train"):
        return None
    W, b = _weights(seed)
    W = [torch.from_numpy(w).cuda().double() for w in W]
    b = [torch.from_numpy(x).cuda().double() for x in b]
    X, t = _rows(case, seed)
    train = case["kind"] == "train"
    X = X.to(torch.bfloat16).double() if train else X.double()
    H = [X]
    for i in range(3):
        H.append((H[-1] @ W[i] + b[i]).clamp(min=0))
    y = (H[3] @ W[3] + b[3])[:, 0]
    if not train:
        return y
    e = y - t.double()
    dz = (2 * e / len(e))[:, None]
    gW, gb = [None] * 4, [None] * 4
    for i in (3, 2, 1, 0):
        gW[i], gb[i] = H[i].T @ dz, dz.sum(0)
        if i:
            dz = (dz @ W[i].T) * (H[i] > 0)
    lr, eps = 1e-3, 1e-8
    adam = lambda w, g: w - lr * g / (g.abs() + eps)
    return {"y": y, "loss": (e * e).mean()[None], "gW": gW, "gb": gb,
            "W": [adam(w, g) for w, g in zip(W, gW)], "b": [adam(x, g) for x, g in zip(b, gb)]}
