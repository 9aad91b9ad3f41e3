"""The work this library is used for, as measurable cases.

Every case is one call chain a user's program makes through
``distributedpanga_b200.pipeline``; ``listed()`` names the sizes that are
measured, ``draw()`` gives more of the same ranges.  Inputs follow the
generators of ``distributedpanga_b200.synth`` (contig length laws, repeat
content, divergence), made here on the GPU from the seed so that a genome of
hundreds of Mbp takes a fraction of a second.

Kinds:

* ``genomes``  -- a GDB already in host memory (2-bit image and contig
  table), uploaded, indexed, merged, sorted and aligned, the alignments read
  back: one job of the drop-in pipeline.  Families: ``small`` (uniform bases,
  5 % divergence), ``chromset`` (40 % GC, log-normal contigs, 10 % repeats,
  structural variants), ``full`` (40 % interspersed repeats, tandem arrays)
  and ``pangenome`` (one reference and its haplotypes in one GDB).
* ``served``   -- one query assembly (FASTA text) against a resident target.
* ``ingest``   -- a FASTA text to a GDB (2-bit image, contig, scaffold and
  header tables).
* ``requests`` -- a list of Local_Alignment requests on loaded contigs.
* ``stages``   -- the reference's stage functions one after the other on host
  buffers in the reference's byte formats, as its driver calls them.
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from distributedpanga_b200 import gdb, pipeline

FREQ = 10  # the reference driver's frequency cutoff

# Largest sizes of each kind, in bases (a drawn case stays below them).
RANGE = {"small": (20_000, 4_000_000), "chromset": (2_000_000, 100_000_000), "full": (2_000_000, 200_000_000),
         "pangenome": (100_000, 3_000_000), "served": (300_000, 10_000_000), "ingest": (100_000, 300_000_000),
         "requests": (200, 40_000), "stages": (50_000, 3_000_000)}


def listed():
    return [
        # two plasmid- or BAC-sized genomes: launches, synchronisations and fixed tables count
        {"name": "pair 2x41kb", "kind": "genomes", "family": "small", "bases": 41_003},
        # the smallest of the reference's benchmark shapes: 2 Mbp, 5 % divergence
        {"name": "pair 2x2Mb", "kind": "genomes", "family": "small", "bases": 2_000_000},
        # a small eukaryote's two haplotypes
        {"name": "chromset 2x23Mb", "kind": "genomes", "family": "chromset", "bases": 23_170_411},
        # the chromosome-set shape at its full size
        {"name": "chromset 2x100Mb", "kind": "genomes", "family": "chromset", "bases": 100_000_000},
        # repeat-rich genomes, many contigs
        {"name": "full 2x20Mb", "kind": "genomes", "family": "full", "bases": 20_000_000},
        # the largest: repeat-rich at a size whose tables are far beyond L2
        {"name": "full 2x200Mb", "kind": "genomes", "family": "full", "bases": 200_000_000},
        # batched form: 17 genomes of 2.5 Mbp in one GDB, nearly identical
        {"name": "pangenome 17x2.5Mb", "kind": "genomes", "family": "pangenome", "bases": 2_500_000},
        # served form: a query against a resident target that carries the record of its own calls
        {"name": "served 60Mb+4Mb", "kind": "served", "bases": 4_000_000, "target": 60_000_000, "divergence": 0.02,
         "reuse": True},
        # a chromosome-scale FASTA from pinned memory
        {"name": "ingest 200Mb", "kind": "ingest", "bases": 200_000_000, "width": 80},
        # an aligner's inner call on its own: seed hits to extend
        {"name": "requests 20k", "kind": "requests", "count": 20_000, "divergence": 0.03},
        # the reference's driver, stage by stage, on host buffers
        {"name": "stages 2x1Mb", "kind": "stages", "bases": 1_000_003},
    ]


def draw(rng):
    kind = rng.choice(["genomes"] * 6 + ["served", "ingest", "requests", "stages"])
    family = rng.choice(["small", "chromset", "full", "pangenome"]) if kind == "genomes" else None
    lo, hi = RANGE[family or kind]
    size = int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    if kind == "genomes":
        return {"kind": kind, "family": family, "bases": size}
    if kind == "served":
        target = int(math.exp(rng.uniform(math.log(5_000_000), math.log(60_000_000))))
        return {"kind": kind, "bases": min(size, target // 2), "target": target,
                "divergence": round(rng.uniform(0.005, 0.05), 4), "reuse": rng.random() < 0.75}
    if kind == "ingest":
        return {"kind": kind, "bases": min(size, 190_000_000), "width": rng.choice([60, 70, 80, 100])}
    if kind == "requests":
        return {"kind": kind, "count": min(size, 19_999), "divergence": round(rng.uniform(0.005, 0.06), 4)}
    return {"kind": kind, "bases": min(size, 1_000_000)}


# ---- the context -----------------------------------------------------------
# A program makes one context and sends its jobs through it, so all states in
# use share one; it goes when the last of them does.
_CONTEXTS: "weakref.WeakValueDictionary[str, pipeline.Device]" = weakref.WeakValueDictionary()


def context() -> pipeline.Device:
    d = _CONTEXTS.get("0")
    if d is None:
        d = pipeline.Device(0)
        _CONTEXTS["0"] = d
    return d


# ---- genomes on the GPU ------------------------------------------------------
class Maker:
    """Bases (uint8 0..3) on the GPU and lengths on the host, from one seed."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)
        self.h = np.random.default_rng(seed)

    def uniform(self, n: int) -> torch.Tensor:
        return torch.rand(n, device="cuda", generator=self.g)

    def below(self, n: int, hi: int, dtype=torch.uint8) -> torch.Tensor:
        return torch.randint(0, hi, (n,), device="cuda", dtype=dtype, generator=self.g)

    def bases(self, n: int, gc: float = 0.5) -> torch.Tensor:
        if gc == 0.5:
            return self.below(n, 4)
        r = self.uniform(n)
        at = (1.0 - gc) / 2.0
        return ((r >= at).to(torch.uint8) + (r >= 0.5).to(torch.uint8) + (r >= 1.0 - at).to(torch.uint8))

    def substitute(self, s: torch.Tensor, rate) -> torch.Tensor:
        """Other bases at ``rate`` of positions (a number, or one per position)."""
        n = s.numel()
        return torch.where(self.uniform(n) < rate, (s + 1 + self.below(n, 3)) & 3, s)

    def indels(self, s: torch.Tensor, rate: float, lengths, gc: float):
        """Insertions and deletions (half each) at ``rate`` of positions; also
        the place of each base of s in the result."""
        n = s.numel()
        k = int(self.h.binomial(n, rate))
        pos = torch.from_numpy(np.unique(self.h.integers(0, n, size=k))).cuda()
        k = pos.numel()
        ln = torch.from_numpy(lengths(k).astype(np.int64)).cuda()
        ins = torch.from_numpy(self.h.random(k) < 0.5).cuda()
        edge = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        at, dl = pos[~ins], ln[~ins]
        one = torch.ones_like(at, dtype=torch.int32)
        edge.index_add_(0, at, one)
        edge.index_add_(0, torch.clamp(at + dl, max=n), -one)
        count = (torch.cumsum(edge, 0)[:n] == 0).to(torch.int64)
        count.index_add_(0, pos[ins], ln[ins])
        start = torch.cumsum(count, 0) - count
        out = self.bases(int(count.sum()), gc)
        kept = torch.cumsum(edge, 0)[:n] == 0
        last = (start + count - 1)[kept]  # a kept base follows what is inserted before it
        out[last] = s[kept]
        return out, start

    def invert(self, s: torch.Tensor, count: int, lo: int, hi: int) -> torch.Tensor:
        out, n = s.clone(), s.numel()
        for _ in range(count):
            ln = int(self.h.integers(lo, hi + 1))
            if ln < n:
                p = int(self.h.integers(0, n - ln))
                out[p:p + ln] = 3 - out[p:p + ln].flip(0)
        return out

    def translocate(self, s: torch.Tensor, count: int, lo: int, hi: int) -> torch.Tensor:
        out = s
        for _ in range(count):
            n = out.numel()
            ln = int(self.h.integers(lo, hi + 1))
            if ln < n // 2:
                p = int(self.h.integers(0, n - ln))
                rest = torch.cat([out[:p], out[p + ln:]])
                q = int(self.h.integers(0, rest.numel()))
                out = torch.cat([rest[:q], out[p:p + ln], rest[q:]])
        return out

    def owners(self, n: int, ln: np.ndarray, start: np.ndarray) -> torch.Tensor:
        """Which of the placed pieces covers each position (the last placed; -1 none)."""
        l, st = torch.from_numpy(ln).cuda(), torch.from_numpy(start).cuda()
        piece = torch.repeat_interleave(torch.arange(len(ln), device="cuda", dtype=torch.int32), l)
        first = torch.cumsum(l, 0) - l
        at = torch.arange(piece.numel(), device="cuda") - first[piece.long()] + st[piece.long()]
        own = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        return own.scatter_reduce_(0, at, piece, "amax")

    def pieces(self, n: int, fraction: float, draw_len) -> np.ndarray:
        """Lengths of pieces that sum to about ``fraction`` of n."""
        out, covered = [], 0
        while covered < fraction * n:
            ln = np.minimum(draw_len(max(64, int(fraction * n / 3000))), n - 1)
            c = np.cumsum(ln) + covered
            take = int(np.searchsorted(c, fraction * n)) + 1
            out.append(ln[:take])
            covered = int(c[min(take, len(c)) - 1])
        return np.concatenate(out).astype(np.int64)

    def repeats(self, s: torch.Tensor, fraction: float, families: int, lo: int, hi: int, gc: float) -> torch.Tensor:
        """``fraction`` of s overwritten by 10-20 % diverged copies, either strand, of repeat families."""
        n = s.numel()
        unit = np.minimum(self.h.integers(lo, hi + 1, size=families), n - 1)
        fam = self.h.integers(0, families, size=max(1, round(fraction * n / float(unit.mean()))))
        ln = unit[fam].astype(np.int64)
        start = (self.h.random(len(ln)) * (n - ln)).astype(np.int64)
        cons = self.bases(int(unit.sum()), gc)
        ufirst = torch.from_numpy(np.cumsum(unit) - unit).cuda()
        own = self.owners(n, ln, start)
        on = (own >= 0).nonzero().squeeze(1)
        o = own[on].long()
        off = on - torch.from_numpy(start).cuda()[o]
        rc = torch.from_numpy(self.h.random(len(ln)) < 0.5).cuda()[o]
        l = torch.from_numpy(ln).cuda()[o]
        copy = cons[ufirst[torch.from_numpy(fam).cuda()[o]] + torch.where(rc, l - 1 - off, off)]
        copy = torch.where(rc, 3 - copy, copy)
        div = torch.from_numpy(self.h.uniform(0.10, 0.20, size=len(ln)).astype(np.float32)).cuda()[o]
        out = s.clone()
        out[on] = self.substitute(copy, div)
        return out

    def tandems(self, s: torch.Tensor, fraction: float, lo: int, hi: int) -> torch.Tensor:
        """``fraction`` of s overwritten by tandem arrays (unit 2-200 bases, 2 % diverged)."""
        n = s.numel()
        ln = self.pieces(n, fraction, lambda k: self.h.integers(lo, hi + 1, size=k))
        unit = self.h.integers(2, 201, size=len(ln))
        start = (self.h.random(len(ln)) * (n - ln)).astype(np.int64)
        u = torch.from_numpy(unit).cuda()
        cons = self.bases(int(unit.sum()))
        own = self.owners(n, ln, start)
        on = (own >= 0).nonzero().squeeze(1)
        o = own[on].long()
        off = on - torch.from_numpy(start).cuda()[o]
        out = s.clone()
        out[on] = self.substitute(cons[(torch.cumsum(u, 0) - u)[o] + off % u[o]], 0.02)
        return out

    def cut_uniform(self, n: int, lo: int, hi: int) -> list:
        """Contig lengths U[lo, hi]; a short tail joins the last."""
        out, p = [], 0
        while p < n:
            ln = int(self.h.integers(lo, hi + 1))
            ln = n - p if n - p - ln < lo else ln
            out.append(ln)
            p += ln
        return out

    def cut_lognormal(self, n: int, median: float, lo: int, hi: int = 1 << 30) -> list:
        out, p = [], 0
        while p < n:
            ln = int(min(hi, max(lo, self.h.lognormal(math.log(median), 1.0))))
            ln = n - p if n - p - ln < lo else ln
            out.append(ln)
            p += ln
        return out


def geometric(m: Maker):
    return lambda k: m.h.geometric(1.0 / 3.0, size=k)


def genomes(m: Maker, family: str, n: int) -> list:
    """(genome, contig lengths) of one GDB, as synth's generator of that name makes them."""
    if family == "small":
        f = n / 2_000_000
        a = m.bases(n)
        b, _ = m.indels(m.substitute(a, 0.05), 0.005, lambda k: m.h.integers(1, 11, size=k), 0.5)
        b = m.invert(b, 20, max(40, int(5_000 * f)), max(80, int(50_000 * f)))
        lo, hi = max(200, int(50_000 * f)), max(400, int(500_000 * f))
        return [(a, m.cut_uniform(n, lo, hi)), (b, m.cut_uniform(b.numel(), lo, hi))]
    if family == "chromset":
        f = n / 100_000_000
        lo, hi = max(20, int(300 * min(1.0, f * 10))), max(40, int(6000 * min(1.0, f * 10)))
        a = m.repeats(m.bases(n, 0.40), 0.10, 300, lo, hi, 0.40)
        b, _ = m.indels(m.substitute(a, 0.015), 0.002, geometric(m), 0.40)
        svlo, svhi = max(50, int(10_000 * f)), max(100, int(1_000_000 * f))
        b = m.translocate(m.invert(b, 50, svlo, svhi), 50, svlo, svhi)
        med, least = max(2_000, 2_000_000 * f), max(100, int(10_000 * f))
        return [(a, m.cut_lognormal(n, med, least)), (b, m.cut_lognormal(b.numel(), med, least))]
    if family == "full":
        f = n / 1_000_000_000
        a = m.repeats(m.bases(n), 0.40, 300, max(20, int(300 * min(1.0, f * 10))),
                      max(40, int(6000 * min(1.0, f * 10))), 0.5)
        a = m.tandems(a, 0.03, max(50, int(500 * min(1.0, f * 10))), max(100, int(10_000 * min(1.0, f * 10))))
        b, _ = m.indels(m.substitute(a, 0.02), 0.005, lambda k: m.h.integers(1, 11, size=k), 0.5)
        b = m.invert(b, 20, max(40, int(5_000 * f)), max(80, int(50_000 * f)))
        lo, hi = max(200, int(50_000 * f)), max(400, int(500_000 * f))
        return [(a, m.cut_uniform(n, lo, hi)), (b, m.cut_uniform(b.numel(), lo, hi))]
    f = max(n / 50_000_000, 0.05)
    lo, hi, med = int(10_000 * f), int(5_000_000 * f), 224_000 * f
    svlo, svhi = max(50, int(1_000 * n / 50_000_000)), max(100, int(100_000 * n / 50_000_000))
    ref = m.bases(n)
    out = [(ref, m.cut_lognormal(n, med, lo, hi))]
    for _ in range(16):
        d = float(m.h.uniform(0.001, 0.01))
        h, _ = m.indels(m.substitute(ref, d), d / 10, geometric(m), 0.5)
        h = m.translocate(m.invert(h, 10, svlo, svhi), 5, svlo, svhi)
        out.append((h, m.cut_lognormal(h.numel(), med, lo, hi)))
    return out


def contig_set(parts: list) -> gdb.ContigSet:
    """The GDB image and tables of (genome, contig lengths) parts, in host memory."""
    rows, lens, pad = [], [], torch.zeros(3, dtype=torch.uint8, device="cuda")
    for s, cuts in parts:
        p = 0
        for ln in cuts:
            rows.append(s[p:p + ln])
            if ln & 3:
                rows.append(pad[:4 - (ln & 3)])
            lens.append(ln)
            p += ln
    q = torch.cat(rows).view(-1, 4)
    bps = (q[:, 0] | (q[:, 1] << 2) | (q[:, 2] << 4) | (q[:, 3] << 6)).cpu().numpy()
    clen = np.array(lens, dtype=np.int64)
    nbytes = (clen + 3) // 4
    counts = sum(torch.bincount(s, minlength=4) for s, _ in parts).cpu().numpy()
    return gdb.ContigSet(bps=bps, clen=clen, boff=np.cumsum(nbytes) - nbytes,
                         freq=(counts / counts.sum()).astype(np.float32))


def fasta(parts: list, prefix: str, width: int = 80, runs: int = 0, m: Maker | None = None) -> torch.Tensor:
    """FASTA text of the parts' contigs, on the GPU; ``runs`` stretches of N in each part, a third of it lower case."""
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")
    out, at = [], 0
    for s, cuts in parts:
        t = letters[s.long()]
        if runs:
            n = t.numel()
            t[: n // 3] |= 0x20
            for _ in range(runs):
                ln = int(m.h.integers(1, max(3, min(2000, n // 1000))))  # never a whole contig
                p = int(m.h.integers(0, max(1, n - ln)))
                t[p:p + ln] = ord("N")
        p = 0
        for ln in cuts:
            out.append(torch.tensor(list(b">%s%d sample\n" % (prefix.encode(), at)), dtype=torch.uint8).cuda())
            full = ln // width
            lines = torch.full((full, width + 1), ord("\n"), dtype=torch.uint8, device="cuda")
            lines[:, :width] = t[p:p + full * width].view(full, width)
            out.append(lines.view(-1))
            if ln % width:
                out.append(t[p + full * width:p + ln])
                out.append(torch.full((1,), ord("\n"), dtype=torch.uint8, device="cuda"))
            p += ln
            at += 1
    return torch.cat(out)


def target_genome(m: Maker, n: int) -> list:
    """One genome with chromset's bases and repeats, contigs of median 2 Mbp."""
    a = m.repeats(m.bases(n, 0.40), 0.10, 300, 300, 6000, 0.40)
    f = max(n / 1_000_000_000, 0.05)
    return [(a, m.cut_lognormal(n, 2_000_000 * f, int(10_000 * f)))]


# ---- the interface -----------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    m, kind = Maker(seed), case["kind"]
    st = {"kind": kind, "dev": context(), "room": room(case)}
    if kind in ("genomes", "stages"):
        st["cs"] = contig_set(genomes(m, case.get("family", "small"), case["bases"]))
    elif kind == "served":
        target = target_genome(m, case["target"])
        a = target[0][0]
        p = int(m.h.integers(0, a.numel() - case["bases"] + 1))
        q = a[p:p + case["bases"]]
        q = 3 - q.flip(0) if m.h.random() < 0.25 else q
        q, _ = m.indels(m.substitute(q, case["divergence"]), case["divergence"] / 10, geometric(m), 0.40)
        cuts = m.cut_lognormal(q.numel(), 1_000_000, max(100, min(10_000, q.numel() // 4)))
        st["query"] = fasta([(q, cuts)], "q").cpu().numpy().tobytes()
        st["target"] = pipeline.Target(fasta(target, "t").cpu().numpy().tobytes(), reuse=case["reuse"], freq=FREQ)
    elif kind == "ingest":
        n = case["bases"]
        text = fasta([(m.bases(n, 0.41), m.cut_lognormal(n, max(2_000, n / 40), max(100, n // 400)))], "chr",
                     case["width"], 50, m)
        pinned = torch.empty(text.numel(), dtype=torch.uint8, pin_memory=True)
        pinned.copy_(text)
        st["text"] = pinned
    elif kind == "requests":
        st["cs"], st["req"] = request_list(m, case["count"], case["divergence"])
    return st


def request_list(m: Maker, count: int, divergence: float):
    """Two genomes and ``count`` seed hits between them, as the chain driver
    passes them on: a diagonal band at an antidiagonal, nine in ten on true
    homology and the rest chance hits."""
    n = max(100_000, 250 * count)
    a = m.bases(n)
    b, start = m.indels(m.substitute(a, divergence), divergence / 10, geometric(m), 0.5)
    # contigs of 2-10 kbp: an extension ends at a contig's end after a few thousand bases
    ca = np.array(m.cut_uniform(n, 2_000, 10_000))
    cb = np.array(m.cut_uniform(b.numel(), 2_000, 10_000))
    ea, eb = np.cumsum(ca), np.cumsum(cb)
    x = m.h.integers(0, n, size=4 * count)
    y = start[torch.from_numpy(x).cuda()].cpu().numpy()
    chance = m.h.random(4 * count) < 0.1
    y = np.where(chance, m.h.integers(0, b.numel(), size=4 * count), y)
    i, j = np.searchsorted(ea, x, side="right"), np.searchsorted(eb, np.minimum(y, b.numel() - 1), side="right")
    px, py = x - (ea[i] - ca[i]), np.minimum(y, b.numel() - 1) - (eb[j] - cb[j])
    # a band's start points lie inside both contigs
    ok = (px > 150) & (py > 150) & (px < ca[i] - 150) & (py < cb[j] - 150)
    px, py, i, j = (v[ok][:count] for v in (px, py, i, j))
    w = m.h.integers(0, 64, size=len(px))
    lo = px - py - m.h.integers(0, 64, size=len(px)) % (w + 1)
    req = np.stack([i, j + len(ca), np.zeros_like(i), lo, lo + w, px + py, np.full_like(i, -1), np.full_like(i, -1)],
                   axis=1).astype(np.int32)
    return contig_set([(a, ca.tolist()), (b, cb.tolist())]), np.ascontiguousarray(req)


def room(case: dict) -> dict:
    """Places for each output of a case: well above what its inputs can give.
    How many alignments, contigs or seeds come out depends on the seed; the
    outputs are laid out in arrays of one size, the rest zero."""
    kind, n = case["kind"], case["bases"] if "bases" in case else case["count"]
    if kind == "genomes":
        rec, trace = {"small": (2_000, n // 8), "chromset": (4_000 + n // 4_000, n // 4),
                      "full": (4_000 + n // 400, n // 3), "pangenome": (4_000 + n // 12, 8 * n)}[case["family"]]
        return {"records": rec * 9, "offsets": rec + 1, "trace": trace + 50_000}
    if kind == "served":
        g = n + case["target"]
        return {"records": (5_000 + g // 2_000) * 9, "offsets": 5_001 + g // 2_000, "trace": g // 15 + 50_000}
    if kind == "ingest":
        return {"bps": n // 4 + 4_096, "contigs": 4 * 4_096, "scaffolds": 4 * 4_096, "headers": 65_536, "count": 4}
    if kind == "requests":
        return {"paths": n * 7, "offsets": n + 1, "trace": 250 * n}
    return {"records": 2 * n * 17 + 10_000, "nseeds": 14 * n + 10_000, "cseeds": 8 * n + 10_000, "nbuck": 4_096,
            "cbuck": 4_096, "panel0": 14 * n + 10_000, "off0": 4_096, "panel1": 8 * n + 10_000, "off1": 4_096}


def laid_out(st: dict, **outputs) -> dict:
    out = {}
    for name, a in outputs.items():
        flat = a.reshape(-1)
        out[name] = np.zeros(st["room"][name], dtype=a.dtype)
        out[name][:flat.size] = flat
    return out


def run(st: dict):
    dev, kind = st["dev"], st["kind"]
    if kind == "genomes":
        cs = st["cs"]
        dev.gdb_load(cs)
        dev.set_freq(cs.freq)
        nrec = dev.index_build(want_entries=False)
        nseeds = dev.merge(FREQ)
        dev.align()
        recs, toff, tr = dev.alignments()
        return {"sizes": np.array([nrec, *nseeds, len(recs)]), **laid_out(st, records=recs, offsets=toff, trace=tr)}
    if kind == "served":
        sizes = dev.serve_load(st["target"], st["query"])
        nseeds = dev.merge(FREQ)
        dev.align()
        recs, toff, tr = dev.alignments()
        return {"sizes": np.array([*sizes, *nseeds, len(recs)]),
                **laid_out(st, records=recs, offsets=toff, trace=tr)}
    if kind == "ingest":
        t = dev.gdb_ingest_fasta(st["text"].data_ptr(), nbytes=st["text"].numel())
        return laid_out(st, bps=t.bps, contigs=t.contigs, scaffolds=t.scaffolds,
                        headers=np.frombuffer(t.headers, dtype=np.uint8), count=t.count)
    if kind == "requests":
        cs = st["cs"]
        dev.gdb_load(cs)
        dev.set_freq(cs.freq)
        path, toff, tr = dev.local_alignment(st["req"])
        return laid_out(st, paths=path, offsets=toff, trace=tr)
    cs = st["cs"]
    dev.gdb_load(cs)
    posb, ctgb, _ = gdb.record_sizing(cs)
    dbyte, _ = gdb.diag_sizing(cs, ctgb)
    rec = dev.sort_records(dev.extract_to_records(), posb, ctgb)
    ent, cum, largest = dev.build_kmer_adapter(rec, posb, ctgb)
    nseed, cseed, nbuck, cbuck = dev.self_adaptamer_merge(ent, cum, posb, ctgb, FREQ, cs.ncontig)
    out = {"records": rec, "nseeds": nseed, "cseeds": cseed, "nbuck": nbuck, "cbuck": cbuck}
    for comp, seeds in ((0, nseed), (1, cseed)):
        out["panel%d" % comp], out["off%d" % comp] = dev.reimport_sort(seeds, posb, ctgb, comp, cs.ncontig,
                                                                       cs.maxctg, dbyte)
    return {"sizes": np.array([*rec.shape, *nseed.shape, *cseed.shape, largest]), **laid_out(st, **out)}


def work(case: dict) -> dict:
    """Bytes of the inputs and outputs (no floating-point arithmetic on any path).

    genomes and served: the k-mer records (16 bytes each, 0.8 per base, read
    and written once by the sort) are what the path cannot do without besides
    the 2-bit image; requests: each side of an extension reads its packed
    bases once and writes a trace; stages: the reference's 17-byte records
    and 14-byte entries cross the host boundary."""
    kind = case["kind"]
    if kind == "genomes":
        g = case["bases"] * (17 if case["family"] == "pangenome" else 2)
        return {"bytes": g / 4 + 2 * 16 * 0.8 * g, "flops": 0.0}
    if kind == "served":
        g = case["bases"] + case["target"]
        return {"bytes": case["bases"] + 2 * 16 * 0.8 * g, "flops": 0.0}
    if kind == "ingest":
        return {"bytes": case["bases"] * (1 + 1 / case["width"] + 0.25), "flops": 0.0}
    if kind == "requests":
        return {"bytes": case["count"] * (32 + 28 + 2 * 4_000 / 4 + 4 * 40), "flops": 0.0}
    return {"bytes": 2 * case["bases"] * (0.25 + 0.8 * (3 * 17 + 14) + 2 * 0.8 * 14), "flops": 0.0}
