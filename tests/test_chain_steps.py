"""A band block's chains, found many seeds a step: seeds loaded for one pair so
that a stream holds as many as the steps take (32, 256) or one more or less,
with ties between the streams and breaks in the chains at the steps' ends, one
block per case, against the scalar aligner on the same seeds.  Integers: equal."""
import numpy as np
import pytest

from test_align_host import aht, aln_lines, run_unit  # noqa: F401 (aht: a fixture)

LA, LB, BANDS = 100_000, 60_000, 5
COUNTS = [1, 31, 32, 33, 63, 64, 65, 255, 256, 257, 287, 288, 289, 512, 513, 545]
BREAK = 2000


def block(rng, n1, n2, gap, edge, tie):
    """(antidiagonal, match length) of the seeds of the two streams.  edge:
    where a seed of the first starts that far past the chain's end."""
    out = []
    for st, n in enumerate((n1, n2)):
        a, end, seeds = int(rng.integers(0, 200)), 0, []
        for i in range(n):
            a += int(rng.integers(0, gap))
            if st == 0 and edge is not None and i in (32, 288, n - 1):
                a = max(a, end + edge)
            if st == 1 and tie and i % 3 == 0 and out[0]:
                later = [x for x, _ in out[0] if x >= a]
                a = later[0] if later else a
            seeds.append((a, int(rng.integers(12, 41))))
            end = max(end, a + 2 * seeds[-1][1])
        out.append(seeds)
    return out


def pair(seed):
    """Contigs a and b, b's stretches copies of a's on the diagonals of the
    blocks, and the seeds (match length, a's position, b's)."""
    from distributedpanga_b200 import synth
    rng = np.random.default_rng(seed)
    a, b = synth.random_bases(rng, LA, 0.5), synth.random_bases(rng, LB, 0.5)
    cases = []
    for n1 in COUNTS:
        for n2 in (0, int(rng.choice([1, 32, 33, 300]))):
            cases.append((n1, n2, int(rng.choice([2, 12, 60])), None, bool(rng.integers(0, 2))))
    for edge in (BREAK - 2, BREAK - 1, BREAK, BREAK + 1):
        for n1, n2 in ((33, 0), (289, 0), (289, 40), (600, 0)):
            cases.append((n1, n2, 12, edge, False))
    cases = [cases[i] for i in rng.permutation(len(cases))]
    seeds = []
    for c, (n1, n2, gap, edge, tie) in enumerate(cases):
        band = (LA + 8000) // 64 + BANDS * c
        base, j0 = 64 * band - LA, int(rng.integers(0, 30_000))
        d = base + 40
        if c < 12:
            j = 1000 + 4800 * c
            b[j:j + 3000] = synth.substitute(rng, a[j + d:j + d + 3000], 0.03)
            j0 = max(j - int(rng.integers(0, 3000)), 0)
        for st, part in enumerate(block(rng, n1, n2, gap, edge, tie)):
            for at, lcp in part:
                anti = 2 * j0 + base + 200 + at
                diag = base + 64 * st + 2 * int(rng.integers(0, 32)) + (anti & 1)
                i, j = (anti + diag) // 2, (anti - diag) // 2
                if 0 <= j < LB and i < LA:
                    seeds.append((lcp, i, j))
    return [a, b], seeds


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_chains_equal_the_scalar_scan(dev, oracle, aht, seed):  # noqa: F811
    from distributedpanga_b200 import gdb
    ctgs, seeds = pair(seed)
    cs = gdb.from_contigs(ctgs)
    posb, ctgb, _ = gdb.record_sizing(cs)
    dbyte, swide = gdb.diag_sizing(cs, ctgb)
    raw = np.zeros((len(seeds), 1 + 2 * (posb + ctgb)), np.uint8)
    for s, (lcp, i, j) in enumerate(seeds):
        raw[s] = np.frombuffer(bytes([lcp]) + i.to_bytes(posb, "little") + bytes(ctgb) +
                               j.to_bytes(posb, "little") + (1).to_bytes(ctgb, "little"), np.uint8)
    raw = raw[np.random.default_rng(seed).permutation(len(raw))]
    arr, off = oracle.reimport_sort(raw, posb, ctgb, 0, cs.ncontig, cs.maxctg, dbyte)
    out, pairs = run_unit(aht, cs, arr, off, dict(swide=swide, dbyte=dbyte, ctgb=ctgb), 0)
    want = [" ".join(x.split()) for x in aln_lines(out)]
    assert len(want) >= 4 and int(pairs[:, 2].sum()) > 500
    from distributedpanga_b200.pipeline import alignment_lines
    dev.gdb_load(cs)
    dev.seeds_load(0, raw)
    dev.seeds_load(1, raw[:0])
    dev.diag_sort(0)
    dev.diag_sort(1)
    try:
        for build in (2, 5):
            dev.set_build(build)
            dev.align()
            assert dev.align_stats()["calls"] == int(pairs[:, 2].sum())
            assert [" ".join(x.split()) for x in alignment_lines(*dev.alignments())] == want
    finally:
        dev.set_build(0)
