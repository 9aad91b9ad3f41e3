"""Extensions shared between the calls of a launch (align_share.cuh) against
the same launch's calls growing alone: contigs of many lines, one divergence
per case, on both strands, with tandem arrays, unrelated stretches and exact
copies of a contig in them (equal waves of two pairs), and with the band
ranges that decide which calls meet.  Alignments and traces: equal."""
import numpy as np
import pytest


def contigs(div: float):
    from distributedpanga_b200 import synth
    rng = np.random.default_rng(int(1000 * div) + 17)

    def evolve(s, at):
        return s if at == 0 else synth.indels(rng, synth.substitute(rng, s, at), at / 6,
                                              lambda k: rng.integers(1, 12, size=k), 0.45)

    a = synth.random_bases(rng, 400_031, 0.45)
    unit = synth.random_bases(rng, 53, 0.5)
    a[90_000:94_000] = np.resize(unit, 4000)             # a tandem array across a line
    b = evolve(a, div)
    cut = 150_000
    c = np.concatenate([evolve(a[:cut], div), synth.random_bases(rng, 30_000, 0.5), synth.revcomp(evolve(a[cut:], div))])
    return [a, b, b.copy(), c, evolve(a[60_000:130_001], div)]


@pytest.mark.gpu
@pytest.mark.parametrize("div", [0.0, 0.002, 0.01, 0.05, 0.12])
def test_shared_equals_alone(dev, div):
    from distributedpanga_b200 import gdb
    g = gdb.from_contigs(contigs(div))
    dev.gdb_load(g)
    dev.index_build(want_entries=False)
    dev.merge(10)
    out = {}
    try:
        for ranges in (48, 400, 0):
            dev.set_ranges(ranges)
            for build in (5, 3, 2, 2):
                dev.set_build(build)
                dev.align()
                got = dev.alignments()
                want = out.setdefault("alone", got)
                assert all(np.array_equal(x, y) for x, y in zip(got, want)), (ranges, build)
    finally:
        dev.set_build(0)
        dev.set_ranges(0)
    rec = out["alone"][0]
    assert len(rec) > 5
    if div <= 0.01:
        assert (rec[:, 2] - rec[:, 1] > 65_536).any()    # paths of many lines
