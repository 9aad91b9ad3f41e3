"""The device's Local_Alignment run on the CPU (tests/native/warp_lanes.h)
where a launch's shared extensions run out of something, and in the builds
that only many-pair launches take, against the oracle's scalar restatement.
Integers: equal."""
import numpy as np
import pytest

from test_warp_lanes import check, lanes, on_lanes, scalar  # noqa: F401 (lanes: a fixture)
from test_wave_widths import contigs, requests


def one_path(seed):
    """Calls along one alignment of three lines, late ones first in turn."""
    from distributedpanga_b200 import synth
    rng = np.random.default_rng(seed)
    a = synth.random_bases(rng, 40_000, 0.45)
    b = synth.indels(rng, synth.substitute(rng, a, 0.01), 0.002, lambda k: rng.integers(1, 9, size=k), 0.5)
    req = []
    for x in (9000, 300, 20_000, 2500, 17_000, 700):
        y = x * len(b) // len(a)
        req.append([0, 1, 0, x - y - 20, x - y + 20, x + y, -1, -1])
    return [a, b], req


# what runs out; the entries, records and list places there are
@pytest.mark.parametrize("entries,records,listed", [(4096, 4096, 1 << 20), (0, 4096, 1 << 20), (1, 4096, 1 << 20),
                                                    (3, 4096, 1 << 20), (4096, 0, 1 << 20), (4096, 1, 1 << 20),
                                                    (4096, 3, 1 << 20), (4096, 4096, 0), (4096, 4096, 90),
                                                    (4096, 4096, 400)])
@pytest.mark.parametrize("turns", [0, 300])
def test_paths_are_the_same_where_sharing_runs_out(lanes, turns, entries, records, listed):  # noqa: F811
    cs, req = one_path(7)
    out = on_lanes(lanes, cs, req, turns=turns, seed=5, entries=entries, records=records, listed=listed)
    assert (out.err == 0).all() and out.open == 0 and out.misplaced == 0
    check(out, scalar(cs, req))
    assert out.entries <= entries and out.records <= records
    if entries == records == 4096:
        assert out.entries > 3 and out.pebble + out.head > 0
        assert (out.failed > 0) == (listed < 1 << 20)
        if listed == 1 << 20:
            assert out.joined > 0


@pytest.mark.parametrize("blocks", [False, True])
@pytest.mark.parametrize("div", [0.0, 0.06, 0.2])
def test_both_loops_equal_the_scalar_aligner(lanes, blocks, div):  # noqa: F811
    """The loops of the builds with many resident warps (blocks False) and of
    those with few, bands around where a wave changes form."""
    cs = contigs(div)
    req = np.concatenate([requests(cs, w)[::3] for w in (1, 30, 31, 32, 33, 64, 65, 124, 129)])
    out = on_lanes(lanes, cs, req, blocks=blocks, share=False, cells=40_000)
    assert (out.err == 0).all()
    check(out, scalar(cs, req))
