"""Which band blocks are scanned, decided 32 seeds at a time: a pair cut into
parts of few seeds, so that the parts' ends and the pair's last band fall
everywhere in those groups, against the whole pair scanned by one warp."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["edge_mix", "small_s002"])
def test_parts_equal_whole(dev, case):
    from conftest import load_case
    cs, dig = load_case(case)
    dev.gdb_load(cs)
    dev.index_build(want_entries=False)
    dev.merge(dig["freq_cutoff"])
    try:
        dev.set_ranges(-1)
        dev.align()
        want = dev.alignments()
        assert len(want[0]) > 0
        for seeds in (1, 2, 3, 7, 31, 32, 33, 63, 64, 65, 97, 127, 128, 129, 161, 300):
            for build in (2, 5):
                dev.set_build(build)
                dev.set_ranges(seeds)
                dev.align()
                assert all(np.array_equal(x, y) for x, y in zip(dev.alignments(), want)), (seeds, build)
    finally:
        dev.set_build(0)
        dev.set_ranges(0)
