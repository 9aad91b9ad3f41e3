"""That extensions are shared on the GPU at all: a path of many lines that many
calls lead into, in the build that shares and in one that does not."""
import numpy as np
import pytest

from test_shared_extensions import contigs


@pytest.mark.gpu
@pytest.mark.parametrize("div", [0.002, 0.01])
def test_calls_of_a_launch_meet(dev, div):
    from distributedpanga_b200 import gdb
    dev.gdb_load(gdb.from_contigs(contigs(div)))
    dev.index_build(want_entries=False)
    dev.merge(10)
    try:
        dev.set_ranges(48)
        dev.set_build(3)
        dev.align()
        alone, none = dev.alignments(), dev.share_stats()
        dev.set_build(2)
        dev.align()
        shared, stats = dev.alignments(), dev.share_stats()
    finally:
        dev.set_build(0)
        dev.set_ranges(0)
    assert all(np.array_equal(x, y) for x, y in zip(alone, shared))
    assert not any(none.values())
    # the longest path crosses every line of 400 kbp, 48 of them, but the last
    # few; some call or scout enters each and another arrives there
    assert stats["launches"] >= 1 and stats["entries"] > 40 and stats["records"] > 0 and stats["scouts"] > 0
    assert stats["joins_past_mark"] + stats["joins_before_mark"] + stats["joins_own_tip"] > 0
