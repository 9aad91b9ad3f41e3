"""Copies of pageable memory in chunks by several threads (hostcopy.h) against
the driver's copies of pinned memory, in and out of the device, at sizes around
the smallest staged copy and around whole chunks."""
import numpy as np
import pytest

MB = 1 << 20


@pytest.mark.gpu
@pytest.mark.parametrize("nbytes", [4 * MB - 18, 4 * MB, 4 * MB + 18, 5 * MB + 1, 16 * MB, 17 * MB - 7, 53 * MB + 5])
def test_pageable_equals_pinned(dev, nbytes):
    import torch
    posb, ctgb = 4, 2
    n = -(-nbytes // (12 + posb + ctgb))
    rng = np.random.default_rng(nbytes)
    rec = np.zeros((n, 12 + posb + ctgb), dtype=np.uint8)
    rec[:, 2:] = rng.integers(0, 256, size=(n, 10 + posb + ctgb), dtype=np.uint8)
    rec[:, -1] &= 0x7f
    pinned = torch.from_numpy(rec.copy()).pin_memory().numpy()
    assert dev.L.pga_sort_records(dev.h, pinned.ctypes.data, n, posb, ctgb) == 0
    got = dev.sort_records(rec, posb, ctgb)
    assert np.array_equal(got, pinned)
    assert not np.array_equal(got, rec)


@pytest.mark.gpu
def test_taken_buffers_outlive_their_call(dev):
    """The driver's record buffer stays valid while an array of it does."""
    from distributedpanga_b200 import gdb, synth
    rng = np.random.default_rng(5)
    dev.gdb_load(gdb.from_contigs([synth.random_bases(rng, 400_000, 0.5)]))
    a = dev.extract_to_records()
    keep, want = a[1000:2000], a.copy()
    b = dev.extract_to_records()
    assert np.array_equal(a, b) and np.array_equal(keep, want[1000:2000])
    del a, b
    assert np.array_equal(keep, want[1000:2000])
    keep[:] = 0
