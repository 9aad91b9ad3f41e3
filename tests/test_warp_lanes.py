"""The device's Local_Alignment run on the CPU, a call per warp on the lanes of
tests/native/warp_lanes.h, against the oracle's scalar restatement: the table
of shared extensions in cases whose calls must meet, and in a chosen order.
Integers: equal."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from test_wave_widths import NATIVE, load_host

EVEN = np.full(4, 0.25, np.float32)


@pytest.fixture(scope="module")
def lanes():
    so, src = os.path.join(NATIVE, "libwarp_host.so"), os.path.join(NATIVE, "warp_host.cpp")
    deps = [src, os.path.join(NATIVE, "warp_lanes.h")] + [
        os.path.join(ROOT, "distributedpanga_b200", "csrc", f)
        for f in ("align_core.cuh", "align_share.cuh", "align_spec.h", "align_warp.cuh")]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-U_FORTIFY_SOURCE", "-Wno-unknown-pragmas",
                        "-x", "c++", "-o", so, src], check=True)
    L = C.CDLL(so)
    vp, i64 = C.c_void_p, C.c_int64
    L.warp_host.argtypes = [vp, C.c_int, vp, vp, i64, vp, vp, i64, vp, vp, i64, vp]
    L.warp_host.restype = C.c_int
    return L


class Out:
    """Paths, traces, and what was shared."""

    def __init__(self, path, trace, stat):
        self.path, self.err, self.trace = path[:, :6], path[:, 6], trace
        self.entries, self.records = int(stat[0]), int(stat[1])
        self.none, self.head, self.pebble, self.misplaced = (int(v) for v in stat[2:6])
        self.open, self.done, self.joined, self.failed = (int(v) for v in stat[6:10])


def on_lanes(L, cs, req, blocks=True, share=True, turns=0, seed=1, entries=4096, records=4096, listed=1 << 20, cut=-1,
             cells=200_000, freq=EVEN):
    seq = np.concatenate(cs).astype(np.uint8)
    ln = np.array([len(c) for c in cs], np.int64)
    req = np.ascontiguousarray(req, np.int32)
    opt = np.array([blocks, share, turns, seed, entries, records, listed, cut], np.int64)
    path, stat = np.zeros((len(req), 7), np.int32), np.zeros(10, np.int64)
    tr = np.zeros(4 * len(req) * (int(ln.max()) // 100 + 4), np.uint16)
    assert L.warp_host(seq.ctypes.data, len(cs), ln.ctypes.data, freq.ctypes.data, len(req), req.ctypes.data,
                       opt.ctypes.data, cells, path.ctypes.data, tr.ctypes.data, len(tr), stat.ctypes.data) == 0
    return Out(path, tr[: path[:, 5].sum()], stat)


def scalar(cs, req, freq=EVEN):
    seq = np.concatenate(cs).astype(np.uint8)
    ln = np.array([len(c) for c in cs], np.int64)
    req = np.ascontiguousarray(req, np.int32)
    want = np.zeros((len(req), 6), np.int32)
    tr = np.zeros(4 * len(req) * (int(ln.max()) // 100 + 4), np.uint16)
    assert load_host().la_host(seq.ctypes.data, len(cs), ln.ctypes.data, freq.ctypes.data, len(req), req.ctypes.data,
                               want.ctypes.data, tr.ctypes.data, len(tr)) == 0
    return want, tr[: want[:, 5].sum()]


def check(out, want):
    bad = np.flatnonzero((out.path != want[0]).any(axis=1))
    assert len(bad) == 0, (bad.tolist(), out.path[bad[0]].tolist(), want[0][bad[0]].tolist())
    assert np.array_equal(out.trace, want[1])


@pytest.mark.parametrize("seed", [33, 34, 35, 39, 48, 49, 57])
def test_an_entry_names_a_pebble_from_after_its_line(lanes, seed):
    """A tandem array carries calls that start in it with a wide band past one
    line and close to the next; an extension then enters the first line late,
    joins another at the next, and no trace mark lies between."""
    rng = np.random.default_rng(seed)
    n = 30_000
    a = rng.integers(0, 4, n).astype(np.uint8)
    unit = rng.integers(0, 4, int(rng.integers(1, 4))).astype(np.uint8)
    lo, hi = int(rng.integers(2000, 7000)), int(rng.integers(16180, 16330))
    a[lo:hi] = np.resize(unit, hi - lo)
    if a[hi] == a[hi - len(unit)]:
        a[hi] = (a[hi] + 1) & 3
    b = a.copy()
    p = hi + int(rng.integers(1, 12))
    while p < 16_500:
        b[p] = (b[p] + 1 + rng.integers(0, 3)) & 3
        p += int(rng.integers(4, 26))
    for q in rng.integers(16_600, n, 8):
        b[q] = (b[q] + 1) & 3
    w = int(rng.integers(33, 60))
    req = [[0, 1, 0, -(w // 2), w - 1 - w // 2, 2 * x, -1, -1]
           for x in (int(rng.integers(13_500, 15_200)), lo + int(rng.integers(60, 1000)), lo + int(rng.integers(60, 1000)))]
    req.append([0, 1, 0, -1, 1, 2 * int(rng.integers(60, 1000)), -1, -1])
    out = on_lanes(lanes, [a, b], req)
    assert out.joined > 0 and out.open == 0
    assert out.misplaced == 0
    check(out, scalar([a, b], req))


@pytest.mark.parametrize("seed", [1, 2, 5, 8])
def test_a_failing_walk_closes_its_record(lanes, seed):
    """A call that owns entries joins another and then cannot walk its path
    back: it reports the error, and no record stays open for others to wait
    on."""
    from distributedpanga_b200 import synth
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 4, 40_000).astype(np.uint8)
    b = synth.indels(rng, synth.substitute(rng, a, 0.1), 0.05, lambda k: rng.integers(1, 4, size=k), 0.5)
    req = []
    for x in (12_500, 200, 2800, 1500):
        y = x * len(b) // len(a)
        req.append([0, 1, 0, x - y - 25, x - y + 25, x + y, -1, -1])
    out = on_lanes(lanes, [a, b], req, turns=300, seed=seed, cut=2, cells=400_000)
    assert out.err.tolist() == [0, 0, 0x102, 0]
    assert out.open == 0 and out.failed > 0
