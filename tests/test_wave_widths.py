"""Local_Alignment on the device against the oracle's scalar restatement, on
requests chosen where a wave changes form: starting bands around the narrow
wave's 31 diagonals and around whole passes of 32, waves that widen past an
alignment's end, sequence ends that clip the window from either side, borders
that keep it from growing, tandem and identical sequences (long snakes, many
trace marks per step), and both strands.  Integers: equal."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

NATIVE = os.path.join(ROOT, "tests", "native")
WIDTHS = [1, 2, 19, 20, 21, 29, 30, 31, 32, 33, 63, 64, 65, 124, 129, 700]


def load_host():
    so, src = os.path.join(NATIVE, "libla_host.so"), os.path.join(NATIVE, "la_host.cpp")
    deps = [src, os.path.join(ROOT, "oracle", "scalar_align.cuh")] + [
        os.path.join(ROOT, "distributedpanga_b200", "csrc", f) for f in ("align_core.cuh", "align_spec.h")]
    if not os.path.exists(so) or any(os.path.getmtime(d) > os.path.getmtime(so) for d in deps):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-x", "c++", "-o", so, src], check=True)
    L = C.CDLL(so)
    L.la_host.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p,
                          C.c_int64]
    L.la_host.restype = C.c_int
    return L


def contigs(div: float):
    from distributedpanga_b200 import synth
    rng = np.random.default_rng(int(1000 * div) + 3)
    a = synth.random_bases(rng, 9037, 0.45)
    b = a if div == 0 else synth.indels(rng, synth.substitute(rng, a, div), div / 6,
                                        lambda k: rng.integers(1, 8, size=k), 0.45)
    unit = synth.random_bases(rng, 37, 0.5)
    t = synth.substitute(rng, np.resize(unit, 3001), 0.03)              # tandem array
    u = np.concatenate([synth.random_bases(rng, 1500, 0.5), a[2000:3100],  # homology inside unrelated sequence
                        synth.random_bases(rng, 1500, 0.5)])
    r = synth.revcomp(b)
    return [a, b, t, u, r, synth.random_bases(rng, 150, 0.5)]


def requests(cs, width: int):
    rng = np.random.default_rng(width)
    out = []

    def add(i, j, comp, x, y, w, lb=-1, hb=-1):
        la, lb_ = len(cs[i]), len(cs[j])
        lo = x - y - w // 2
        for e in (lo, lo + w - 1):      # the band's start points lie in the contigs
            px = (x + y + e) >> 1
            if not (0 <= px <= la and 0 <= px - e <= lb_):
                return
        out.append([i, j, comp, lo, lo + w - 1, x + y, lb, hb])

    n = len(cs[0])
    for x in (0, 1, width // 2 + 1, 400, 2500, n // 2, n - width - 2, n - 1, n):
        y = min(x, len(cs[1]))
        add(0, 1, 0, x, y, width)
        add(1, 0, 0, y, x, width)
    for x in (0, 500, 4000, n - 400):                      # the other strand
        add(0, 4, 1, x, min(x, len(cs[4])), width)
    for x in (300, 1100, 2600):                            # tandem: many diagonals go far
        add(2, 2, 0, x, x - 37 if x > 37 else x, width)
    for x in (2000, 2500, 3099):                           # ends in unrelated sequence on both sides
        add(0, 3, 0, x, x - 500, width)
    for lb, hb in ((0, 0), (0, -1), (-1, 3), (5, 40)):     # borders
        add(0, 1, 0, 3000, 3000, width, lb, hb)
    for _ in range(6):                                     # chance hits
        i, j = int(rng.integers(0, 6)), int(rng.integers(0, 6))
        add(i, j, int(rng.integers(0, 2)), int(rng.integers(0, len(cs[i]))), int(rng.integers(0, len(cs[j]))), width)
    return np.array(out, dtype=np.int32)


@pytest.mark.gpu
@pytest.mark.parametrize("div", [0.0, 0.01, 0.06, 0.2])
def test_waves_equal_the_scalar_aligner(dev, div):
    from distributedpanga_b200 import gdb
    L = load_host()
    cs = contigs(div)
    g = gdb.from_contigs(cs)
    dev.gdb_load(g)
    dev.set_freq(g.freq)
    req = np.concatenate([requests(cs, w) for w in WIDTHS])
    path, toff, tr = dev.local_alignment(req)
    want = np.zeros((len(req), 6), np.int32)
    wtr = np.zeros(len(req) * 400, np.uint16)
    seq = np.concatenate(cs).astype(np.uint8)
    ln = np.array([len(c) for c in cs], np.int64)
    freq = np.ascontiguousarray(g.freq, np.float32)
    assert L.la_host(seq.ctypes.data, len(cs), ln.ctypes.data, freq.ctypes.data, len(req), req.ctypes.data,
                     want.ctypes.data, wtr.ctypes.data, len(wtr)) == 0
    assert (path[:, 6] == 0).all()
    bad = np.flatnonzero((path[:, :6] != want).any(axis=1))
    assert len(bad) == 0, (req[bad[0]].tolist(), path[bad[0]].tolist(), want[bad[0]].tolist())
    assert np.array_equal(tr, wtr[: toff[-1]])
    assert (want[:, 1] - want[:, 0] > 800).sum() > 30      # many are real alignments
