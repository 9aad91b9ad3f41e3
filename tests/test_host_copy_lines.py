"""Which copies of pageable memory are staged by several threads (hostcopy.h), on
the CPU with fake device memory: copies out to fresh pages from 4 MB on, copies in
from 8 MB, copies out to pages that are there from 20 MB."""
import os
import subprocess

import pytest

from conftest import ROOT

NATIVE = os.path.join(ROOT, "tests", "native")
MB = 1 << 20


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("hostcopy") / "hostcopy_lines")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(NATIVE, "fake_cuda"), "-o", exe,
                    os.path.join(NATIVE, "hostcopy_lines.cpp"), "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("at", [0, 16, 4095])
@pytest.mark.parametrize("way,pages,line,most", [("in", "warm", 8 * MB, 4), ("out", "warm", 20 * MB, 4),
                                                 ("out", "fresh", 4 * MB, 8)])
def test_threads_from_the_line_on(lines, way, pages, line, most, at):
    # the copying thread is one of them
    cores = os.cpu_count() or 1
    for nbytes, threads in ((line - 1, 0), (line, min(most, cores) - 1), (line + 3 * MB + 5, min(most, cores) - 1)):
        r = subprocess.run([lines, str(nbytes), way, pages, str(at)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout == "%d 1\n" % threads, (nbytes, r.returncode, r.stdout, r.stderr)
