"""The staged host copies (hostcopy.h) on the CPU with fake device memory: where
memory or a thread runs out while they start, the copy is made by the threads
that did start."""
import os
import subprocess

import pytest

from conftest import ROOT

NATIVE = os.path.join(ROOT, "tests", "native")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("hostcopy") / "hostcopy_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(NATIVE, "fake_cuda"), "-o", exe,
                    os.path.join(NATIVE, "hostcopy_check.cpp"), "-ldl"], check=True)
    return exe


@pytest.mark.parametrize("memory,thread", [(0, 0), (0, 1), (0, 3), (1, 0), (2, 0), (3, 0)])
def test_copies_with_the_threads_there_are(check, memory, thread):
    r = subprocess.run([check, str(memory), str(thread)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
