"""The peel's grid barrier counts arrivals in 32 bits and never resets them: it
has to hold across the wrap, which a graph of tens of millions of peel rounds
(a path of 5.8e7 vertices) reaches.  The arithmetic is the kernel's own header,
run on the host; on the GPU every peel by the whole grid crosses the wrap, since
its counter starts 1000 arrivals before it."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host C++ compiler")
@pytest.mark.parametrize("blocks,first", [(148, 0), (148, 2**32 - 1000), (148, 2**32 - 148), (148, 2**31 - 500),
                                          (1, 2**32 - 2), (132, 2**32 - 7)])
def test_barrier_holds_across_the_wrap(tmp_path, blocks, first):
    exe = str(tmp_path / "barrier_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", f"-I{os.path.join(ROOT, 'rdmce_b200', 'csrc')}",
                    os.path.join(ROOT, "tests", "cpp", "barrier_check.cc"), "-o", exe], check=True, timeout=300)
    r = subprocess.run([exe, str(blocks), str(first), "40"], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert "BARRIER OK" in r.stdout
