"""Staged copies when the host fails them: no exception and no abort leaves
the copy (it is made by the callers of a C entry), what was copied is whole."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gpu-svo_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_failures_of_the_host(tmp_path):
    exe = str(tmp_path / "hostcopy_fake")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I/usr/local/cuda/include", "-I" + CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "hostcopy_fake.cpp"), os.path.join(CSRC, "svo_hostcopy.cpp"), "-ldl"],
                   check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, (p.returncode, p.stdout[-2000:], p.stderr[-2000:])
