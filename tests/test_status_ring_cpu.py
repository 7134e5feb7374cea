"""The status words' book-keeping (csrc/fmb_status_ring.h) on the host: calls of several threads, words in any order."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_status_ring(tmp_path):
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "ring")
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", os.path.join(ROOT, "tests", "native", "status_ring_test.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
