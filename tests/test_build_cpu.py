"""What the build leaves behind: one C++ runtime in the process."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PKG = os.path.join(ROOT, "flash_moba_b200")


def test_extension_has_no_cxx_runtime_of_its_own():
    nm = shutil.which("nm")
    if nm is None:
        pytest.skip("no nm")
    for so in ("_fmb_torch.so", "libflashmoba_b200.so"):
        out = subprocess.run([nm, "-D", "--defined-only", os.path.join(PKG, so)], capture_output=True, text=True, check=True).stdout
        # the locale's identity is defined in the runtime itself, never in code that only uses it
        assert "_ZNKSt6locale2id5_M_idEv" not in out, so
