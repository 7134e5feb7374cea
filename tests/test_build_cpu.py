"""What the build leaves behind: one C++ runtime in the process, an extension that fits the running torch."""
import importlib.metadata
import importlib.util
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PKG = os.path.join(ROOT, "flash_moba_b200")


def _build_module():
    spec = importlib.util.spec_from_file_location("fmb_build", os.path.join(PKG, "build.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_extension_has_no_cxx_runtime_of_its_own():
    nm = shutil.which("nm")
    if nm is None:
        pytest.skip("no nm")
    for so in ("_fmb_torch.so", "libflashmoba_b200.so"):
        out = subprocess.run([nm, "-D", "--defined-only", os.path.join(PKG, so)], capture_output=True, text=True, check=True).stdout
        # the locale's identity is defined in the runtime itself, never in code that only uses it
        assert "_ZNKSt6locale2id5_M_idEv" not in out, so


def test_extension_is_rebuilt_for_another_torch(monkeypatch, tmp_path):
    b = _build_module()
    built = []
    monkeypatch.setattr(b, "BUILD", str(tmp_path))
    monkeypatch.setattr(b, "_sources", lambda: [])            # (nothing to compile: the host extension alone)
    monkeypatch.setattr(b, "_build_torch_ext", lambda log: built.append(log))
    version = [importlib.metadata.version("torch")]
    monkeypatch.setattr(b.importlib.metadata, "version", lambda name: version[0])
    b.build()
    b.build()
    assert len(built) == 1                                    # no stamp yet, then up to date
    version[0] = "0.0"
    b.build()
    assert len(built) == 2
