"""What the build leaves behind: one C++ runtime in the process, an extension that fits the running torch, and the
register counts that the kernels' hand-over of registers counts on."""
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


def test_register_counts_are_checked_at_build_time():
    b = _build_module()
    source = open(os.path.join(PKG, "csrc", "fmb_attn_tc.cu")).read()
    log = "".join(f"ptxas info    : Compiling entry function '_ZN3fmb18{k}I6__halfLi64EEEvPi' for 'sm_100a'\nptxas info    : Used {n} "
                  "registers, used 1 barriers\n" for k, n in (("fwd_main_tc_kernel", 72), ("bwd_main_tc_kernel", 96), ("other", 40)))
    b.check_registers("fmb_attn_tc.cu", source, log)
    with pytest.raises(RuntimeError, match="fwd_main_tc_kernel was built with"):
        b.check_registers("fmb_attn_tc.cu", source, log.replace("Used 72", "Used 71"))
    with pytest.raises(RuntimeError, match="bwd_main_tc_kernel was built with"):
        b.check_registers("fmb_attn_tc.cu", source, log.replace("bwd_main", "bwd_side"))
    b.check_registers("fmb_gate.cu", "", "")
