"""In-tree build of libflashmoba_b200.so with nvcc for sm_100a (no torch headers involved) and of
_fmb_torch.so, the C++ host path of the PyTorch front end, with the host compiler.

    python flash_moba_b200/build.py [--force]

Objects go to flash_moba_b200/_build/, the libraries next to this file, so that the built
libraries travel with a snapshot of the source tree.
"""
import concurrent.futures
import importlib.metadata
import os
import re
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libflashmoba_b200.so")
TORCH_EXT = os.path.join(HERE, "_fmb_torch.so")
TORCH_SRC = os.path.join(CSRC, "fmb_torch.cpp")
TORCH_HDR = os.path.join(CSRC, "fmb_status_ring.h")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]
# --use_fast_math must not touch the CUDA-core validation engine or the combine kernels'
# exp/log: those files are built without it.
PRECISE = {"fmb_attn_simt.cu", "fmb_attn_common.cu", "fmb_gate.cu", "fmb_pool.cu"}


# Kernels that hand registers from some warps to others count on the launch's share per thread: (source, kernel, the
# constant in the source that names it).  A wrong hand-over would never return, so a compiler that allocates
# another number fails the build (and the launches check it once more).
REGISTERS = [("fmb_attn_tc.cu", "fwd_main_tc_kernel", "kFwdRegsLaunch"), ("fmb_attn_tc.cu", "bwd_main_tc_kernel", "kBwdRegsLaunch"),
             ("fmb_attn_tc_wide.cu", "bwd_wide_tc_kernel", "kBwRegsLaunch")]


def check_registers(src_name, source, log):
    """Raises if the compiler's report (-Xptxas -v) on `src_name` shows another number of registers than its text counts on."""
    for name, kernel, constant in REGISTERS:
        if name != src_name:
            continue
        want = int(re.search(constant + r" = (\d+)", source).group(1))
        got = [int(n) for entry, n in re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", log, flags=re.S)
               if kernel in entry]
        if not got or any(n != want for n in got):
            raise RuntimeError(f"{src_name}: {kernel} was built with {got} registers per thread, {constant} = {want} expected")


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    hdrs += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return max(os.path.getmtime(h) for h in hdrs)


def _compile(nvcc, src, obj, log):
    flags = [f for f in NVCC_FLAGS if not (f == "--use_fast_math" and os.path.basename(src) in PRECISE)]
    flags = flags + os.environ.get("FMB_EXTRA_NVCC_FLAGS", "").split()
    cmd = [nvcc] + flags + ["-I", INCLUDE, "-c", src, "-o", obj]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    with open(log, "w") as f:
        f.write(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout[-4000:]}")
    try:
        with open(src) as f:
            check_registers(os.path.basename(src), f.read(), r.stdout)
    except RuntimeError:
        os.remove(obj)                   # not taken for built by the next run
        raise
    return obj


def _build_torch_ext(log):
    """_fmb_torch.so: links against the torch libraries of the running interpreter and against
    libflashmoba_b200.so (found beside it at run time).  The shared libstdc++ is named: a compiler that has
    only the static one would give the extension a second copy, whose streams (a number in a TORCH_CHECK message) crash
    when they meet those of torch's."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    torch_lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_fmb_torch"]
    for d in cpp_extension.include_paths() + [sysconfig.get_path("include"), os.path.join(cuda, "include")]:
        cmd += ["-isystem", d]
    cmd += [TORCH_SRC, "-o", TORCH_EXT, "-L", HERE, "-lflashmoba_b200", "-L", torch_lib, "-ltorch_python", "-ltorch",
            "-ltorch_cpu", "-lc10", "-lc10_cuda", "-L", os.path.join(cuda, "lib64"), "-lcudart", "-l:libstdc++.so.6", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    with open(log, "w") as f:
        f.write(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        raise RuntimeError("g++ failed on fmb_torch.cpp:\n" + r.stdout[-4000:])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is out of date and link the shared library; returns its path."""
    nvcc = _nvcc()
    os.makedirs(BUILD, exist_ok=True)
    dep_t = _deps_mtime()
    jobs, objs = [], []
    for s in _sources():
        src = os.path.join(CSRC, s)
        obj = os.path.join(BUILD, s[:-3] + ".o")
        objs.append(obj)
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), dep_t):
            jobs.append((src, obj, os.path.join(BUILD, s[:-3] + ".log")))
    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for fut in [ex.submit(_compile, nvcc, *j) for j in jobs]:
                o = fut.result()
                if verbose:
                    print("compiled", os.path.basename(o))
    if jobs or not os.path.exists(LIB):
        cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout[-4000:])
        if verbose:
            print("linked", LIB)
    header_t = max(os.path.getmtime(f) for f in [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)] + [TORCH_HDR])
    # the extension holds the layouts of the torch it was compiled against
    made_for, stamp = f"{sys.version} torch {importlib.metadata.version('torch')}", os.path.join(BUILD, "fmb_torch.made_for")
    fits = os.path.exists(stamp) and open(stamp).read() == made_for
    if force or not fits or not os.path.exists(TORCH_EXT) or os.path.getmtime(TORCH_EXT) < max(os.path.getmtime(TORCH_SRC), header_t):
        _build_torch_ext(os.path.join(BUILD, "fmb_torch.log"))
        with open(stamp, "w") as f:
            f.write(made_for)
        if verbose:
            print("linked", TORCH_EXT)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
