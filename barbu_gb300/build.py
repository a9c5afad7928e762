"""Build the hair-simulation library in tree.

barbu_gb300/csrc/*.cu -> barbu_gb300/lib/libhairsim.so, for sm_103a only, and
the binding's call module, csrc/hs_pycalls.c -> barbu_gb300/_hscalls<suffix>,
the suffix of this interpreter (its ABI).
One nvcc process per translation unit, in parallel, then one link. Host code
is compiled without floating-point contraction so host-side parameter
arithmetic rounds like the device's.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libhairsim.so")
CALLS = os.path.join(HERE, "_hscalls" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
ARCH = ["-gencode", "arch=compute_103a,code=sm_103a"]


def nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return cand


def sources() -> list[str]:
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _compile(src: str, verbose_ptxas: bool) -> str:
    obj = os.path.join(BUILD, os.path.basename(src) + ".o")
    cmd = [nvcc(), *ARCH, "-O3", "-lineinfo", "-std=c++17", "-fmad=false", "-prec-div=true", "-prec-sqrt=true",
           "-Xcompiler", "-fPIC,-fvisibility=hidden,-ffp-contract=off", "-I", os.path.join(ROOT, "include"),
           "-I", CSRC, "-c", src, "-o", obj]
    if verbose_ptxas:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
    if verbose_ptxas:
        sys.stderr.write(r.stderr)
    return obj


def build_calls() -> str | None:
    """The binding's call module, or None (and a line on stderr) where it cannot
    be compiled, without a C compiler or Python.h: the binding then makes every
    call through ctypes."""
    tmp = CALLS + ".tmp"
    cmd = [shutil.which("gcc") or "cc", "-O2", "-fPIC", "-shared", "-fvisibility=hidden", "-Wall", "-I",
           sysconfig.get_paths()["include"], os.path.join(CSRC, "hs_pycalls.c"), "-o", tmp]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        failed = None if r.returncode == 0 else (r.stderr.strip().splitlines() or ["compiler error"])[0]
    except OSError as e:
        failed = str(e)
    if failed is None:
        os.replace(tmp, CALLS)
        return CALLS
    sys.stderr.write(f"{os.path.basename(CALLS)} not built, calls go through ctypes: {failed}\n")
    if os.path.exists(CALLS):  # of older sources
        os.remove(CALLS)
    return None


def build(verbose_ptxas: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    os.makedirs(LIB_DIR, exist_ok=True)
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose_ptxas), srcs))
    tmp = LIB + ".tmp"
    cmd = [nvcc(), *ARCH, "-shared", "-o", tmp, *objs, "-lcudart_static", "-lrt", "-lpthread", "-ldl"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_calls()
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(verbose_ptxas="-v" in sys.argv))
