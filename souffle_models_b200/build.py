"""In-tree build of the native library (nvcc, sm_100a only).

Plays the part of cpp/build_all_bindings.sh:1-21 and the per-model setup.py files of the
reference (cpp/bert/setup.py:11-46): one command builds everything the bindings need.
    python -m souffle_models_b200.build
"""
from __future__ import annotations

import functools
import os
import re
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libsouffle_b200.so")

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-shared", "-Xcompiler", "-fPIC", "--cudart", "shared",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the native library cannot be built")
    return exe


def _sources():
    return [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC))] + [
        os.path.join(HERE, "..", "include", "souffle_b200.h")]


def is_stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    return any(os.path.getmtime(s) > t for s in _sources())


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles csrc/souffle_b200.cu (which includes every kernel) into lib/libsouffle_b200.so."""
    if not force and not is_stale():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    cmd = [_nvcc(), *NVCC_FLAGS, "-o", LIB_PATH, os.path.join(CSRC, "souffle_b200.cu")]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if verbose:
        sys.stderr.write(res.stderr)
    return LIB_PATH


@functools.lru_cache(maxsize=None)
def _ptxas_log() -> str:
    """What `ptxas -v` prints for the library's one source file, compiled without linking."""
    import tempfile
    with tempfile.TemporaryDirectory() as tmp:
        cmd = [_nvcc(), "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-Xptxas", "-v", "-c",
               "-o", os.path.join(tmp, "x.o"), os.path.join(CSRC, "souffle_b200.cu")]
        res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    return res.stderr


def stack_frames() -> dict:
    """{function: largest stack frame in bytes} of the kernels and their out-of-line device functions."""
    out, func = {}, None
    for line in _ptxas_log().splitlines():
        m = re.search(r"Function properties for (\w+)", line)
        if m:
            func = m.group(1)
        m = re.search(r"(\d+) bytes stack frame", line)
        if m and func:
            out[func] = max(out.get(func, 0), int(m.group(1)))
    return out


def resource_usage() -> dict:
    """Compiles without linking and returns {function: (registers, spill_store_bytes, spill_load_bytes)} from
    `ptxas -v`: the kernels, and the out-of-line device functions they call (registers 0 for those: ptxas reports
    none per function).  The persistent kernels must not spill in their stages: a spilling epilogue cost 10-25%
    end to end."""
    out, name, func = {}, None, None
    spills = (0, 0)
    for line in _ptxas_log().splitlines():
        m = re.search(r"Compiling entry function '(\w+)'", line)
        if m:
            name = m.group(1)
        m = re.search(r"Function properties for (\w+)", line)
        if m:
            func = m.group(1)
        m = re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line)
        if m:
            spills = (int(m.group(1)), int(m.group(2)))
            if func != name:                      # an out-of-line device function of the kernel being compiled
                out.setdefault(func, (0,) + spills)
        m = re.search(r"Used (\d+) registers", line)
        if m and name:
            out[name] = (int(m.group(1)),) + spills
            name = None
    return out


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
