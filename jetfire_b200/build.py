"""Build ``libjetfire_b200.so`` in-tree with nvcc for sm_100a.

    python -m jetfire_b200.build [--force]

The library is plain C ABI (``include/jetfire_b200.h``); Python loads it with ctypes
(``jetfire_b200._lib``).  Beside it ``_host.so`` is built from ``csrc/torch_host.cpp``: the
tensor-taking half of ``ops.py``, a CPython extension against the installed torch and this
library.  The build is skipped when both are newer than every source file and ``_host.so`` was built against
the installed torch.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libjetfire_b200.so"
HOST = PKG / "_host.so"
SOURCES = ["pack_append.cu", "decode_scan.cu", "decode_scan_k4v4.cu", "topk_select.cu", "decode_finish.cu", "decode_static.cu",
           "jf_misc.cu", "mirror_append.cu", "mirror_correct.cu", "adapter_step.cu", "cpu_correction.cpp", "numa_place.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-O3", "-Xcompiler", "-pthread"]


def nvcc_path() -> str:
    cand = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(cand).exists():
        raise RuntimeError("nvcc not found; set NVCC or put it on PATH")
    return cand


def torch_stamp() -> str:
    """What ``_host.so`` is built against, as text inside it: torch's interfaces change with its version."""
    import torch
    return f"jetfire_b200._host for torch {torch.__version__}"


def up_to_date() -> bool:
    if not LIB.exists() or not HOST.exists() or (torch_stamp() + "\0").encode() not in HOST.read_bytes():
        return False
    t = min(LIB.stat().st_mtime, HOST.stat().st_mtime)
    deps = list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.cpp")) + list(CSRC.glob("*.h")) + \
        [PKG.parent / "include" / "jetfire_b200.h"]
    return all(d.stat().st_mtime <= t for d in deps)


def host_command(nvcc: str) -> list[str]:
    """The compile-and-link command of ``_host.so``; its libraries are found next to it at run time."""
    import sysconfig

    import torch
    base = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc).resolve().parents[1]
    inc = [base / "include", base / "include/torch/csrc/api/include", cuda / "include", sysconfig.get_paths()["include"]]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DJF_TORCH_STAMP="{torch_stamp()}"',
            *(f"-I{i}" for i in inc),
            str(CSRC / "torch_host.cpp"), "-o", str(HOST), f"-L{base / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu",
            "-ltorch", "-lc10_cuda", "-lc10", f"-L{PKG}", "-ljetfire_b200", "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and up_to_date():
        return LIB
    objdir = PKG / "build"
    objdir.mkdir(exist_ok=True)
    nvcc = nvcc_path()
    objs = []
    procs = []
    for src in SOURCES:
        obj = objdir / (src.rsplit(".", 1)[0] + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *os.environ.get("JF_NVCC_EXTRA", "").split(), "-c", str(CSRC / src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(str(obj))
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose and out.strip():
            print(out)
    link = [nvcc, "-shared", "-o", str(LIB), *objs, "-lpthread",
            "-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    r = subprocess.run(host_command(nvcc), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"building {HOST.name} failed:\n{r.stdout}")
    return LIB


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
