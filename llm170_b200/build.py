"""Builds ``libw4a16_b200.so`` in-tree with nvcc for sm_100a (cross-compiles without a GPU), and ``_native.so``, the
CPython binding of its forward calls (g++ against torch's headers)."""
from __future__ import annotations

import hashlib
import importlib.util
import os
import subprocess
import sys
import sysconfig
from importlib.metadata import version

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SO = os.path.join(HERE, "libw4a16_b200.so")
NATIVE_SO = os.path.join(HERE, "_native.so")
HASH = SO + ".srchash"
SOURCES = ["dec.cu", "repack.cu", "gemv.cu", "gemv_sk.cu", "gemv_rb.cu", "gemm_tc.cu", "gemm_ts.cu", "moe.cu", "moe_host.cu", "gemv_static.cu", "loader.cu", "head.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall", "--shared", "-cudart", "static",
]
NATIVE_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]


def source_hash() -> str:
    """sha256 over the CUDA sources, the public header and the compiler flags: what the binary is made from."""
    h = hashlib.sha256()
    files = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC))
    files.append(os.path.join(os.path.dirname(HERE), "include", "w4a16_b200.h"))
    for f in files:
        if f.endswith(".o"):
            continue
        h.update(os.path.basename(f).encode())
        with open(f, "rb") as fh:
            h.update(fh.read())
    h.update(" ".join(NVCC_FLAGS + SOURCES + NATIVE_FLAGS + [version("torch"), sys.version]).encode())
    return h.hexdigest()


def _stale() -> bool:
    """The binary is current when the hash recorded beside it equals the hash of the sources (file times do not
    survive a copy of the tree to another machine; contents do)."""
    if not all(os.path.exists(f) for f in (SO, NATIVE_SO, HASH)):
        return True
    with open(HASH) as fh:
        return fh.read().strip() != source_hash()


def _native_command() -> list[str]:
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    inc = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           "/usr/local/cuda/include", sysconfig.get_paths()["include"]]
    return (["g++"] + NATIVE_FLAGS + ["-I" + i for i in inc] + [os.path.join(CSRC, "native.cpp"), "-o", NATIVE_SO] +
            ["-L" + os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda",
             "-lc10"])


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return SO
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    flags = NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else [])
    # one process per source (the sources take from seconds to a minute each), then one link
    objs = [os.path.join(CSRC, os.path.splitext(s)[0] + ".o") for s in SOURCES]
    jobs = [("native.cpp", subprocess.Popen(_native_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True))]
    for src, obj in zip(SOURCES, objs):
        cmd = [nvcc] + [f for f in flags if f not in ("--shared",)] + ["-c", os.path.join(CSRC, src), "-o", obj]
        jobs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = []
    for what, p in jobs:
        out = p.communicate()[0]
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            failed.append(what)
    if failed:
        raise RuntimeError("failed building " + ", ".join(failed))
    r = subprocess.run([nvcc] + NVCC_FLAGS + objs + ["-o", SO], capture_output=True, text=True)
    if r.returncode != 0:
        sys.stderr.write(r.stdout + r.stderr)
        raise RuntimeError("nvcc failed linking libw4a16_b200.so")
    for obj in objs:
        os.remove(obj)
    with open(HASH, "w") as fh:
        fh.write(source_hash() + "\n")
    return SO


if __name__ == "__main__":
    build(force=True, verbose="-v" in sys.argv)
    print(SO)
