"""Builds ``libw4a16_b200.so`` in-tree with nvcc for sm_100a (cross-compiles without a GPU), and ``_native.so``, the
CPython binding of its forward calls (g++ against torch's headers).  The library needs nvcc alone: where torch is not
installed -- a build for a C or Rust host -- or with ``--library`` the binding is left out."""
from __future__ import annotations

import hashlib
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import tempfile
from importlib.metadata import version

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SO = os.path.join(HERE, "libw4a16_b200.so")
NATIVE_SO = os.path.join(HERE, "_native.so")
HASH = SO + ".srchash"
NATIVE_HASH = NATIVE_SO + ".srchash"
SOURCES = ["dec.cu", "repack.cu", "gemv.cu", "gemv_sk.cu", "gemv_rb.cu", "gemv_rg.cu", "gemv_rg_timeline.cu", "gemv_moe.cu", "gemv_moe_few.cu", "gemm_tc.cu", "gemm_ts.cu", "gemm_ts2.cu", "moe.cu", "moe_host.cu", "gemv_static.cu", "loader.cu", "head.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden,-Wall", "--shared", "-cudart", "static",
]
NATIVE_FLAGS = ["-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]


def _digest(files, *more: str) -> str:
    h = hashlib.sha256()
    for f in files:
        h.update(os.path.basename(f).encode())
        with open(f, "rb") as fh:
            h.update(fh.read())
    h.update(" ".join(more).encode())
    return h.hexdigest()


_PUBLIC_HEADER = os.path.join(os.path.dirname(HERE), "include", "w4a16_b200.h")


def source_hash() -> str:
    """sha256 over the CUDA sources, the public header and the compiler flags: what the library is made from."""
    files = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))
    return _digest(files + [_PUBLIC_HEADER], *NVCC_FLAGS, *SOURCES)


def native_hash() -> str:
    """The same for the binding, which also depends on the installed torch and Python."""
    return _digest([os.path.join(CSRC, "native.cpp"), _PUBLIC_HEADER], *NATIVE_FLAGS, version("torch"), sys.version)


def _current(so: str, record: str, want: str) -> bool:
    """A binary is current when the hash recorded beside it equals the hash of its sources (file times do not
    survive a copy of the tree to another machine; contents do)."""
    if not (os.path.exists(so) and os.path.exists(record)):
        return False
    with open(record) as fh:
        return fh.read().strip() == want


def _install(made: str, so: str, record: str, made_from: str) -> None:
    # renamed into place: a process that loads the library meanwhile sees the old file or the new one
    os.replace(made, so)
    with open(record, "w") as fh:
        fh.write(made_from + "\n")


def _nvcc() -> str:
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def _native_command(out: str) -> list[str]:
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(_nvcc()) or _nvcc())))   # .../bin/nvcc
    inc = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    return (["g++"] + NATIVE_FLAGS + ["-I" + i for i in inc] + [os.path.join(CSRC, "native.cpp"), "-o", out] +
            ["-L" + os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda",
             "-lc10"])


def build(force: bool = False, verbose: bool = False, native: bool = True) -> str:
    """Builds what is out of date (everything with ``force``).  ``native``: the binding too, where torch is installed."""
    native = native and importlib.util.find_spec("torch") is not None
    lib_from, native_from = source_hash(), native_hash() if native else ""
    lib_job = force or not _current(SO, HASH, lib_from)
    native_job = native and (force or not _current(NATIVE_SO, NATIVE_HASH, native_from))
    if not (lib_job or native_job):
        return SO
    nvcc = _nvcc()
    compile_flags = [f for f in NVCC_FLAGS if f != "--shared"] + (["-Xptxas", "-v"] if verbose else [])
    # beside the results, so that they can be renamed into place; one folder per build, so that two of them do not meet
    tmp = tempfile.mkdtemp(prefix=".build_", dir=os.path.dirname(SO))
    running = []

    def start(what: str, cmd: list[str]):
        running.append((what, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        return running[-1]

    def finish(jobs):
        failed = []
        for what, p in jobs:
            out = p.communicate()[0]
            if verbose or p.returncode != 0:
                sys.stderr.write(out)
            if p.returncode != 0:
                failed.append(what)
        if failed:
            raise RuntimeError("failed building " + ", ".join(failed))

    try:
        binding = os.path.join(tmp, os.path.basename(NATIVE_SO))
        binding_job = start("native.cpp", _native_command(binding)) if native_job else None
        if lib_job:
            # one process per source (the sources take from seconds to a minute each), then one link
            objs = [os.path.join(tmp, os.path.splitext(s)[0] + ".o") for s in SOURCES]
            finish([start(src, [nvcc] + compile_flags + ["-c", os.path.join(CSRC, src), "-o", obj])
                    for src, obj in zip(SOURCES, objs)])
            made = os.path.join(tmp, os.path.basename(SO))
            finish([start(os.path.basename(SO), [nvcc] + NVCC_FLAGS + objs + ["-o", made])])
            _install(made, SO, HASH, lib_from)
        if native_job:
            finish([binding_job])          # after the library: it stands even if the binding does not build
            _install(binding, NATIVE_SO, NATIVE_HASH, native_from)
    finally:
        for _, p in running:
            if p.poll() is None:
                p.kill()
                p.communicate()
        shutil.rmtree(tmp, ignore_errors=True)
    return SO


if __name__ == "__main__":
    build(force=True, verbose="-v" in sys.argv, native="--library" not in sys.argv)
    print(SO)
