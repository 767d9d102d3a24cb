"""The host code between the entry points and the kernels, on a stand-in for the CUDA runtime (fake_cudart.cpp): what is launched, cleared
and awaited, in which order and on which stream."""
import os
import shutil
import subprocess

import pytest

from llm170_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["dec.cu", "moe.cu", "moe_host.cu", "repack.cu"]      # the rest is not called


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("host")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if shutil.which(nvcc) is None:
        pytest.skip("no nvcc")
    jobs = [(["-c", os.path.join(build.CSRC, s)], str(tmp / (s + ".o"))) for s in SOURCES]
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1"]
    commands = [[nvcc, *flags, *args, "-o", out] for args, out in jobs]
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(nvcc) or nvcc))), "include")
    jobs.append((None, str(tmp / "fake.o")))
    commands.append(["g++", "-std=c++17", "-O1", "-I" + include, "-c", os.path.join(HERE, "fake_cudart.cpp"), "-o", jobs[-1][1]])
    running = [subprocess.Popen(c, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True) for c in commands]
    for p in running:
        text = p.communicate()[0]
        assert p.returncode == 0, text
    exe = str(tmp / "host")
    subprocess.run(["g++", "-no-pie", "-Wl,--unresolved-symbols=ignore-all", "-z", "lazy", *[out for _, out in jobs], "-o", exe], check=True)

    def run(*args):
        out = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=60)
        assert out.returncode == 0, (out.returncode, out.stdout, out.stderr)
        return out.stdout.splitlines()

    return run


def _kernels(lines):
    return [ln.split()[1] for ln in lines if ln.startswith("kernel ")]


def test_expert_counts_are_clear_before_the_first_call_counts(host):
    lines = host("moe")
    assert lines.count("returned 0") == 2
    assert not [ln for ln in lines if ln.startswith("UNORDERED")], lines
    first_clear = next(i for i, ln in enumerate(lines) if ln.startswith("clear counts"))
    first_count = next(i for i, ln in enumerate(lines) if "moe_topk" in ln)
    assert first_clear < first_count


# a launch that fails ends the call with an error: nothing that would read its tables is launched, and no count is left for the next call
SORT = ["moe_topk", "moe_offsets", "moe_place_gather", "matmul", "matmul", "moe_combine"]
SMALL = ["moe_topk", "moe_route_small", "matmul", "matmul", "moe_combine"]


@pytest.mark.parametrize("tokens,chain,bad", [(256, SORT, i) for i in range(6)] + [(9, SMALL, i) for i in range(5)])
def test_a_failed_launch_ends_the_call(host, tokens, chain, bad):
    lines = host("moe", bad, tokens)
    at = next(i for i, ln in enumerate(lines) if ln.startswith("returned"))
    first, second = lines[:at], lines[at + 1:]
    assert lines[at] != "returned 0" and second[-1] == "returned 0"
    ran = _kernels(first)
    assert len(ran) == bad and all(c in k for c, k in zip(chain, ran)), ran
    ran = _kernels(second)
    assert len(ran) == len(chain) and all(c in k for c, k in zip(chain, ran)), ran
    if chain is SORT and bad < 2:
        refused = next(i for i, ln in enumerate(lines) if ln.startswith("refused"))
        assert lines[refused + 1] == "clear counts stream2"
    assert not [ln for ln in lines if ln.startswith("UNORDERED")]


@pytest.mark.parametrize("what,cleared", [("scratch", ["tickets stream2"]), ("status", ["status stream1", "tickets stream1"]),
                                          ("exchange", ["exchange stream1", "block stream1"]), ("timeline", ["block stream1"])])
def test_what_launches_count_on_is_clear_before_them(host, what, cleared):
    lines = host(what)
    assert [ln[len("clear "):] for ln in lines if ln.startswith("clear ")] == cleared
    assert not [ln for ln in lines if ln.startswith("UNORDERED")], lines
    assert _kernels(lines) == ["matmul"]


# what an upload learns about its scales comes with the repack: no pass, copy or wait of its own in groups of 128
@pytest.mark.parametrize("bf16", [0, 1])
def test_upload_of_128_channel_groups_waits_no_more_than_of_32(host, bf16):
    want = host("upload", -1, 32, bf16)
    assert want[-1] == "returned 0" and sum("repack_q_kernel" in k or "repack_s_kernel" in k for k in _kernels(want)) == 2
    assert host("upload", -1, 128, bf16) == want
