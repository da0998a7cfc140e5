"""Kernels compiled for the host (tests/kernels/host_emu): one block's threads as fibers, run in
orders that the hardware allows but hardly ever takes.

walk_pipeline_check: the cooperative walk's pipeline with one warp late at every barrier must
walk as the reference's serial recurrence does, bit for bit, with all threads at the same
barriers: stopping at the edges of its sub-batches, at the last breakpoint (bounded or not),
with every variable fixed, with f'' at its lower limit, without a history, over several chunks,
in double and in float.

projgr_reads_check: the projected-gradient norm must not read a bound (nor x) that nbd says is
not there; those arrays lie on unreadable pages."""
import os
import re
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
KERNELS = os.path.join(HERE, "kernels")
CSRC = os.path.join(os.path.dirname(HERE), "lbfgsb-gpu_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def _between(text, first, after):
    a = text.index(first)
    return text[a:text.index(after, a)]


def _compile(tmp, check, opt="-O1"):
    exe = tmp / check
    subprocess.run(["g++", "-std=c++17", opt, "-ffp-contract=off", "-w", f"-I{tmp}",
                    f"-I{os.path.join(KERNELS, 'host_emu')}", f"-I{CSRC}",
                    os.path.join(KERNELS, check + ".cpp"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.fixture(scope="module")
def walk_exe(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("walk")
    s = _source("walk.cuh")
    body = (_between(s, "constexpr int kWalkThreads", "// One level of the radix select")
            + _between(s, "constexpr int kWalkRows", "// Lists the breakpoints with the whole grid"))
    # the shared-memory loads and stores in PTX are restated by the check
    body = re.sub(r"__device__ __forceinline__ void (lds4|sts4)\(.*?\n}\n", "", body, flags=re.S)
    (tmp / "walk_slice.cuh").write_text(
        "constexpr int kWalkChunk = 1024;\nnamespace lbfgsb_b200 {\n" + body + "\n}\n")
    return _compile(tmp, "walk_pipeline_check")


@pytest.mark.parametrize("real", ["f64", "f32"])
@pytest.mark.parametrize("what", ["stop", "end", "bounded", "fixed", "limit", "nohist", "chunks"])
def test_walk_pipeline(walk_exe, what, real):
    r = subprocess.run([walk_exe, real, what], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.fixture(scope="module")
def projgr_exe(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("projgr")
    body = _between(_source("noalloc.cu"), "constexpr int kNoAllocThreads",
                    "// Address of the scratch on the current device")
    (tmp / "projgr_slice.cuh").write_text("namespace lbfgsb_b200 {\n" + body + "\n}\n")
    return _compile(tmp, "projgr_reads_check", "-O0")  # -O1 drops loads that are not used


@pytest.mark.parametrize("per_thread", [1, 4, 16])
def test_projgr_reads_only_bounds_that_exist(projgr_exe, per_thread):
    r = subprocess.run([projgr_exe, str(per_thread)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
