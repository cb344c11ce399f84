"""The end of the bucket reduction (csrc/msm_reduce.cuh) run on the host with
its warp and block intrinsics emulated (tests/native/reduce_check.cpp): the
in-place rounds of every level against the levels of reduce_level_kernel, within
the shared memory that the launch asks for.  And the rule that says how many of
an accumulation's ranges hold entries."""
import os
import subprocess

import pytest

from conftest import NATIVE, PKG

CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
MIN_ENTRIES = 240  # ACC_MIN_ENTRIES


@pytest.fixture(scope="module")
def check():
    out = os.path.join(NATIVE, "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "reduce_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=bounds,null,alignment", "-fno-sanitize-recover=all", "-U_FORTIFY_SOURCE",
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(NATIVE, "emulation"), "-I" + CUDA_INCLUDE,
                    "-o", exe, os.path.join(NATIVE, "reduce_check.cpp")], check=True)

    def run(*args):
        done = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
        assert done.returncode == 0, done.stderr
        return done.stdout
    return run


@pytest.mark.parametrize("log_g", [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 15])
def test_tail(check, log_g):
    """From no level at all (one entry) over tails that start at level 0, with one
    and two rounds a level, to those behind earlier levels."""
    check(log_g)


@pytest.mark.parametrize("threads,ranges", [(75776, 75776), (75776, 151552), (128, 384)])
def test_active_ranges(check, threads, ranges):
    edge = ranges * MIN_ENTRIES
    for total in (0, 1, threads - 1, threads, threads + 1, ranges, edge - 1, edge, edge + 1, 1 << 36):
        most = threads if ranges > threads and total < edge else ranges
        active = int(check("ranges", total, ranges, threads))
        assert active == min(total, most), total
        assert active <= total  # every active range holds at least one entry
