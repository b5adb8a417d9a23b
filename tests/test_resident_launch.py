"""The launch of the one-launch loops where the device has no room for a block
on every SM (tea_resident_launch.h, built for the host): it tries smaller grids
until one fits, and gives every other error back at once."""
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "tealeaf_opencl_gb300", "csrc")
TOO_LARGE = 720  # cudaErrorCooperativeLaunchTooLarge


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if cxx is None or not os.path.exists(nvcc):
        pytest.skip("no host C++ compiler or CUDA headers")
    out = str(tmp_path_factory.mktemp("launch") / "launch.so")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    # -Bsymbolic: its own cudaGetLastError, not one that the process has loaded
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", CSRC, "-I", include,
                    os.path.join(HERE, "native", "resident_launch_harness.cpp"), "-o", out],
                   check=True)
    return ctypes.CDLL(out)


def attempt(harness, blocks, room, other=0):
    tried = (ctypes.c_int * 512)()
    n, cleared = ctypes.c_int(), ctypes.c_int()
    e = harness.try_launch(blocks, room, other, tried, ctypes.byref(n), ctypes.byref(cleared))
    return e, list(tried)[:n.value], cleared.value


@pytest.mark.parametrize("blocks", [1, 2, 7, 8, 9, 76, 152])
def test_smaller_grids_until_one_fits(harness, blocks):
    for room in range(1, 160):
        e, tried, cleared = attempt(harness, blocks, room)
        assert e == 0 and tried[0] == blocks and 1 <= tried[-1] <= room
        assert tried == sorted(set(tried), reverse=True)
        assert cleared == len(tried) - 1  # no error left behind
        assert tried[-1] >= min(blocks, room) * 3 // 4  # and most of the room is used


def test_no_room_at_all_and_other_errors_are_returned(harness):
    e, tried, cleared = attempt(harness, 152, 0)
    assert e == TOO_LARGE and tried[-1] == 1 and cleared == len(tried) - 1
    assert attempt(harness, 152, 152, other=2) == (2, [152], 0)
