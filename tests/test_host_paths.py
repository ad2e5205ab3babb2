"""Host code of the library without a GPU: its object files linked with a host
stand-in of the CUDA runtime (host_cuda.h), which records launches and can
refuse memory.  Each case is a function of host_paths.cpp."""
import glob
import importlib.util
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "aces-ii_b200")
CUDA = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.isdir(CUDA):
        pytest.skip("g++ or the CUDA headers are not available")
    spec = importlib.util.spec_from_file_location("acesb200_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    build.build()
    out = str(tmp_path_factory.mktemp("host") / "host_paths")
    cmd = ["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(PKG, "csrc"), "-I", CUDA,
           os.path.join(HERE, "host_paths.cpp"), *sorted(glob.glob(os.path.join(build.BUILD, "*.o"))),
           "-lpthread", "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return out


@pytest.mark.parametrize("case", ["no_room_for_partials", "blocks_stay_with_their_call",
                                  "entry_points_wait", "first_launch_in_order",
                                  "failed_producer_leaves_zeros", "wide_tiles_need_plain_rows",
                                  "tile_choices_by_width", "empty_segments_are_refused"])
def test_host_path(exe, case):
    r = subprocess.run([exe, case], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
