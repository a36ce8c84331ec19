"""The coarse operator's index arithmetic (csrc/coarse_index.h) at its limits, on the host: up to
1024 planes of aggregates along one axis (the bins an axis may have), and beyond."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nnpp-mg-implant-corrosion-3d_gb300", "csrc")
AGGREGATES = 3000  # the coarse space's largest


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("coarse_index") / "libcheck.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "coarse_index_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("planes", [1, 2, 3, 13, 14, 64, 127, 511, 512, 513, 517, 1023, 1024, 1028, 1545, 2048, 3000])
def test_growth_covers_every_plane_pair_once(check, planes):
    m = AGGREGATES // planes
    tiles = min(-(-m // 64), 4)  # 64 x 64 tiles of a plane's block
    most = ctypes.c_longlong(0)
    assert check.check_growth(planes, tiles, ctypes.byref(most)) == 0
    if planes >= 512:
        assert most.value > 65535  # past gridDim.y's and gridDim.z's limit, within gridDim.x's
