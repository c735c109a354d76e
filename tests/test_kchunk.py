"""The k chunk a context starts on (csrc/kchunk.h), over grids from a column of
four points to the largest sizes: the chunks of a launch are its grid.y (at most
65,535), and a grid few columns wide does not march in chunks of one or two
planes once its CTAs are several times the GPU's slots (each chunk starts with
six planes of its own)."""
import ctypes as C
import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cbns3d_cuda_b200" / "csrc"
GXX = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
SOURCE = """
#include "kchunk.h"
extern "C" int start(int IM, int JM, int KM, int ntiles, int fp32) {
  return cbns::kchunk_start(IM, JM, KM, ntiles, 148, fp32 != 0);
}
"""


@pytest.fixture(scope="module")
def start(tmp_path_factory):
    if not GXX:
        pytest.skip("compiles csrc/kchunk.h with g++, which is not here")
    d = tmp_path_factory.mktemp("kchunk")
    (d / "k.cpp").write_text(SOURCE)
    subprocess.run([GXX, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), "-o", str(d / "k.so"), str(d / "k.cpp")],
                   check=True, capture_output=True)
    return C.CDLL(str(d / "k.so")).start


@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("IM", [4, 5, 8, 18, 64, 300])
def test_chunk_of_every_size(start, IM, fp32):
    slots = 148 * (3 if fp32 else 2)
    for JM in (4, 6, 12, 17, 47, 300):
        tiles = -(-(IM - 2) // 16) * -(-(JM - 2) // 15)
        for KM in (4, 5, 9, 18, 45, 130, 700, 5000, 20000, 66000, 200000, 600000, 2000000, 6000000):
            if (IM + 4) * (JM + 4) * (KM + 4) * 5 > 2e9:
                break
            kc = start(IM, JM, KM, tiles, fp32)
            chunks = -(-(KM - 2) // kc)
            assert 1 <= kc <= KM - 2 and chunks <= 65535, (IM, JM, KM, kc)
            if kc <= 2:
                assert tiles * chunks <= 6 * slots, (IM, JM, KM, kc)
