"""CPU: the length of the padded level arrays.  Passes over whole arrays (p = p + e) move
pairs of words from the first one on, so the allocated length has to be even, whatever the
block sizes; block bases are 3 mod 64, so the cells alone end on an odd word."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hydro3d_b200", "csrc")
HARNESS = """
#include "h3d_internal.h"
extern "C" void level_words(int n, const h3d_block_desc* d, int g, long long* words, long long* end) {
  const h3d::LevelGeom G = h3d::make_level_geom(std::vector<h3d_block_desc>(d, d + n), g, true);
  const h3d::BlkLev& B = G.bl.back();
  *words = G.n_elems;
  *end = B.off + B.sxy * (B.nz + 2);  // one past the last block's words
}
void h3d::set_call_error(const std::string&) {}
"""
W, P = 4, 5


@pytest.fixture(scope="module")
def level_words(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("level_words")
    (d / "level_words.cpp").write_text(HARNESS)
    so = str(d / "level_words.so")
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(d / "level_words.cpp"),
                    os.path.join(CSRC, "h3d_halo.cpp"), "-o", so], check=True)
    return C.CDLL(so).level_words


@pytest.mark.parametrize("nblk,n,ngrid", [
    ((1, 1, 1), (64, 64, 64), 4),
    ((2, 2, 2), (96, 96, 96), 6),
    ((2, 1, 2), (18, 10, 6), 2),     # odd coarse extents
    ((1, 3, 1), (5, 7, 9), 1),       # odd extents
    ((1, 1, 1), (2, 2, 2), 2),       # one cell on the coarsest level
])
def test_whole_array_pairs_stay_in_range(h3d, level_words, nblk, n, ngrid):
    blocks = h3d.topology.block_grid(nblk, n, [P, P, W, W, W, W], [1.0 / 32] * 3, ngrid)
    arr = (type(blocks[0]) * len(blocks))(*blocks)
    for g in range(1, ngrid + 1):
        words, end = C.c_longlong(), C.c_longlong()
        level_words(len(blocks), arr, g, C.byref(words), C.byref(end))
        assert words.value >= end.value
        last = 2 * ((words.value + 1) // 2 - 1)  # first word of the last pair of a pass over `words`
        assert last + 1 < words.value, (g, words.value)
