"""How a batch of rays is dealt out to warps and blocks (csrc/deal.h), on the
CPU: every ray once, for batches up to the largest 32-bit count."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include "deal.h"
extern "C" uint32_t chunk(uint32_t n, uint32_t w, uint32_t most) { return gprt::deal_chunk(n, w, most); }
extern "C" uint32_t at(uint32_t n, uint64_t k) { return gprt::deal_at(n, k); }
// rays dealt to all blocks of `threads` threads, and the steps the first block took
extern "C" uint64_t blocks(uint32_t n, uint32_t grid, uint32_t threads, uint64_t* steps) {
  uint64_t rays = 0;
  *steps = 0;
  for (uint32_t b = 0; b < grid; b++)
    gprt::deal_blocks(n, b * threads, grid * threads, [&](uint64_t base) {
      rays += base + threads < n ? threads : n - base;
      *steps += b == 0;
    });
  return rays;
}
"""
WARPS, BLOCKS = 152 * 8 * 4, 152 * 8  # a full grid
SIZES = [1, 63, WARPS, 64 * WARPS + 1, 2 ** 31 - 1, 2 ** 31 + 5, 2 ** 32 - WARPS, 2 ** 32 - WARPS + 1, 2 ** 32 - 1]


@pytest.fixture(scope="module")
def deal(tmp_path_factory):
    d = tmp_path_factory.mktemp("deal")
    src, lib = d / "deal.cpp", d / "libdeal.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), str(src), "-o",
                    str(lib)], check=True)
    dll = C.CDLL(str(lib))
    dll.chunk.restype = dll.at.restype = C.c_uint32
    dll.at.argtypes = [C.c_uint32, C.c_uint64]
    dll.chunk.argtypes = [C.c_uint32] * 3
    dll.blocks.restype = C.c_uint64
    dll.blocks.argtypes = [C.c_uint32] * 3 + [C.POINTER(C.c_uint64)]
    return dll


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("warps", [4, WARPS])
def test_chunks_cover_the_batch(deal, n, warps):
    chunk = deal.chunk(n, warps, 64)
    assert 1 <= chunk <= 64
    assert chunk == 64 or warps * chunk >= n  # smaller chunks only when one round deals everything
    last = (n - 1) // chunk
    for k in {0, min(1, last), warps - 1, warps, last, last + 1}:
        assert deal.at(n, k * chunk) == min(n, k * chunk)
        assert deal.at(n, k * chunk + chunk) == min(n, k * chunk + chunk)


@pytest.mark.parametrize("n", SIZES)
def test_blocks_cover_the_batch(deal, n):
    steps = C.c_uint64()
    assert deal.blocks(n, BLOCKS, 128, C.byref(steps)) == n
    assert steps.value == -(-n // (BLOCKS * 128))
