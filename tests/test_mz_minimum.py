"""Slot values of minimizer tables at the smallest line count that the library
takes for each layout, where they fill the sector's slots: 31 bits of B8x32
sectors at 2^(2k-28) lines (k <= 27), 40 bits of B6x40 sectors at 2^(2k-37). Every
place of a k-mer stays clear of the sentinels, and no two k-mers share one."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

import corpus

REPO = Path(__file__).resolve().parents[1]
SOURCE = r"""
#include <cstdint>
#include "mz_core.cuh"
using namespace ibs;
// Both places of canonical codes (the second a copy of the first where a k-mer has one).
extern "C" void places(const uint64_t *codes, uint64_t n, uint32_t k, uint64_t nLines, uint64_t *bucket, uint64_t *slot)
{
    TableGeom g{};
    g.k = k;
    g.bits = 2 * k;
    g.nBuckets = nLines * mz::kSectorsPerLine;
    g.fpBits = 2 * mz::m_of(k) - (63 - __builtin_clzll(nLines));
    for (uint64_t i = 0; i < n; ++i)
        if (mz::placements(codes[i], g, bucket + 2 * i, slot + 2 * i) < 2) {
            bucket[2 * i + 1] = bucket[2 * i];
            slot[2 * i + 1] = slot[2 * i];
        }
}
"""


@pytest.fixture(scope="module")
def places(tmp_path_factory):
    d = tmp_path_factory.mktemp("shim")
    (d / "places.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(REPO / "gpu-ibs_b200" / "csrc"),
                    "-o", str(d / "places.so"), str(d / "places.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "places.so"))

    def call(codes, k, lines):
        b, s = np.zeros((len(codes), 2), np.uint64), np.zeros((len(codes), 2), np.uint64)
        lib.places(codes.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(len(codes)), ctypes.c_uint32(k),
                   ctypes.c_uint64(lines), b.ctypes.data_as(ctypes.c_void_p), s.ctypes.data_as(ctypes.c_void_p))
        return b, s
    return call


@pytest.mark.parametrize("k,bits", [(k, 31) for k in range(16, 28)] + [(k, 40) for k in range(16, 32)])
def test_slots_at_the_fewest_lines(places, k, bits):
    rng = np.random.default_rng(k + bits)
    lines = 1 << max(0, 2 * k - (28 if bits == 31 else 37))
    seq = rng.integers(0, 4, 60_000).astype(np.uint8)
    for unit in range(1, 9):  # equal smallest keys in one k-mer
        seq[3000 * unit:3000 * unit + 300] = np.tile(rng.integers(0, 4, unit), 300)[:300]
    for i in range(300):  # reverse palindromes
        half = rng.integers(0, 4, 20)
        seq[30_000 + 40 * i:30_040 + 40 * i] = np.concatenate([half, 3 - half[::-1]])
    codes = np.unique(np.concatenate([corpus.canonical_codes_np(bytes(np.frombuffer(b"ACGT", np.uint8)[seq]), k),
                                      corpus.random_codes(rng, 100_000, k)]))
    for n in (lines, lines + lines // 3 + 1):
        b, s = places(codes, k, n)
        assert (b < 4 * n).all() and (s < (1 << bits)).all()
        if bits == 31:
            assert s.max() < 0xFFFFFFFC
        two = (b[:, 0] != b[:, 1]) | (s[:, 0] != s[:, 1])
        line = np.concatenate([b[:, 0], b[two, 1]]) >> np.uint64(2)
        slot = np.concatenate([s[:, 0], s[two, 1]])
        assert len(np.unique(np.stack([line, slot], axis=1), axis=0)) == len(line)
