"""Minimizer tables: what the scan kernel looks up is always a place that the
build files the k-mer under, for every k and on either strand, with repeats
(several smallest keys in one k-mer) and reverse-palindromic minimizers."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

REPO = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def places_shim(tmp_path_factory):
    out = tmp_path_factory.mktemp("shim") / "mz_places_shim.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(REPO / "gpu-ibs_b200" / "csrc"),
                    "-o", str(out), str(REPO / "tests" / "native" / "mz_places_shim.cpp")], check=True)
    lib = ctypes.CDLL(str(out))
    lib.mz_unfiled.restype = ctypes.c_uint64
    return lib


@pytest.mark.parametrize("k", range(16, 32))
def test_every_lookup_is_filed(places_shim, k):
    rng = np.random.default_rng(k)
    seq = rng.integers(0, 4, 60_000).astype(np.uint8)
    for unit in (1, 2, 3, 5, 7, 11):  # tandem repeats: equal m-mers inside one k-mer
        at = 1000 + 3000 * unit
        seq[at:at + 600] = np.tile(rng.integers(0, 4, unit).astype(np.uint8), 600)[:600]
    for i in range(400):  # sequences that equal their reverse complement
        half = rng.integers(0, 4, 24).astype(np.uint8)
        seq[40_000 + 48 * i:40_048 + 48 * i] = np.concatenate([half, 3 - half[::-1]])[:max(0, 60_000 - 40_000 - 48 * i)]
    nb = 4 << max(2 * k - (28 if k <= 27 else 37), 1)
    for s in (seq, np.ascontiguousarray(3 - seq[::-1])):
        bad = places_shim.mz_unfiled(s.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(len(s)), ctypes.c_uint32(k),
                                     ctypes.c_uint64(nb))
        assert bad == 0
