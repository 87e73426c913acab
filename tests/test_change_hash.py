"""The change-detection hash (csrc/change_hash.h) on the host: bit flips in one
word and in several, at every length of the tail and at the edges of the four
threads' slices."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from ray_tracing_gb300 import build as _build

SPLIT = 4 << 20
SOURCE = """
#include "change_hash.h"
extern "C" uint64_t words(const void* p, size_t n) { return rtgb::hash_words(rtgb::kHashSeed, p, n); }
extern "C" uint64_t bytes(const void* p, size_t n) { return rtgb::hash_bytes(rtgb::kHashSeed, p, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("change_hash")
    (d / "hash.cpp").write_text(SOURCE)
    subprocess.run(["g++", *_build.CXX_FLAGS, "-shared", "-I", str(_build.CSRC), str(d / "hash.cpp"), "-o",
                    str(d / "hash.so"), "-lpthread"], check=True)
    lib = C.CDLL(str(d / "hash.so"))
    for f in (lib.words, lib.bytes):
        f.restype, f.argtypes = C.c_uint64, [C.c_void_p, C.c_size_t]
    return lib


def _of(f, a):
    return f(a.ctypes.data, a.nbytes)


def test_every_bit_counts_at_every_length(lib):
    rng = np.random.default_rng(1)
    for n in range(1, 150):
        a = rng.integers(0, 256, n, dtype=np.uint8)
        seen = {_of(lib.words, a)}
        for i in range(n):
            for bit in (0, 3, 7):
                a[i] ^= 1 << bit
                seen.add(_of(lib.words, a))
                a[i] ^= 1 << bit
        distinct = len(seen)
        assert distinct == 1 + 3 * n, n


def test_sign_flips_do_not_cancel(lib):
    """Every pair and many larger sets of sign flips of a float array: spheres
    are 5 words, triangles 27, a lane takes every sixteenth pair."""
    rng = np.random.default_rng(2)
    a = rng.standard_normal(432).astype(np.float32).view(np.uint32)
    sign = np.uint32(0x80000000)
    seen, count = {_of(lib.words, a)}, 1
    for i in range(432):
        a[i] ^= sign
        for j in range(i + 1, 432):
            a[j] ^= sign
            seen.add(_of(lib.words, a))
            a[j] ^= sign
            count += 1
        a[i] ^= sign
    # both signs of a word one to six steps of a lane after a flipped high half, and the mirrored axes
    for i in range(1, 300, 2):
        for step in range(1, 7):
            b = a.copy()
            b[[i, i - 1 + 16 * step, i + 16 * step]] ^= sign
            seen.add(_of(lib.words, b))
            count += 1
    for stride in (3, 5, 9, 27):
        for start in range(stride):
            b = a.copy()
            b[start::stride] ^= sign
            seen.add(_of(lib.words, b))
            count += 1
    distinct = len(seen)
    assert distinct == count


@pytest.mark.parametrize("size", [SPLIT - 1, SPLIT, SPLIT + 1, SPLIT + 255, SPLIT + 256, 5000007])
def test_slices_of_a_large_array(lib, size):
    rng = np.random.default_rng(size)
    a = rng.integers(0, 256, size, dtype=np.uint8)
    base = _of(lib.bytes, a)
    assert all(_of(lib.bytes, a) == base for _ in range(3))
    part = size // 4 // 64 * 64
    places = sorted({p for edge in (0, part, 2 * part, 3 * part, size) for p in (edge - 1, edge, edge + 7) if 0 <= p < size})
    seen = {base}
    for p in places:
        a[p] ^= 0x80
        seen.add(_of(lib.bytes, a))
        a[p] ^= 0x80
    assert len(seen) == 1 + len(places)
    # the sign of a word's upper float in two slices
    for first, second in ((7, part + 7), (part + 7, 2 * part + 7), (2 * part + 7, 3 * part + 7)):
        a[[first, second]] ^= 0x80
        seen.add(_of(lib.bytes, a))
        a[[first, second]] ^= 0x80
    assert len(seen) == 4 + len(places)
