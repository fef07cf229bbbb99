"""The sort key that groups heavy rows by output chunk (chunkkey.h, the header
the kernel includes): chunks in order up to the most a call may have, windowed
rows before narrow ones, larger rows first."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gsparc_b200", "csrc")
SRC = '#include "chunkkey.h"\nextern "C" uint64_t key(uint64_t c, int n, uint64_t p) { return gs::heavy_chunk_key(c, n, p); }\n'
CHUNKS = [0, 1, (1 << 19) - 1, 1 << 19, (1 << 19) + 1, (1 << 20) - 1, 1 << 20, (1 << 20) + 40]
PRODUCTS = [1, 2, 1023, 1 << 31, 1 << 40]


@pytest.fixture(scope="module")
def key(tmp_path_factory):
    d = tmp_path_factory.mktemp("key")
    (d / "k.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", str(d / "k.so"), str(d / "k.cpp")],
                   check=True)
    f = ctypes.CDLL(str(d / "k.so")).key
    f.restype, f.argtypes = ctypes.c_uint64, [ctypes.c_uint64, ctypes.c_int, ctypes.c_uint64]
    return f


def test_order(key):
    want = [(c, n, p) for c in CHUNKS for n in (0, 1) for p in reversed(PRODUCTS)]
    keys = [key(*w) for w in want]
    assert keys == sorted(keys) and len(set(keys)) == len(keys)


@pytest.mark.parametrize("p", [1 << 42, 1 << 45, (1 << 63) + 5])
def test_huge_rows_stay_in_their_chunk(key, p):
    for c in CHUNKS[:-1]:
        assert key(c, 0, p) <= key(c, 0, 1) < key(c, 1, p) <= key(c, 1, 1) < key(c + 1, 0, p)
