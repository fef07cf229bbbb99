"""The run lookup table of a group of jobs (runtab.h, the header the kernels
include) built and read on the CPU: every contract key of every job finds the
run that a search for (job, key) finds, also where Y indices outside their
modes leave contract parts above the job's width."""
import ctypes
import os
import random
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gsparc_b200", "csrc")

SRC = r"""
#include "runtab.h"
#include <cstddef>
using namespace gs;
// runs: sorted (job << kby | contract part); job j has ncbits[j] contract bits
// and its words from word0[j].  bits/first: zero at entry.
extern "C" void build(const uint64_t *runs, size_t n, int kby, const int *ncbits, const uint64_t *word0,
                      uint32_t *bits, uint32_t *first) {
    const uint64_t km = kby >= 64 ? ~0ull : (1ull << kby) - 1;
    for (size_t r = 0; r < n; ++r) {
        const uint64_t j = kby >= 64 ? 0 : runs[r] >> kby, c = runs[r] & km;
        const bool same = r > 0 && (kby >= 64 ? 0 : runs[r - 1] >> kby) == j;
        const bool lead = !same || ((runs[r - 1] & km) >> 5) != (c >> 5);
        if (!run_in_table(c, ncbits[j])) continue;
        const uint64_t w = word0[j] + (c >> 5);
        bits[w] |= 1u << (c & 31);
        if (lead) first[w] = (uint32_t)r;
    }
}
extern "C" uint64_t find(const uint32_t *bits, const uint32_t *first, uint64_t word0, uint64_t c, uint64_t none) {
    return run_of_key(bits[word0 + (c >> 5)], first[word0 + (c >> 5)], c, none);
}
"""


@pytest.fixture(scope="module")
def tab(tmp_path_factory):
    d = tmp_path_factory.mktemp("runtab")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", str(d / "t.so"), str(d / "t.cpp")],
                   check=True)
    lib = ctypes.CDLL(str(d / "t.so"))
    lib.find.restype = ctypes.c_uint64
    lib.find.argtypes = [ctypes.c_void_p, ctypes.c_void_p] + [ctypes.c_uint64] * 3
    return lib


def check(tab, jobs, kby):
    """jobs: (contract bits, distinct contract parts of Y, in any order)."""
    runs = np.array(sorted((j << kby) | c for j, (_, cs) in enumerate(jobs) for c in cs), np.uint64)
    nb = np.array([b for b, _ in jobs], np.int32)
    words = [((1 << b) + 31) >> 5 for b, _ in jobs]
    word0 = np.concatenate([[0], np.cumsum(words)]).astype(np.uint64)
    bits, first = np.zeros(sum(words), np.uint32), np.zeros(sum(words), np.uint32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    tab.build(p(runs), ctypes.c_size_t(len(runs)), kby, p(nb), p(word0), p(bits), p(first))
    where = {int(k): r for r, k in enumerate(runs)}
    for j, (b, _) in enumerate(jobs):
        for c in range(1 << b):
            want = where.get((j << kby) | c, len(runs))
            assert tab.find(p(bits), p(first), int(word0[j]), c, len(runs)) == want, (j, c)


def test_out_of_range_index_stays_out(tab):
    # job 0: contract size 1000 (10 bits), indices 5 and 1031; job 1 follows
    check(tab, [(10, [5, 1031]), (12, list(range(0, 4096, 3)))], 20)
    # every key of the job has a run and one index lies a whole width above
    check(tab, [(8, list(range(256)) + [256]), (8, list(range(256)))], 14)


@pytest.mark.parametrize("seed", range(40))
def test_random_groups(tab, seed):
    r = random.Random(seed)
    kby = r.randrange(12, 20)
    jobs = []
    for _ in range(r.randrange(1, 6)):
        b = r.randrange(0, 11)
        cs = set(r.sample(range(1 << b), r.randrange(0, (1 << b) + 1)))
        if r.random() < 0.6:
            cs |= {r.randrange(1 << b, 1 << kby) for _ in range(r.randrange(1, 30))}
        jobs.append((b, sorted(cs)))
    check(tab, jobs, kby)
