"""Host-sink results gathered from staging pieces (no GPU): one piece, ring
pieces that reuse the staging, pieces that land in place, two key words; the
staging pool hands every taker a buffer of its own and closes cleanly."""
import threading

import numpy as np
import pytest

from gsparc_b200 import api


class _Plain:
    def __init__(self, nnz):
        self.nnz = nnz
        self.keys, self.vals = np.zeros(nnz, np.uint64), np.zeros(nnz, np.float32)
        self.kp, self.vp = self.keys.ctypes.data, self.vals.ctypes.data


@pytest.mark.parametrize("kw", [1, 2])
@pytest.mark.parametrize("cap,total", [(8, 0), (8, 1), (8, 7), (8, 8), (8, 9), (8, 100), (64, 63)])
@pytest.mark.parametrize("in_place", [False, True])
def test_pieces(kw, cap, total, in_place):
    rng = np.random.default_rng(total)
    k = rng.integers(0, 1 << 60, kw * total).astype(np.uint64)
    v = rng.random(total, dtype=np.float32)
    if in_place:  # the whole result fits the caller's arrays; pieces of 5
        st, step = _Plain(kw * max(cap, total)), 5
    else:
        st, step = _Plain(kw * cap), cap
    col = api._Collect(st, kw)
    for first in range(0, total, step):
        n = min(step, total - first)
        at = first if in_place else 0
        st.keys[kw * at: kw * (at + n)] = k[kw * first: kw * (first + n)]
        st.vals[at: at + n] = v[first: first + n]
        col.add(st.kp + 8 * kw * at, st.vp + 4 * at, n, first)
    st.keys[:] = 0  # results are copies
    keys, vals = col.result()
    assert keys.shape == ((total, 2) if kw == 2 else (total,)) and vals.shape == (total,)
    assert np.array_equal(keys.reshape(-1), k) and np.array_equal(vals, v)


def test_pool():
    pool = api._StagingPool(2)
    taken = []

    def take():
        taken.append(pool.take(api.STAGING_NNZ))
    ts = [threading.Thread(target=take) for _ in range(5)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert len({s.kp for s in taken}) == 5
    assert pool.take(97).nnz == 97
    for s in taken:
        s.keys[0] = 1
        pool.give(s)
    pool.close()
    pool.give(pool.take(api.STAGING_NNZ))
    assert not pool._free
