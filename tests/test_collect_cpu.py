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


class _Driver:
    """Stands in for the library: which buffers are registered, a batch that does nothing."""

    def __init__(self):
        self.registered = set()

    def gsparc_host_pin(self, p, n):
        self.registered.add(p.value)
        return 0

    def gsparc_host_unpin(self, p):
        self.registered.remove(p.value)
        return 0

    def gsparc_sptc_batch(self, *a):
        return 0


class _Operand:
    handle = None


class _Ctx:
    handle = None

    def __init__(self):
        self._staging = api._StagingPool(2)


@pytest.mark.parametrize("bad", [(_Operand, _Operand, [0], [0, 1]), (_Operand, _Operand, [0]),
                                 (_Operand, None, [0], [0])])
def test_malformed_job_keeps_the_staging(monkeypatch, bad):
    drv = _Driver()
    monkeypatch.setattr(api, "lib", lambda: drv)
    ctx, good = _Ctx(), (_Operand, _Operand, [0], [0])
    for _ in range(3):
        with pytest.raises((ValueError, AttributeError)):
            api.sptc_batch(ctx, [good, bad])
    res, _ = api.sptc_batch(ctx, [good])
    assert res[0].keys.size == 0 and len(drv.registered) == 1 == len(ctx._staging._free)
    st = ctx._staging.take(api.STAGING_NNZ)
    assert st.pinned  # the pool still has one to give
    ctx._staging.give(st)
    ctx._staging.close()
    assert not drv.registered


def test_dropped_staging_is_unregistered(monkeypatch):
    drv = _Driver()
    monkeypatch.setattr(api, "lib", lambda: drv)
    pool = api._StagingPool(2)
    st = pool.take(api.STAGING_NNZ)
    assert drv.registered == {st.buf.ctypes.data}
    del st
    assert not drv.registered


@pytest.mark.parametrize("kw", [1, 2])
@pytest.mark.parametrize("pieces", [[8], [8, 1], [8] * 5 + [3], [8] * 300 + [1]])
def test_results_hold_no_spare_memory(monkeypatch, kw, pieces):
    monkeypatch.setattr(api, "SPARE_NNZ", 0)
    st = _Plain(kw * 8)
    col = api._Collect(st, kw)
    for k, n in enumerate(pieces):
        st.keys[:], st.vals[:] = k, k
        col.add(st.kp, st.vp, n, 8 * k)
    keys, vals = col.result()
    want = np.repeat(np.arange(len(pieces)), pieces)
    assert np.array_equal(vals, want) and np.array_equal(keys.reshape(-1), np.repeat(want, kw))
    for a in (keys, vals):
        assert (a if a.base is None else a.base).nbytes == a.nbytes
