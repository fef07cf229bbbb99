"""Planning kernels (run table, column table, rows, classes, units) against the
oracle at the sizes where a tile of 2048 items ends, with the column ranks from
presence bits (small Y free index spaces) and from the sort (large ones), alone
and in a batch of jobs of both kinds, whose common space takes the sort."""
import numpy as np
import pytest

import gsparc_b200 as gb
import oracle_bind as ob
import value_bar

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 2047, 2048, 2049, 6145]
FREE = [1, 2, 300, 70000, 1 << 27]  # 2^27: sorted


@pytest.fixture(scope="module")
def ctx():
    c = gb.Context(0)
    yield c
    c.close()


def _pair(nx, ny, free, seed):
    rng = np.random.default_rng(seed)
    rows, c = max(2, nx // 3), max(2, ny // 4)
    x = np.stack([rng.integers(0, rows, nx), rng.integers(0, c, nx)]).astype(np.uint64)
    y = np.stack([rng.integers(0, c, ny), rng.integers(0, free, ny)]).astype(np.uint64)
    y[1, 0] = free - 1
    return (gb.CooTensor([rows, c], x, rng.standard_normal(nx).astype(np.float32)),
            gb.CooTensor([c, free], y, rng.standard_normal(ny).astype(np.float32)))


def _same(r, z):
    assert r.ir_nnz == z.ir_nnz and r.nnz == z.nnz
    assert np.array_equal(r.keys, z.keys)
    value_bar.max_rel_err(r.vals, z.vals)


@pytest.mark.parametrize("free", FREE)
@pytest.mark.parametrize("n", SIZES)
def test_sizes(ctx, n, free):
    X, Y = _pair(n, SIZES[(SIZES.index(n) + FREE.index(free)) % len(SIZES)], free, n + free)
    c = max(X.dims[1], Y.dims[0])
    X.dims[1] = Y.dims[0] = c
    _same(gb.SpTC(X, Y, [1], [0], ctx=ctx), ob.sptc(X, Y, [1], [0]))


@pytest.mark.parametrize("frees", [[300, 1, 70000, 2, 33], [300, 1 << 27, 2]])
def test_batch(ctx, frees):
    jobs, want, keep = [], [], []
    for k, free in enumerate(frees):
        X, Y = _pair(SIZES[-1 - k], SIZES[3 + k % 4], free, k)
        X.dims[1] = Y.dims[0] = max(X.dims[1], Y.dims[0])
        want.append(ob.sptc(X, Y, [1], [0]))
        keep += [ctx.upload(X), ctx.upload(Y)]
        jobs.append((keep[-2], keep[-1], [1], [0]))
    got, _ = gb.sptc_batch(ctx, jobs)
    for r, z in zip(got, want):
        _same(r, z)


@pytest.mark.parametrize("nshards", [2, 5])
def test_shards(ctx, nshards):
    X, Y = _pair(6145, 2049, 300, 3)
    X.dims[1] = Y.dims[0] = max(X.dims[1], Y.dims[0])
    dx, dy = ctx.upload(X), ctx.upload(Y)
    z = ob.sptc(X, Y, [1], [0])
    parts = [gb.sptc(ctx, dx, dy, [1], [0], shard=k, nshards=nshards) for k in range(nshards)]
    assert np.array_equal(np.concatenate([p.keys for p in parts]), z.keys)
    value_bar.max_rel_err(np.concatenate([p.vals for p in parts]), z.vals)


@pytest.mark.parametrize("space", [2, 31, 32, 33, 5000, 1 << 28])  # 2^28: runs found by search
def test_contract_space(ctx, space):
    rng = np.random.default_rng(space)
    used = np.unique(np.concatenate([rng.integers(0, space, 900), [0, space - 1]]))
    x = np.stack([rng.integers(0, 500, 6000), rng.choice(used, 6000)]).astype(np.uint64)
    y = np.stack([rng.choice(used[::2], 3000), rng.integers(0, 400, 3000)]).astype(np.uint64)
    X = gb.CooTensor([500, space], x, rng.standard_normal(6000).astype(np.float32))
    Y = gb.CooTensor([space, 400], y, rng.standard_normal(3000).astype(np.float32))
    for sort in (0, 1):
        ctx.set_sort(sort)
        try:
            _same(gb.SpTC(X, Y, [1], [0], ctx=ctx), ob.sptc(X, Y, [1], [0]))
        finally:
            ctx.set_sort(0)
