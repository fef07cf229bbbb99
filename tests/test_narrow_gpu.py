"""Heavy rows over a narrow column space (at most 1024 distinct columns): column
counts around the words of marks and the limit, rows of one slice and of
several, runs of one entry, a Y that repeats coordinates, output chunks, plans
and batches, against the FP64 oracle."""
import numpy as np
import pytest

import gsparc_b200 as gb
import oracle_bind as ob
import value_bar

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = gb.Context(0)
    yield c
    c.close()


def _pair(ncols, rows, run, seed, dup=False, values="normal"):
    """rows: X nonzeros of every row; Y: 64 contract indices with about `run` entries each."""
    rng = np.random.default_rng(seed)
    nc = 64
    yc, yf = [], []
    for c in range(nc):
        n = max(1, min(ncols, int(rng.integers(1, 2 * run))))
        f = rng.integers(0, ncols, n) if dup else rng.choice(ncols, n, replace=False)
        yc += [c] * n
        yf += list(f)
    yc += [0] * ncols if not dup else []  # one full run: every column is there
    yf += list(range(ncols)) if not dup else []
    y = np.unique(np.array([yc, yf]), axis=1) if not dup else np.array([yc, yf])
    x = np.concatenate([np.stack([np.full(n, r), rng.integers(0, nc, n)]) for r, n in enumerate(rows)], axis=1)
    px, py = rng.permutation(x.shape[1]), rng.permutation(y.shape[1])
    X = gb.CooTensor([max(2, len(rows)), nc], x[:, px].astype(np.uint64), rng.standard_normal(x.shape[1]).astype(np.float32))
    Y = gb.CooTensor([nc, max(2, ncols)], y[:, py].astype(np.uint64), rng.standard_normal(y.shape[1]).astype(np.float32))
    return X, Y


def _same(r, z):
    assert r.ir_nnz == z.ir_nnz and r.nnz == z.nnz
    assert np.array_equal(r.keys, z.keys)
    value_bar.max_rel_err(r.vals, z.vals)


@pytest.mark.parametrize("dup", [False, True])
@pytest.mark.parametrize("ncols", [1, 2, 31, 32, 33, 300, 1023, 1024, 1025])
def test_columns(ctx, ncols, dup):
    X, Y = _pair(ncols, [5, 40, 700, 3000, 1, 9000], max(2, ncols // 8), ncols, dup)
    _same(gb.SpTC(X, Y, [1], [0], gb.ACCUM_DENSE, ctx=ctx), ob.sptc(X, Y, [1], [0]))
    _same(gb.SpTC(X, Y, [1], [0], ctx=ctx), ob.sptc(X, Y, [1], [0]))


@pytest.mark.parametrize("run", [1, 2, 40, 200])
def test_runs(ctx, run):
    X, Y = _pair(200, [4000] * 3 + [100000 // run], run, run)
    _same(gb.SpTC(X, Y, [1], [0], gb.ACCUM_DENSE, ctx=ctx), ob.sptc(X, Y, [1], [0]))


def test_chunks_plan_shards(ctx):
    import torch
    X, Y = _pair(300, [300] * 40 + [5000] * 5, 60, 9)
    z = ob.sptc(X, Y, [1], [0])
    _same(gb.SpTC(X, Y, [1], [0], ctx=ctx, max_chunk_nnz=1000), z)
    dx, dy = ctx.upload(X), ctx.upload(Y)
    parts = [gb.sptc(ctx, dx, dy, [1], [0], shard=k, nshards=3) for k in range(3)]
    assert np.array_equal(np.concatenate([p.keys for p in parts]), z.keys)
    p = gb.Plan(ctx, [(dx, dy, [1], [0])], max_chunk_nnz=2000)
    keys, vals = torch.empty(z.nnz, dtype=torch.int64, device="cuda"), torch.empty(z.nnz, device="cuda")
    for scale in (1.0, -2.0):
        dx.set_values((X.val * scale).astype(np.float32))
        p.refresh()
        for k in range(p.nchunks):
            f, n = p.chunk(k)
            p.execute(k, keys[f:f + n], vals[f:f + n])
        p.check()
        assert p.nchunks > 1 and np.array_equal(keys.cpu().numpy().view(np.uint64), z.keys)
        value_bar.max_rel_err(vals.cpu().numpy(), z.vals * scale)
    p.close()


def test_batch_with_wide_columns(ctx):
    shapes = [(300, [2000] * 4), (5000, [400] * 9), (17, [60000, 3]), (1024, [3000] * 2)]
    pairs = [_pair(nc, rows, 50, i, dup=i == 2) for i, (nc, rows) in enumerate(shapes)]
    jobs = [(ctx.upload(X), ctx.upload(Y), [1], [0], a) for (X, Y), a in zip(pairs, (0, 1, 1, -1))]
    got, _ = gb.sptc_batch(ctx, jobs)
    for r, (X, Y) in zip(got, pairs):
        _same(r, ob.sptc(X, Y, [1], [0]))
