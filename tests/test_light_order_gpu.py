"""The order in which a light row adds its products: that of the contract keys,
whatever the order of the input, the jobs beside it in a batch, and the bits
that X is sorted by (from 4,096 nonzeros on by their free bits alone; the rows
are padded with unmatched nonzeros to both sides of that).  The sums cancel to a 1e-9th of their terms, so that another
order shows in the last bits; the values are compared bit for bit with the same
compensated sums in float32 on the CPU."""
import numpy as np
import pytest

import gsparc_b200 as gb

pytestmark = pytest.mark.gpu

SHAPES = [(45, 6), (33, 31), (3, 300), (64, 3), (65, 3), (127, 8), (128, 8), (1000, 1), (1024, 1)]  # contract keys, columns: products of a row


@pytest.fixture(scope="module")
def ctx():
    c = gb.Context(0)
    yield c
    c.close()


def _job(keys, cols, con, rows, unmatched, seed):
    """Every row has a nonzero at every one of `keys` contract keys and `unmatched`
    others; Y is all ones over the keys and columns."""
    r = np.random.default_rng(seed)
    perm = r.permutation(con)
    cs, others = np.sort(perm[:keys]), perm[keys:]
    big = (r.standard_normal((rows, keys // 2)) * 1e5).astype(np.float32)
    v = np.concatenate([big, -big, (r.standard_normal((rows, keys - 2 * (keys // 2))) * 1e-4).astype(np.float32)], 1)
    v[:, -1] += np.float32(1e-4)
    v = r.permuted(v, axis=1)
    x = [np.repeat(np.arange(rows), keys), np.tile(cs, rows)]
    xv = v.reshape(-1)
    if unmatched:
        x = [np.concatenate([x[0], np.repeat(np.arange(rows), unmatched)]),
             np.concatenate([x[1], r.choice(others, rows * unmatched)])]
        xv = np.concatenate([xv, r.standard_normal(rows * unmatched).astype(np.float32)])
    y = np.stack([np.repeat(cs, cols), np.tile(np.arange(cols), keys)]).astype(np.uint64)
    s, c = v[:, 0].copy(), np.zeros(rows, np.float32)
    for k in range(1, keys):
        t = s + v[:, k]
        b = t - s
        c += (s - (t - b)) + (v[:, k] - b)
        s = t
    X = gb.CooTensor([rows, con], np.stack(x).astype(np.uint64), xv)
    return X, gb.CooTensor([con, cols], y, np.ones(keys * cols, np.float32)), np.repeat(s + c, cols)


def _shuffled(X, seed):
    p = np.random.default_rng(seed).permutation(X.val.size)
    return gb.CooTensor(X.dims, X.idx[:, p].copy(), X.val[p].copy())


@pytest.mark.parametrize("unmatched", [0, 5000, 12000])
@pytest.mark.parametrize("keys,cols", SHAPES)
def test_input_order(ctx, keys, cols, unmatched):
    X, Y, want = _job(keys, cols, 1 << 14, 2, unmatched, keys)
    for seed in range(3):
        r = gb.SpTC(_shuffled(X, seed), Y, [1], [0], ctx=ctx)
        assert r.stats["heavy_rows"] == 0
        assert np.array_equal(r.vals, want)


@pytest.mark.parametrize("keys,cols", SHAPES)
def test_company(ctx, keys, cols):
    # contract keys of 12, 14, 17 and 6 bits, short and long rows
    jobs = [_job(keys, cols, 1 << 12, 40, 0, 1), _job(keys, cols, 1 << 14, 2, 12000, 2), _job(keys, cols, 1 << 17, 7, 0, 3),
            _job(min(keys, 60), cols, 1 << 6, 9, 0, 4)]
    for pick in ([0, 1, 2, 3], [1, 1], [3, 1], [2, 0]):
        dev = [(ctx.upload(_shuffled(jobs[k][0], k)), ctx.upload(jobs[k][1])) for k in pick]
        got, _ = gb.sptc_batch(ctx, [(x, y, [1], [0]) for x, y in dev])
        for r, k in zip(got, pick):
            assert r.stats["heavy_rows"] == 0
            assert np.array_equal(r.vals, jobs[k][2])
        for x, y in dev:
            x.free()
            y.free()
