"""Heavy rows by their number of runs: at and past the sizes where a row's runs
are searched by warps or by threads, dropped by one warp or by the CTA, and kept
in shared memory or not, with runs that give a window more than 1024 entries,
one entry or none, against the FP64 oracle."""
import numpy as np
import pytest

import gsparc_b200 as gb
import oracle_bind as ob
import value_bar

pytestmark = pytest.mark.gpu

NC, COLS = 520, 40000


@pytest.fixture(scope="module")
def ctx():
    c = gb.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def Y():
    rng = np.random.default_rng(7)
    ci, col = [], []
    for c in range(NC):
        if c % 5 == 0:  # neighbouring columns: one window takes thousands of them
            start = int(rng.integers(0, COLS - 3000))
            k = np.arange(start, start + 3000)
        elif c % 5 == 1:
            k = rng.integers(0, COLS, 1)
        else:
            k = np.unique(rng.integers(0, COLS, 300))
        ci.append(np.full(k.size, c))
        col.append(k)
    ci, col = np.concatenate(ci), np.concatenate(col)
    order = rng.permutation(ci.size)
    return gb.CooTensor([NC, COLS], np.stack([ci, col])[:, order].astype(np.uint64),
                        rng.standard_normal(ci.size).astype(np.float32))


@pytest.mark.parametrize("runs", [2, 16, 17, 32, 33, 64, 65, 128, 129, 511, 512, 513])
@pytest.mark.parametrize("cap", [0, 256])
def test_heavy_runs(ctx, Y, runs, cap):
    rng = np.random.default_rng(runs)
    rows = [np.sort(rng.permutation(NC)[:runs]) for _ in range(3)]
    rows[0][0] = 0  # a long run in every such row
    x = np.unique(np.stack([np.repeat(np.arange(3), runs), np.concatenate(rows)]), axis=1)
    X = gb.CooTensor([3, NC], x.astype(np.uint64), rng.standard_normal(x.shape[1]).astype(np.float32))
    ctx.set_tiles(0, cap)
    try:
        r = gb.SpTC(X, Y, [1], [0], ctx=ctx)
    finally:
        ctx.set_tiles(0, 0)
    z = ob.sptc(X, Y, [1], [0])
    assert r.stats["heavy_rows"] >= 1
    assert r.ir_nnz == z.ir_nnz and np.array_equal(r.keys, z.keys)
    value_bar.max_rel_err(r.vals, z.vals)
