"""Heavy rows whose Y free indices fit 32 bits (columns carried by the products)
and do not (ranks looked up in the column table), with kept bitmaps and with
marked windows, at the default, the smallest and the largest window, against
the FP64 oracle."""
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


def _pair(free, seed):
    rng = np.random.default_rng(seed)
    nc, ny, nx = 40, 60000, 900
    yi = [rng.integers(0, nc, ny)] + [np.minimum((rng.random(ny) ** 3 * d).astype(np.int64), d - 1) for d in free]
    y = np.unique(np.stack(yi), axis=1)
    x = np.stack([(rng.random(nx) ** 2 * 30).astype(np.int64), rng.integers(0, nc, nx)])
    Y = gb.CooTensor([nc] + list(free), y[:, rng.permutation(y.shape[1])].astype(np.uint64),
                     rng.standard_normal(y.shape[1]).astype(np.float32))
    X = gb.CooTensor([30, nc], x.astype(np.uint64), rng.standard_normal(nx).astype(np.float32))
    return X, Y


@pytest.mark.parametrize("free", [(50000,), (1 << 20, 1 << 12), (1 << 20, 1 << 14)])  # 16, 32 and 34 bits
@pytest.mark.parametrize("cap", [0, 256, 8192])
@pytest.mark.parametrize("kept", [True, False])
def test_heavy_columns(ctx, free, cap, kept):
    X, Y = _pair(free, len(free))
    ctx.set_tiles(0, cap)
    ctx.set_row_bitmaps(kept)
    try:
        r = gb.SpTC(X, Y, [1], [0], ctx=ctx)
    finally:
        ctx.set_tiles(0, 0)
        ctx.set_row_bitmaps(True)
    z = ob.sptc(X, Y, [1], [0])
    assert r.stats["heavy_rows"] > 10
    assert r.ir_nnz == z.ir_nnz and np.array_equal(r.keys, z.keys)
    value_bar.max_rel_err(r.vals, z.vals)
