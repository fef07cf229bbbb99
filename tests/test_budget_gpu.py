"""Memory a call needs and a plan holds: a budget that takes the operands, the
planning and one long output row, and plans no larger than their rows."""
import numpy as np
import pytest

import gsparc_b200 as gb

pytestmark = pytest.mark.gpu


def _coo(dims, rng, *idx):
    return gb.CooTensor(dims, np.stack(idx).astype(np.uint64), rng.standard_normal(len(idx[0])).astype(np.float32))


def _rows_beside_a_long_one(rows, ny):
    """`rows` unmatched rows of one nonzero each, and one row that matches all of Y."""
    r = np.random.default_rng(1)
    X = _coo([rows + 1, 4000], r, np.concatenate([np.zeros(2000, np.int64), 1 + np.arange(rows)]),
             np.concatenate([np.arange(2000), 2000 + r.integers(0, 2000, rows)]))
    return X, _coo([4000, 1 << 21], r, r.integers(0, 2000, ny), np.arange(ny))


@pytest.mark.parametrize("rows,ny,mb", [(300000, 2000000, 231), (600000, 1000000, 184)])
def test_long_row_fits(rows, ny, mb):
    X, Y = _rows_beside_a_long_one(rows, ny)
    with gb.Context(0, mb * 1000000) as ctx:
        dx, dy = ctx.upload(X), ctx.upload(Y)
        assert gb.sptc(ctx, dx, dy, [1], [0], sink="discard").nnz == ny
        dx.free()
        dy.free()


def _plan_shapes():
    r = np.random.default_rng(2)
    n = 2000000
    yield (_coo([1000000, 4000], r, r.integers(0, 1000000, n), r.integers(0, 4000, n)),
           _coo([4000, 50], r, r.integers(0, 4000, 1000), r.integers(0, 50, 1000)), 78)  # single-run rows
    n = 1200000
    yield (_coo([400000, 3000], r, r.integers(0, 400000, n), r.integers(0, 3000, n)),
           _coo([3000, 700000], r, r.integers(0, 3000, 30000), r.integers(0, 700000, 30000)), 78)  # light rows
    n = 1000000
    yield (_coo([200, 4096], r, r.integers(0, 200, n), r.integers(0, 4096, n)),
           _coo([4096, 300], r, r.integers(0, 4096, 10000), r.integers(0, 300, 10000)), 86)  # narrow rows
    n = 2000000
    yield (_coo([300, 4000], r, r.integers(0, 300, 1000), r.integers(0, 4000, 1000)),
           _coo([4000, 1 << 22], r, r.integers(0, 4000, n), r.integers(0, 1 << 22, n)), 30)  # few products, a large Y
    yield (_coo([4, 2000], r, np.zeros(2000, np.int64), np.arange(2000)),
           _coo([2000, 1 << 21], r, r.integers(0, 2000, n), np.arange(n)), 29)  # one heavy row


@pytest.mark.parametrize("k", range(5))
def test_plan_holds(k):
    X, Y, per_nonzero = list(_plan_shapes())[k]
    with gb.Context(0, 4 << 30) as ctx:
        dx, dy = ctx.upload(X), ctx.upload(Y)
        before = ctx.memory()["in_use"]
        p = gb.Plan(ctx, [(dx, dy, [1], [0])])
        assert p.total > 0
        assert ctx.memory()["in_use"] - before <= per_nonzero * max(X.val.size, Y.val.size) + (1 << 20)
        p.close()
        dx.free()
        dy.free()
