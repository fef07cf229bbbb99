"""Light rows whose products underflow: an output that is zero is +0, as the
accumulators of the longer rows leave it, whatever the products' signs."""
import numpy as np
import pytest

import gsparc_b200 as gb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shared", [False, True])  # columns of one contract key each, or of all of them
@pytest.mark.parametrize("keys,cols", [(2, 3), (5, 40), (100, 8), (200, 5)])
def test_underflow(keys, cols, shared):
    r = np.random.default_rng(keys)
    rows = 30
    x = np.stack([np.repeat(np.arange(rows), keys), np.tile(np.arange(keys), rows)]).astype(np.uint64)
    n = cols if shared else keys * cols
    y = np.stack([np.repeat(np.arange(keys), cols), np.arange(keys * cols) % n]).astype(np.uint64)
    xv = (r.standard_normal(rows * keys) * 1e-25).astype(np.float32)
    yv = (r.standard_normal(keys * cols) * 1e-25).astype(np.float32)
    yv[y[1] == 0] = 1e25  # a column that does not underflow
    with gb.Context(0, 1 << 30) as ctx:
        z = gb.SpTC(gb.CooTensor([rows, keys], x, xv), gb.CooTensor([keys, n], y, yv), [1], [0], ctx=ctx)
    assert z.stats["heavy_rows"] == 0 and z.nnz == rows * n
    v = z.vals.reshape(rows, n)
    assert np.all(v[:, 0] != 0) and np.all(v[:, 1:] == 0)
    assert not np.signbit(v[:, 1:]).any()
