"""Rows over a narrow column space whose runs lie around the length from which a
run is added by itself and around its step sizes, alone, in alternation with
short runs and with runs of one entry, against the FP64 oracle."""
import numpy as np
import pytest

import gsparc_b200 as gb
import oracle_bind as ob
import value_bar

pytestmark = pytest.mark.gpu

NCOLS = 300


@pytest.fixture(scope="module")
def ctx():
    c = gb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("lens", [(63,), (64,), (65,), (127, 128, 129), (64, 3), (1, 300, 31), (191, 63, 192, 64, 193, 1),
                                  (95, 96, 97, 2, 2, 2, 160, 33)])
def test_run_lengths(ctx, lens):
    rng = np.random.default_rng(sum(lens))
    nc = 70
    yc = np.concatenate([np.full(lens[c % len(lens)], c) for c in range(nc)])
    yf = np.concatenate([rng.permutation(NCOLS)[:lens[c % len(lens)]] for c in range(nc)])
    order = rng.permutation(yc.size)
    Y = gb.CooTensor([nc, NCOLS], np.stack([yc, yf])[:, order].astype(np.uint64),
                     rng.standard_normal(yc.size).astype(np.float32))
    xr = np.repeat(np.arange(4), (3, 33, 900, 6000))  # products from a few runs to many slices
    X = gb.CooTensor([4, nc], np.stack([xr, rng.integers(0, nc, xr.size)]).astype(np.uint64),
                     rng.standard_normal(xr.size).astype(np.float32))
    z = ob.sptc(X, Y, [1], [0])
    for accum in (gb.ACCUM_AUTO, gb.ACCUM_DENSE):
        r = gb.SpTC(X, Y, [1], [0], accum, ctx=ctx)
        assert r.ir_nnz == z.ir_nnz and np.array_equal(r.keys, z.keys)
        value_bar.max_rel_err(r.vals, z.vals)
