"""A batched job whose Y has a contract index outside its mode, beside jobs of
wider keys: it fails alone, and the other jobs' results are the oracle's."""
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


def _job(rows, con, cols, nx, ny, seed):
    rng = np.random.default_rng(seed)
    x = np.stack([rng.integers(0, rows, nx), rng.integers(0, con, nx)]).astype(np.uint64)
    y = np.stack([rng.integers(0, con, ny), rng.integers(0, cols, ny)]).astype(np.uint64)
    return (gb.CooTensor([rows, con], x, rng.standard_normal(nx).astype(np.float32)),
            gb.CooTensor([con, cols], y, rng.standard_normal(ny).astype(np.float32)))


@pytest.mark.parametrize("over", [[256], [256, 261, 511], [287, 4095, 1 << 20]])
@pytest.mark.parametrize("bad_at", [0, 1, 2])
def test_contract_index_of_y(ctx, over, bad_at):
    # the bad one: every contract key has a run, rows over 64 columns (narrow);
    # the others: rows over 5,000 columns and over 300
    bad = _job(20, 256, 64, 4000, 9000, 1)
    bad[1].idx[0, : len(over)] = over
    good = [_job(50, 4096, 5000, 6000, 20000, 2), _job(30, 200, 300, 5000, 8000, 3)]
    pairs = good[:bad_at] + [bad] + good[bad_at:]
    dev = [(ctx.upload(X), ctx.upload(Y)) for X, Y in pairs]
    try:
        got, st = gb.sptc_batch(ctx, [(x, y, [1], [0]) for x, y in dev], raise_on_error=False)
        assert st["status"] == 1
        for k, (r, (X, Y)) in enumerate(zip(got, pairs)):
            if k == bad_at:
                assert r.stats["status"] == 1 and r.keys is None
                continue
            z = ob.sptc(X, Y, [1], [0])
            assert r.stats["status"] == 0 and np.array_equal(r.keys, z.keys)
            value_bar.max_rel_err(r.vals, z.vals)
    finally:
        for x, y in dev:
            x.free()
            y.free()
