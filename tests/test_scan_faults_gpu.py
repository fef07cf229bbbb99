"""A prefix sum whose wait gave up after the planning was read back (its error
bit set from the host: nothing waits) fails the call that meets it with
EINTERNAL, and the next call is whole again."""
import numpy as np
import pytest

import gsparc_b200 as gb
from gsparc_b200 import CooTensor

pytestmark = pytest.mark.gpu

EINTERNAL = 7


@pytest.fixture(scope="module")
def ctx():
    c = gb.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def ops(ctx):
    rng = np.random.default_rng(5)
    x = np.stack([rng.integers(0, 40, 4000), rng.integers(0, 300, 4000)]).astype(np.uint64)
    y = np.stack([rng.integers(0, 300, 30000), rng.integers(0, 200, 30000)]).astype(np.uint64)
    X = ctx.upload(CooTensor([40, 300], x, rng.standard_normal(4000).astype(np.float32)))
    Y = ctx.upload(CooTensor([300, 200], y, rng.standard_normal(30000).astype(np.float32)))
    yield X, Y
    X.free()
    Y.free()


def _call(ctx, X, Y, form, chunk):
    if form == "plan":
        p = gb.Plan(ctx, [(X, Y, [1], [0])], max_chunk_nnz=chunk)
        n = p.total
        p.close()
        return n
    if form == "batch":
        return sum(r.nnz for r in gb.sptc_batch(ctx, [(X, Y, [1], [0])] * 3, sink="discard", max_chunk_nnz=chunk)[0])
    return gb.sptc(ctx, X, Y, [1], [0], sink="discard", max_chunk_nnz=chunk).nnz


@pytest.mark.parametrize("form", ["sptc", "batch", "plan"])
@pytest.mark.parametrize("which,chunk", [(1, 0), (1, 500), (2, 0), (2, 500), (3, 500)])
def test_late_scan(ctx, ops, form, which, chunk):
    X, Y = ops
    good = _call(ctx, X, Y, form, chunk)
    in_use = ctx.memory()["in_use"]
    ctx.inject_scan_failure(which)
    try:
        with pytest.raises(gb.GsparcError) as e:
            _call(ctx, X, Y, form, chunk)
    finally:
        ctx.inject_scan_failure(0)
    assert e.value.status == EINTERNAL
    assert ctx.memory()["in_use"] == in_use
    assert _call(ctx, X, Y, form, chunk) == good


def test_chunk_limits_make_chunks(ctx, ops):
    # the third injection needs the chunks' own unit order
    assert gb.sptc(ctx, *ops, [1], [0], sink="discard", max_chunk_nnz=500).stats["chunks"] > 3
