"""Light rows (on-chip merge of a row's sorted runs) against the FP64 oracle at
the sizes where the kernel can go wrong: rows of 2 to 1024 runs, runs of one
entry, group counts that are no power of two, units filled to their capacity,
the larger unit of light_row_max = 2048, repeated columns and a Y that repeats
coordinates (single-run rows then take this path too)."""
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


def _problem(rows, seed, ncols, dup=False):
    """rows: list of run-length lists, one per output row; every run is a contract index of its own length."""
    rng = np.random.default_rng(seed)
    lens = sorted({n for r in rows for n in r})
    variants = 6  # Y runs of each length
    yc, yf = [], []
    for li, n in enumerate(lens):
        for v in range(variants):
            f = rng.choice(ncols, size=n, replace=False) if not dup else rng.integers(0, ncols, size=n)
            yc += [li * variants + v] * n
            yf += list(f)
    xr, xc = [], []
    for r, runs in enumerate(rows):
        for n in runs:
            # a row may meet the same Y run twice: every column of it repeats
            xr.append(r)
            xc.append(lens.index(n) * variants + int(rng.integers(0, variants)))
    x = np.array([xr, xc], np.uint64)
    y = np.array([yc, yf], np.uint64)
    px, py = rng.permutation(x.shape[1]), rng.permutation(y.shape[1])
    dims_c = max(len(lens) * variants, 2)
    X = gb.CooTensor([max(len(rows), 2), dims_c], x[:, px].copy(), rng.standard_normal(len(xr)).astype(np.float32))
    Y = gb.CooTensor([dims_c, ncols], y[:, py].copy(), rng.standard_normal(len(yc)).astype(np.float32))
    return X, Y


CASES = {
    "two_runs": [[1, 1], [2, 1], [31, 33], [512, 512], [1023, 1]] * 3,
    "odd_groups": [[3] * k for k in (2, 3, 5, 7, 9, 17, 31, 33, 63, 65, 127, 129, 255, 257)],
    "ones": [[1] * k for k in (2, 3, 4, 100, 511, 512, 513, 1023, 1024)],
    "full_units": [[256] * 4] * 9 + [[1024 - 7, 7]] * 5 + [[100, 1, 50, 2, 871]] * 4,
    "single": [[5], [1], [64], [1024]],
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("dup", [False, True])
@pytest.mark.parametrize("light_max", [0, 2048])
def test_light_rows(ctx, name, dup, light_max):
    rows = list(CASES[name])
    if light_max:
        rows += [[2048 - 3, 3], [2] * 1024, [1] * 2048, [1500, 548]]
    X, Y = _problem(rows, 7, 4096, dup)
    ctx.set_tiles(light_max, 0)
    try:
        r = gb.SpTC(X, Y, [1], [0], gb.ACCUM_ESC, ctx=ctx)
    finally:
        ctx.set_tiles(0, 0)
    z = ob.sptc(X, Y, [1], [0])
    assert r.ir_nnz == z.ir_nnz and r.nnz == z.nnz
    assert np.array_equal(r.keys, z.keys)
    value_bar.max_rel_err(r.vals, z.vals)
    assert r.stats["heavy_rows"] == 0


def _interleaved(rows):
    """Light rows with single-run rows and a heavy row between them."""
    out = []
    for i, r in enumerate(rows):
        out += [r, [7 + i % 5]]
        if i % 37 == 11:
            out.append([900, 800])
    return out


def test_interleaved_chunks_and_plan(ctx):
    import torch
    X, Y = _problem(_interleaved([[60, 40], [5, 5, 5], [300, 200, 9], [1, 2]] * 40), 11, 5000)
    z = ob.sptc(X, Y, [1], [0])
    for chunk in (0, 3000, 20011):
        r = gb.SpTC(X, Y, [1], [0], ctx=ctx, max_chunk_nnz=chunk)
        assert r.ir_nnz == z.ir_nnz and np.array_equal(r.keys, z.keys)
        value_bar.max_rel_err(r.vals, z.vals)
    dx, dy = ctx.upload(X), ctx.upload(Y)
    p = gb.Plan(ctx, [(dx, dy, [1], [0])], max_chunk_nnz=3000)
    keys, vals = torch.empty(z.nnz, dtype=torch.int64, device="cuda"), torch.empty(z.nnz, device="cuda")
    p.refresh()
    for k in range(p.nchunks):
        f, n = p.chunk(k)
        p.execute(k, keys[f:f + n], vals[f:f + n])
    p.check()
    assert p.nchunks > 5 and np.array_equal(keys.cpu().numpy().view(np.uint64), z.keys)
    value_bar.max_rel_err(vals.cpu().numpy(), z.vals)
    p.close()


def test_without_scratch():
    X, Y = _problem([[512, 500]] * 500, 3, 3000)
    z = ob.sptc(X, Y, [1], [0])
    with gb.Context(0, 24 << 20) as small:  # 6 MB of light products do not fit an eighth
        r = gb.SpTC(X, Y, [1], [0], ctx=small)
        assert r.ir_nnz == z.ir_nnz and np.array_equal(r.keys, z.keys)
        value_bar.max_rel_err(r.vals, z.vals)


@pytest.mark.parametrize("extra", [(1 << 20) - 4096, 1 << 20])
def test_many_columns(ctx, extra):
    """Ranks above and below 2^20: entries of 64 and of 32 bits."""
    X, Y = _problem(CASES["odd_groups"], 5, 4096)
    ncols = 4096 + extra
    unused = Y.dims[0]
    far = np.stack([np.full(extra, unused), 4096 + np.arange(extra)]).astype(np.uint64)
    low = np.stack([np.full(4096, unused + 1), np.arange(4096)]).astype(np.uint64)
    # the matched runs get the highest columns: mirror the free mode
    idx = np.concatenate([Y.idx, far, low], axis=1)
    idx[1] = ncols - 1 - idx[1]
    val = np.concatenate([Y.val, np.ones(extra + 4096, np.float32)])
    Y2 = gb.CooTensor([unused + 2, ncols], idx, val)
    X2 = gb.CooTensor([X.dims[0], unused + 2], X.idx, X.val)
    r = gb.SpTC(X2, Y2, [1], [0], ctx=ctx)
    z = ob.sptc(X2, Y2, [1], [0])
    assert r.ir_nnz == z.ir_nnz and np.array_equal(r.keys, z.keys)
    value_bar.max_rel_err(r.vals, z.vals)
