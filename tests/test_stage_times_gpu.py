"""Stage times cover both operands: a large X beside a small Y shows in the
linearise and sort times, and so does a large Y beside a small X."""
import numpy as np
import pytest

import gsparc_b200 as gb

pytestmark = pytest.mark.gpu

LARGE, SMALL = 20000000, 2000


def _times(nx, ny):
    r = np.random.default_rng(nx)
    X = gb.CooTensor([1 << 24, 500], np.stack([r.integers(0, 1 << 24, nx), r.integers(0, 500, nx)]).astype(np.uint64),
                     r.random(nx, dtype=np.float32))
    Y = gb.CooTensor([500, 1 << 24], np.stack([r.integers(0, 500, ny), r.integers(0, 1 << 24, ny)]).astype(np.uint64),
                     r.random(ny, dtype=np.float32))
    with gb.Context(0, 16 << 30) as ctx:
        dx, dy = ctx.upload(X), ctx.upload(Y)
        st = [gb.sptc(ctx, dx, dy, [1], [0], sink="discard", max_chunk_nnz=1 << 26).stats for _ in range(4)][1:]
        dx.free()
        dy.free()
    for s in st:  # the stages follow one another
        parts = [s[k] for k in ("t_linearize_ms", "t_sort_ms", "t_match_ms", "t_plan_ms", "t_contract_ms")]
        assert min(parts) >= 0 and abs(sum(parts) - s["t_total_ms"]) < 1e-3 * len(parts) + 1e-4 * s["t_total_ms"]
    return [min(s[k] for s in st) for k in ("t_linearize_ms", "t_sort_ms")]


def test_large_operand_shows():
    # 2e7 nonzeros against 2e3: three passes and more of 2e7 pairs (0.3 ms and
    # up each way) against kernels of microseconds
    small = _times(SMALL, SMALL)
    for nx, ny in ((LARGE, SMALL), (SMALL, LARGE)):
        large = _times(nx, ny)
        assert large[0] > 2 * small[0] and large[1] > 2 * small[1], (nx, ny, large, small)
