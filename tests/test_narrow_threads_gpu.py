"""Contractions onto narrow column spaces of different widths on two threads,
each with a context and a plan of its own: one needs more than 48 KB of shared
memory a CTA, the other less, and neither launch may depend on the other's."""
import threading

import numpy as np
import pytest
import torch

import gsparc_b200 as gb
import oracle_bind as ob
import value_bar

pytestmark = pytest.mark.gpu

LAUNCHES = 3000  # of each plan, one after another without waiting


def _pair(cols, seed):
    rng = np.random.default_rng(seed)
    x = np.stack([rng.integers(0, 20, 400), rng.integers(0, 60, 400)]).astype(np.uint64)
    y = np.stack([rng.integers(0, 60, 60000), rng.integers(0, cols, 60000)]).astype(np.uint64)
    return (gb.CooTensor([20, 60], x, rng.standard_normal(400).astype(np.float32)),
            gb.CooTensor([60, cols], y, rng.standard_normal(60000).astype(np.float32)))


def test_two_widths_at_once():
    pairs = [_pair(1000, 1), _pair(40, 2)]
    want = [ob.sptc(X, Y, [1], [0]) for X, Y in pairs]
    failed = []
    start = threading.Barrier(2)

    def work(k):
        X, Y = pairs[k]
        try:
            with gb.Context(0, 1 << 30) as ctx:
                dx, dy = ctx.upload(X), ctx.upload(Y)
                r = gb.sptc(ctx, dx, dy, [1], [0])
                assert r.stats["heavy_rows"] == 20  # all narrow
                plan = gb.Plan(ctx, [(dx, dy, [1], [0])])
                assert plan.nchunks == 1
                keys = torch.empty(plan.total, dtype=torch.int64, device="cuda")
                vals = torch.empty(plan.total, dtype=torch.float32, device="cuda")
                torch.cuda.synchronize()
                start.wait(60)
                for _ in range(LAUNCHES):
                    plan.execute(0, keys, vals)
                torch.cuda.synchronize()
                assert np.array_equal(keys.cpu().numpy().view(np.uint64), want[k].keys)
                value_bar.max_rel_err(vals.cpu().numpy(), want[k].vals)
                plan.close()
                dx.free()
                dy.free()
        except BaseException as e:
            failed.append((k, repr(e)))
            start.abort()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not failed
