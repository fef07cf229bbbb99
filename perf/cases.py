"""Timed cases of the contraction engine, each one pass through the public Python interface.

The cases stand for what programs have the engine do: one contraction of
resident operands whose result stays on the GPU (device sink) or comes to the
host, from a few thousand nonzeros (where launches and latency count) to
outputs of many gigabytes; a narrow output under a large contract space (the
dense-accumulator workload); many mixed contractions in one batch or through
the server; a planned contraction replayed with new values; operands whose
keys need more than 64 bits; two contractions chained.  Shapes, sizes and
distributions are those of gsparc_b200/synth.py and of the tests: uniform or
bounded Zipf coordinates without repeats in random order, values U[0,1),
U[-1,1) or N(0,1).

Inputs are made on the GPU.  A case fixes the pattern of its nonzeros; the seed
turns every mode's indices by an offset of its own (the same for contracted
modes), shuffles the nonzeros and draws their values, so inputs of two seeds
differ in every coordinate and value while the result keeps its size.  `exact`
computes the same result in float64 with torch alone (join on the contract
key, sort by output key, segment sums).
"""
from __future__ import annotations

import math
import random
import zlib

import numpy as np
import torch

import gsparc_b200 as gb
from gsparc_b200 import api

DEV = "cuda" if torch.cuda.is_available() else "cpu"
PRODUCTS_AT_ONCE = 1 << 26  # products expanded together by the float64 join
CTX_BYTES = 72 << 30        # the program's engine memory, mapped once
SERVER_BYTES = 12 << 30

_kept = {}  # the program's one context and one server, as a user's program holds them


def _ctx():
    if "ctx" not in _kept:
        _kept["ctx"] = gb.Context(0, CTX_BYTES)
        _kept["ctx"].reserve()
    return _kept["ctx"]


def _server():
    if "server" not in _kept:
        _kept["server"] = gb.Server(0, SERVER_BYTES)
    return _kept["server"]


# ------------------------------------------------------------------ the cases
def _case(name, call, **kw):
    return dict(name=name, call=call, **kw)


ESC = dict(xdims="2482x2862x14036x17", ydims="", xdist="z1.1", ydist="", cx="2 3", cy="2 3", values="u01")
PLAIN = dict(xdims="1000x1000x1000", ydims="", xdist="u", ydist="", cx="2", cy="2", values="u01")
DENSE = dict(xdims="200x4096x4096", ydims="4096x4096x300", xdist="u z1.2 z1.2", ydist="z1.2 z1.2 u",
             cx="1 2", cy="0 1", values="normal")


def listed():
    return [
        # the smallest useful call, the size of the test fixtures: a sparse result brought to the host; pure latency
        _case("tiny_to_host", "sptc_host_sink", nx=2000, ny=0, accum=0, **PLAIN),
        # the one-call form of the README: host operands in, host result out
        _case("one_call_20k", "one_call", nx=20000, ny=0, accum=0, **PLAIN),
        # the plain workload at its own size: 1e7 products, hardly any of them added together
        _case("plain_100k", "sptc", nx=100000, ny=0, accum=0, **PLAIN),
        # the large-output workload at two sizes: skewed rows, sorted runs of thousands of entries
        _case("esc_155k", "sptc", nx=155000, ny=0, accum=0, **ESC),
        _case("esc_775k", "sptc", nx=775000, ny=0, accum=0, **ESC),
        # the dense-accumulator workload, small with the dense accumulator asked for, and at its own size
        _case("narrow_613k", "sptc", nx=613001, ny=500009, accum=1, **DENSE),
        _case("narrow_10m", "sptc", nx=10000000, ny=10000000, accum=0, **DENSE),
        # mixed contractions of orders 3 to 4 in one batch, results kept on the GPU
        _case("batch_24", "batch", jobs=24, shapes=3, nnz_lo=1000, nnz_hi=200000, orders_hi=4, most=40000000),
        # the same kind of requests (orders 3 to 5) through the server, results to the host
        _case("serve_16", "serve", jobs=16, shapes=5, nnz_lo=10000, nnz_hi=60000, orders_hi=5, most=400000),
        # coordinates planned once, values changing: refresh and every output chunk
        _case("plan_310k", "plan", nx=310000, ny=0, accum=0, **ESC),
        # operand keys over 64 bits (order 5), as the served workload has them
        _case("wide_400k", "sptc", nx=400003, ny=250007, accum=0, xdims="90000x800x100x70000x80000",
              ydims="70000x80000x60000", xdist="z1.2", ydist="z1.2", cx="3 4", cy="0 1", values="u11"),
        # two contractions, the first result staying on the GPU as an operand of the second
        _case("chain_40k", "chain", nx=40000, ny=40000, nt=20000, accum=0, xdims="3000x2000x5000",
              ydims="5000x400x600", tdims="600x1500", xdist="z1.1 z1.1 u", ydist="u z1.1 z1.1", cx="2", cy="0",
              values="u11"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["plain", "esc", "esc", "narrow", "mixed", "batch", "serve", "plan", "wide", "chain", "one_call"])
    accum = rng.choice([0, 0, 0, -1, 1])
    if kind == "plain":
        d = [_log(rng, 300, 3000) for _ in range(3)]
        nx = _log(rng, 2000, 150000)
        while nx * nx / d[2] > 1.5e7 or nx > 0.2 * d[0] * d[1] * d[2]:
            nx = int(nx * 0.8)
        return dict(call=rng.choice(["sptc", "sptc_host_sink"]) if nx < 30000 else "sptc", nx=nx, ny=0, accum=accum,
                    **dict(PLAIN, xdims="x".join(map(str, d))))
    if kind in ("esc", "plan"):
        return dict(call="plan" if kind == "plan" else "sptc", nx=_log(rng, 5000, 300000 if kind == "plan" else 600000),
                    ny=0, accum=rng.choice([0, 0, -1]), **ESC)
    if kind == "narrow":
        rows, cols, c = _log(rng, 20, 400), _log(rng, 20, 600), _log(rng, 1000, 5000)
        return dict(call="sptc", nx=_log(rng, 20000, 3000000), ny=_log(rng, 20000, 3000000), accum=accum,
                    **dict(DENSE, xdims="%dx%dx%d" % (rows, c, c), ydims="%dx%dx%d" % (c, c, cols)))
    if kind in ("batch", "serve"):
        n = rng.randrange(3, 17)
        hi = _log(rng, 20000, 60000) if kind == "serve" else _log(rng, 10000, 200000)
        return dict(call=kind, jobs=n, shapes=rng.randrange(1 << 20), nnz_lo=1000, nnz_hi=hi,
                    orders_hi=5 if kind == "serve" else 4, most=400000 if kind == "serve" else 20000000)
    if kind == "one_call":
        return dict(call="one_call", nx=_log(rng, 1000, 40000), ny=0, accum=0, **PLAIN)
    if kind == "wide":
        f = [_log(rng, 64, 100000) for _ in range(3)]
        while sum(_bits(v) for v in f) > 45:
            f = [_log(rng, 64, 100000) for _ in range(3)]
        c = [_log(rng, 40000, 100000) for _ in range(2)]
        s = "z%.2f" % rng.uniform(1.0, 1.25)
        return dict(call="sptc", nx=_log(rng, 10000, 300000), ny=_log(rng, 10000, 200000), accum=0,
                    xdims="x".join(map(str, f + c)), ydims="x".join(map(str, c + [_log(rng, 1000, 100000)])),
                    xdist=s, ydist=s, cx="3 4", cy="0 1", values="u11")
    if kind == "chain":
        return dict(call="chain", nx=_log(rng, 3000, 40000), ny=_log(rng, 3000, 40000), nt=_log(rng, 1000, 20000),
                    accum=0, xdims="%dx2000x5000" % _log(rng, 500, 3000), ydims="5000x400x600", tdims="600x1500",
                    xdist="z1.1 z1.1 u", ydist="u z1.1 z1.1", cx="2", cy="0", values="u11")
    # one contraction of the batched workload's shapes
    p = _mixed(random.Random(rng.randrange(1 << 30)), 4, 1000, 1000000, 3e8)
    return dict(call="sptc", nx=p["nx"], ny=p["ny"], accum=accum, xdims=p["xdims"], ydims=p["ydims"], xdist=p["xdist"],
                ydist=p["ydist"], cx=p["cx"], cy=p["cy"], values="u11")


def _bits(d):
    return int(d - 1).bit_length()


def _zipf_collision(dim, s):
    """Probability that two draws of a bounded Zipf(s) are the same."""
    w = np.arange(1, dim + 1, dtype=np.float64) ** -s
    w /= w.sum()
    return float((w * w).sum())


def _mixed(r, orders_hi, nnz_lo, nnz_hi, most):
    """One instance of the batched / served workloads (orders 3 to orders_hi, modes log-uniform 64..100k, 1 to 2
    contract modes, Zipf s in [1.0, 1.4]) with at most about `most` matched products."""
    while True:
        ox, oy, nc, s = r.randint(3, orders_hi), r.randint(3, orders_hi), r.randint(1, 2), r.uniform(1.0, 1.4)
        c = [_log(r, 64, 100000) for _ in range(nc)]
        fx = [_log(r, 64, 100000) for _ in range(ox - nc)]
        fy = [_log(r, 64, 100000) for _ in range(oy - nc)]
        if sum(map(_bits, fx + fy)) > 63 or max(sum(map(_bits, fx + c)), sum(map(_bits, fy + c))) > 90:
            continue
        if orders_hi < 5 and max(sum(map(_bits, fx + c)), sum(map(_bits, fy + c))) > 64:
            continue
        nx, ny = _log(r, nnz_lo, nnz_hi), _log(r, nnz_lo, nnz_hi)
        nx = int(min(nx, math.prod(fx + c) // 50))
        ny = int(min(ny, math.prod(fy + c) // 50))
        if nx * ny * math.prod(_zipf_collision(d, s) for d in c) > most:
            continue
        return dict(nx=nx, ny=ny, xdims="x".join(map(str, fx + c)), ydims="x".join(map(str, c + fy)), xdist="z%.3f" % s,
                    ydist="z%.3f" % s, cx=" ".join(str(ox - nc + i) for i in range(nc)),
                    cy=" ".join(map(str, range(nc))), values="u11", accum=0)


def _problems(case):
    """The contractions of one pass, each with its own shapes."""
    if case["call"] in ("batch", "serve"):
        r = random.Random(case["shapes"])
        return [_mixed(r, case["orders_hi"], case["nnz_lo"], case["nnz_hi"], case["most"]) for _ in range(case["jobs"])]
    return [case]


# ------------------------------------------------------------------ inputs
class _Coo:
    """Coordinates [order, nnz] (int64) and values (float32) on the GPU, as DeviceTensor takes them."""

    def __init__(self, dims, idx, val):
        self.dims, self.idx, self.val = dims, idx, val

    def to_host(self):
        return gb.CooTensor(list(self.dims), self.idx.cpu().numpy().astype(np.uint64), self.val.cpu().numpy())


def _ints(text, sep=" "):
    return [int(v) for v in text.split(sep)]


def _draw_mode(g, dim, dist, n):
    if dist == "u":
        return torch.randint(0, dim, (n,), generator=g, device=DEV)
    w = torch.arange(1, dim + 1, device=DEV, dtype=torch.float64) ** -float(dist[1:])
    cdf = torch.cumsum(w, 0)
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * cdf[-1]
    return torch.searchsorted(cdf, u, right=True).clamp_(max=dim - 1)


def _pack(idx, dims):
    """Coordinates in one or two words (low modes in the second)."""
    words, bits = [torch.zeros_like(idx[0])], 0
    for m, d in enumerate(dims):
        b = _bits(d)
        if bits + b > 62:
            words.append(torch.zeros_like(idx[0]))
            bits = 0
        words[-1] = (words[-1] << b) | idx[m]
        bits += b
    return words


def _distinct(idx, dims):
    """Positions of one entry of every distinct coordinate."""
    words = _pack(idx, dims)
    at = None
    for w in reversed(words):
        o = torch.sort(w if at is None else w[at], stable=True)[1]
        at = o if at is None else at[o]
    new = torch.zeros(at.numel(), dtype=torch.bool, device=idx.device)
    new[:1] = True
    for w in words:
        s = w[at]
        new[1:] |= s[1:] != s[:-1]
    return at[new]


def _pattern(g, dims_text, dist_text, nnz):
    dims = _ints(dims_text, "x")
    dist = dist_text.split()
    dist = dist * len(dims) if len(dist) == 1 else dist
    idx = torch.zeros((len(dims), 0), dtype=torch.int64, device=DEV)
    more = nnz
    while idx.shape[1] < nnz:
        n = int(more * 1.3) + 64
        idx = torch.cat([idx, torch.stack([_draw_mode(g, d, t, n) for d, t in zip(dims, dist)])], 1)
        idx = idx[:, _distinct(idx, dims)]
        more = max(2 * more, nnz // 2) if idx.shape[1] < nnz else 0
    idx = idx[:, torch.randperm(idx.shape[1], generator=g, device=DEV)[:nnz]]
    return _Coo(dims, idx, None)


def _seeded(g, t, values, turn):
    """The pattern with mode m turned by turn[m], its nonzeros in another order, and values."""
    nnz = t.idx.shape[1]
    order = torch.randperm(nnz, generator=g, device=DEV)
    idx = torch.stack([(t.idx[m][order] + turn[m]) % d for m, d in enumerate(t.dims)])
    if values == "normal":
        val = torch.randn(nnz, generator=g, device=DEV)
    else:
        val = torch.rand(nnz, generator=g, device=DEV)
        val = 2 * val - 1 if values == "u11" else val
    return _Coo(t.dims, idx, val)


def _inputs(case, seed):
    """[(X, Y, cx, cy)] of the pass, and the third operand of a chain."""
    said = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    g0 = torch.Generator(device=DEV).manual_seed(zlib.crc32(said.encode()))
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = random.Random(seed)
    pairs, T = [], None
    for p in _problems(case):
        cx, cy = _ints(p["cx"]), _ints(p["cy"])
        x = _pattern(g0, p["xdims"], p["xdist"], p["nx"])
        tx = [r.randrange(d) for d in x.dims]
        X = Y = _seeded(g, x, p["values"], tx)
        if p["ydims"]:
            y = _pattern(g0, p["ydims"], p["ydist"], p["ny"])
            ty = [r.randrange(d) for d in y.dims]
            for mx, my in zip(cx, cy):
                ty[my] = tx[mx]
            Y = _seeded(g, y, p["values"], ty)
        pairs.append((X, Y, cx, cy))
        if case["call"] == "chain":  # contracts Y's last mode with its own first one
            t = _pattern(g0, case["tdims"], "u z1.1", case["nt"])
            T = _seeded(g, t, case["values"], [ty[-1], r.randrange(t.dims[1])])
    return pairs, T


# ------------------------------------------------------------------ one pass
class _Request:
    """Operands of one served request; released with the state."""

    def __init__(self, srv, X, Y, cx, cy):
        self.x = srv.upload(X)
        self.y = self.x if Y is X else srv.upload(Y)
        self.cx, self.cy = cx, cy

    def __del__(self):
        for t in {id(self.x): self.x, id(self.y): self.y}.values():
            t.release()


def prepare(case, seed):
    pairs, T = _inputs(case, seed)
    call = case["call"]
    st = {"call": call, "accum": case.get("accum", 0)}
    if call == "one_call":  # a program that read its tensors from files
        X, Y, st["cx"], st["cy"] = pairs[0]
        st["x"] = X.to_host()
        st["y"] = st["x"] if Y is X else Y.to_host()
        st["ctx"] = _ctx()
        return st
    if call == "serve":
        st["srv"] = _server()
        st["requests"] = []
        for X, Y, cx, cy in pairs:
            hx = X.to_host()
            st["requests"].append(_Request(st["srv"], hx, hx if Y is X else Y.to_host(), cx, cy))
        return st
    st["ctx"] = ctx = _ctx()
    torch.cuda.synchronize()
    st["jobs"] = []
    for X, Y, cx, cy in pairs:
        dx = ctx.upload(X)
        st["jobs"].append((dx, dx if Y is X else ctx.upload(Y), cx, cy, st["accum"]))
        for d in st["jobs"][-1][:2]:
            d._keep = None  # the engine has its own copy
    if T is not None:
        st["t"] = ctx.upload(T)
    if call == "plan":
        st["plan"] = p = gb.Plan(ctx, st["jobs"])
        most = max([p.chunk(k)[1] for k in range(p.nchunks)] + [1])
        if p.nchunks == 1:
            st["keys"] = torch.empty(most, dtype=torch.int64, device=DEV)
            st["vals"] = torch.empty(most, dtype=torch.float32, device=DEV)
    return st


class _DeviceArray:
    """Device memory of the engine as an array that torch can read."""

    def __init__(self, ptr, n, kind):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": kind, "data": (ptr, False), "version": 3}


class _Collected:
    """A program's own copy of what a device sink delivers (chunks in order)."""

    def __init__(self):
        self.keys, self.vals = [], []

    def add(self, keys, vals, n):
        if n:
            self.keys.append(torch.as_tensor(_DeviceArray(keys, n, "<i8"), device=DEV).clone())
            self.vals.append(torch.as_tensor(_DeviceArray(vals, n, "<f4"), device=DEV).clone())

    def result(self):
        if len(self.keys) == 1:
            return {"keys": self.keys[0], "vals": self.vals[0]}
        if not self.keys:
            return {"keys": torch.empty(0, dtype=torch.int64, device=DEV), "vals": torch.empty(0, device=DEV)}
        return {"keys": torch.cat(self.keys), "vals": torch.cat(self.vals)}


def _host_result(r):
    return {"keys": r.keys.view(np.int64), "vals": r.vals}


def _to_device(ctx, X, Y, cx, cy, accum):
    out = _Collected()
    gb.sptc(ctx, X, Y, cx, cy, accum, sink="device", on_chunk=lambda k, v, n, first: out.add(k, v, n))
    return out.result()


def run(state):
    call = state["call"]
    if call == "one_call":
        return _host_result(gb.SpTC(state["x"], state["y"], state["cx"], state["cy"], state["accum"], ctx=state["ctx"]))
    if call == "serve":
        srv = state["srv"]
        tickets = [srv.submit(q.x, q.y, q.cx, q.cy) for q in state["requests"]]
        return [_host_result(srv.wait(t)) for t in tickets]
    ctx, jobs = state["ctx"], state["jobs"]
    if call == "sptc_host_sink":
        return _host_result(gb.sptc(ctx, *jobs[0]))
    if call == "sptc":
        return _to_device(ctx, *jobs[0])
    if call == "batch":
        outs = [_Collected() for _ in jobs]
        gb.sptc_batch(ctx, jobs, sink="device", on_chunk=lambda j, k, v, n, first: outs[j].add(k, v, n))
        return [o.result() for o in outs]
    if call == "chain":
        z = gb.sptc_resident(ctx, *jobs[0])
        r = _to_device(ctx, z, state["t"], [z.order - 1], [0], state["accum"])
        z.free()
        return r
    plan = state["plan"]
    plan.refresh()
    if plan.nchunks == 1:
        plan.execute(0, state["keys"], state["vals"])
        n = plan.total
        return {"keys": state["keys"][:n], "vals": state["vals"][:n]}
    keys = torch.empty(plan.total, dtype=torch.int64, device=DEV)
    vals = torch.empty(plan.total, dtype=torch.float32, device=DEV)
    for k in range(plan.nchunks):
        first, n = plan.chunk(k)
        plan.execute(k, keys[first:first + n], vals[first:first + n])
    return {"keys": keys, "vals": vals}


# ------------------------------------------------------------------ float64 join
def _parts(t, cmodes):
    """Free and contract part of every coordinate, as the engine packs them (the first mode highest)."""
    f = torch.zeros_like(t.idx[0])
    for m, d in enumerate(t.dims):
        if m not in cmodes:
            f = (f << _bits(d)) | t.idx[m]
    c = torch.zeros_like(t.idx[0])
    for m in cmodes:
        c = (c << _bits(t.dims[m])) | t.idx[m]
    return f, c


def _join(X, Y, cx, cy, count_only=False):
    """(keys, float64 sums, products) of Z, or (None, outputs, products)."""
    xf, xc = _parts(X, cx)
    yf, yc = _parts(Y, cy)
    nfb = sum(_bits(d) for m, d in enumerate(Y.dims) if m not in cy)
    o = torch.sort(xf, stable=True)[1]
    xf, xc, xv = xf[o], xc[o], X.val[o].double()
    o = torch.sort(yc, stable=True)[1]
    yf, yc, yv = yf[o], yc[o], Y.val[o].double()
    lo = torch.searchsorted(yc, xc)
    cnt = torch.searchsorted(yc, xc, right=True) - lo
    pre = torch.cumsum(cnt, 0)
    total = int(pre[-1]) if pre.numel() else 0
    # whole output rows at a time, so that every key's products are together
    row_end = torch.nonzero(torch.cat([xf[1:] != xf[:-1], torch.ones(1, dtype=torch.bool, device=xf.device)]))[:, 0] + 1
    row_pre = pre[row_end - 1]
    keys, sums, outputs, a, done = [], [], 0, 0, 0
    while done < total:
        r = int(torch.searchsorted(row_pre, torch.tensor(done + PRODUCTS_AT_ONCE, device=xf.device), right=True))
        r = max(r, int(torch.searchsorted(row_pre, torch.tensor(done, device=xf.device), right=True)) + 1)
        b = int(row_end[min(r, row_end.numel()) - 1])
        n = cnt[a:b]
        i = torch.repeat_interleave(torch.arange(a, b, device=xf.device), n)
        j = torch.arange(i.numel(), device=xf.device) - (pre[i] - cnt[i] - done) + lo[i]
        k, at = torch.sort((xf[i] << nfb) | yf[j])
        new = torch.ones(k.numel(), dtype=torch.bool, device=k.device)
        new[1:] = k[1:] != k[:-1]
        if count_only:
            outputs += int(new.sum())
        else:
            seg = torch.cumsum(new, 0) - 1
            s = torch.zeros(int(seg[-1]) + 1, dtype=torch.float64, device=k.device)
            s.index_add_(0, seg, (xv[i] * yv[j])[at])
            keys.append(k[new])
            sums.append(s)
        done = int(pre[b - 1])
        a = b
    if count_only:
        return None, outputs, total
    if not keys:
        return xf[:0], xv[:0], 0
    return torch.cat(keys), torch.cat(sums), total


def _z_tensor(X, Y, cx, cy, keys, sums):
    """A joined result as an operand (X's free modes, then Y's)."""
    dims = [d for m, d in enumerate(X.dims) if m not in cx] + [d for m, d in enumerate(Y.dims) if m not in cy]
    idx, k = [], keys
    for d in reversed(dims):
        idx.append(k & ((1 << _bits(d)) - 1))
        k = k >> _bits(d)
    return _Coo(dims, torch.stack(idx[::-1]), sums)


def exact(case, seed):
    pairs, T = _inputs(case, seed)
    outs = []
    for X, Y, cx, cy in pairs:
        keys, sums, _ = _join(X, Y, cx, cy)
        if T is not None:
            z = _z_tensor(X, Y, cx, cy, keys, sums)
            keys, sums, _ = _join(z, T, [len(z.dims) - 1], [0])
        outs.append({"keys": keys, "vals": sums})
    return outs if case["call"] in ("batch", "serve") else outs[0]


def work(case):
    """Operands read once (8 B an index, 4 B a value; a replayed plan reads values alone), results written once (8 B
    a key, 4 B a value); a multiply and an add for every matched product."""
    pairs, T = _inputs(case, 1)
    b = f = 0
    for X, Y, cx, cy in pairs:
        for t in ([X] if Y is X else [X, Y]):
            b += t.val.numel() * (4 if case["call"] == "plan" else 8 * len(t.dims) + 4)
        if T is None:
            _, n, p = _join(X, Y, cx, cy, count_only=True)
            f += 2 * p
        else:  # the first result is written and read as coordinates
            keys, sums, p = _join(X, Y, cx, cy)
            z = _z_tensor(X, Y, cx, cy, keys, sums)
            _, n, p2 = _join(z, T, [len(z.dims) - 1], [0], count_only=True)
            b += 2 * sums.numel() * (8 * len(z.dims) + 4) + T.val.numel() * (8 * len(T.dims) + 4)
            f += 2 * (p + p2)
        b += 12 * n
    return {"bytes": float(b), "flops": float(f)}
