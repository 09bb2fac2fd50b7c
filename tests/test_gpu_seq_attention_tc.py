"""Prompt attention on the tensor cores against float64 and against the float32 kernel on the same keys and values (a float32
cache holding the bfloat16 values takes that kernel): every form of mask, distance term, sink, weight and gate, head sizes off the
64-element chunks, tiles of keys that end inside a sequence, pages of any size, portions over a long past, key slices, rows whose
reference moves late, and non-finite keys outside a tile.

The tensor-core form holds queries and key weights with all 24 bits (three bfloat16 terms each) and sums in float32, so its error
against float64 may not exceed the float32 kernel's beyond the noise of two such sums: twice, plus 2 units of the largest output."""
import ctypes as C

import numpy as np
import pytest

import pygpukit_b200 as gk
from pygpukit_b200._lib import api

pytestmark = pytest.mark.gpu


def bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32)


def dev16(a):
    return gk.from_numpy((np.ascontiguousarray(a, np.float32).view(np.uint32) >> 16).astype(np.uint16).reshape(a.shape))


class Case:
    """portions [(first position, tokens), ...] of sequences whose earlier keys are in the cache"""

    def __init__(self, portions, H, G, D, Dv, PS=64, chunk=0, window=0, keep=0, cap=0.0, slopes=0, sinks=False, gate=0, prob=False,
                 splits=1, alias=False, seed=0, q_gain=1.0, single=0):
        self.__dict__.update({k: v for k, v in locals().items() if k != "self"})
        rng = np.random.default_rng(seed + H * 100 + D)
        self.scale = D ** -0.5
        S = len(portions)
        ends = [p + n for p, n in portions]
        per = max(-(-e // PS) for e in ends)
        self.table = rng.permutation(S * per + 3)[:S * per].reshape(S, per).astype(np.int32)
        pages = S * per + 3
        self.k = bf16(rng.standard_normal((pages, G, PS, D)).astype(np.float32))
        self.v = self.k if alias else bf16(rng.standard_normal((pages, G, PS, Dv)).astype(np.float32))
        self.T = sum(n for _, n in portions)
        self.ld = H * D + 4
        self.q = (q_gain * rng.standard_normal((self.T, self.ld))).astype(np.float32)
        self.sl = (0.05 * rng.random(H)).astype(np.float32) if slopes else None
        self.sl2 = (1.0 + rng.random(H)).astype(np.float32) if slopes == 2 else None
        self.sink = rng.standard_normal(H).astype(np.float32) if sinks else None
        self.pb = (rng.standard_normal(H) - 2).astype(np.float32) if prob else None
        self.g = rng.standard_normal((self.T, H * Dv)).astype(np.float32)

    def run(self, f32_cache):
        hb = int(api.seq_heads_per_block(self.H, self.G))
        qt = int(api.seq_queries_per_tile(self.H, self.G))
        tiles, row = [], 0
        for s, (p, n) in enumerate(self.portions):
            tiles += [(row + i, 1 if self.single else min(qt, n - i), s, p + i) for i in range(0, n, 1 if self.single else qt)]
            row += n
        assert hb * qt <= 32
        up = gk.from_numpy if f32_cache else dev16
        k = up(self.k)
        v = k if self.alias else up(self.v)
        q, t, tl, g = gk.from_numpy(self.q), gk.from_numpy(self.table), gk.from_numpy(np.asarray(tiles, np.int32)), gk.from_numpy(self.g)
        opt = {n: gk.from_numpy(a) if a is not None else None for n, a in (("sl", self.sl), ("sl2", self.sl2), ("sink", self.sink), ("pb", self.pb))}
        ptr = {n: a.device_ptr if a is not None else None for n, a in opt.items()}
        out = gk.from_numpy(np.full((self.T, self.H * self.Dv), 7.0, np.float32))
        ws = gk.zeros((self.T * self.H * self.splits * (self.Dv + 2),), gk.float32)
        tk = gk.zeros((4096,), gk.int32)
        api.seq_attention_ex3(q.device_ptr, self.ld, 4, g.device_ptr, self.H * self.Dv, 0, self.gate, out.device_ptr, self.H * self.Dv, k.device_ptr,
                              v.device_ptr, self.D, self.D if self.alias else self.Dv, 0 if f32_cache else 2, t.device_ptr, self.table.shape[1],
                              self.PS, tl.device_ptr, len(tiles), ptr["sl"], ptr["sl2"], ptr["sink"], self.H, self.G, self.D, self.Dv, self.chunk,
                              self.window, self.keep, self.scale, self.cap, 1 if self.prob else 0, ptr["pb"], 0.75, 0, 0, None, None, None, 0,
                              self.splits, ws.device_ptr, tk.device_ptr, self.single, None)
        r = out.to_numpy()
        assert (tk.to_numpy() == 0).all()
        err = C.c_int(7)
        api.seq_attention_wait_error(C.byref(err))
        assert err.value == 0
        return r

    def exact(self):
        out, row = np.zeros((self.T, self.H, self.Dv)), 0
        for s, (p, n) in enumerate(self.portions):
            j = np.arange(p + n)
            pg = self.table[s][j // self.PS]
            K = self.k[pg, :, j % self.PS].astype(np.float64)                  # [keys, G, D]
            V = self.v[pg, :, j % self.PS].astype(np.float64)[..., :self.Dv]
            Q = self.q[row:row + n, 4:].reshape(n, self.H, self.D).astype(np.float64)
            i = p + np.arange(n)
            vis = j[None, :] <= i[:, None]
            lo = np.zeros(n, int)
            if self.chunk:
                lo = i // self.chunk * self.chunk
            if self.window:
                lo = np.maximum(lo, i - self.window + 1)
            near = j[None, :] >= lo[:, None]
            if self.window and self.keep:
                near |= j[None, :] < self.keep
            vis &= near
            for h in range(self.H):
                g = h // (self.H // self.G)
                z = Q[:, h] @ K[:, g].T * self.scale
                if self.cap:
                    z = self.cap * np.tanh(z / self.cap)
                d = np.maximum(i[:, None] - j[None, :], 0).astype(np.float64)
                if self.slopes == 1:
                    z = z - self.sl[h].astype(np.float64) * d
                if self.slopes == 2:
                    z = z - self.sl[h].astype(np.float64) * np.log1p(self.sl2[h].astype(np.float64) * d)
                if self.prob:
                    w = np.where(vis, 1 / (1 + np.exp(-(z + self.pb[h]))), 0.0)
                else:
                    z = np.where(vis, z, -np.inf)
                    m = z.max(1, keepdims=True)
                    if self.sinks:
                        m = np.maximum(m, self.sink[h])
                    e = np.exp(z - m)
                    w = e / (e.sum(1, keepdims=True) + (np.exp(self.sink[h] - m) if self.sinks else 0.0))
                out[row:row + n, h] = w @ V[:, g]
            row += n
        out *= 0.75
        if self.gate == 1:
            out /= 1 + np.exp(-self.g.astype(np.float64)).reshape(self.T, self.H, self.Dv)
        if self.gate == 2:
            out /= 1 + np.exp(-self.g[:, :self.H].astype(np.float64))[:, :, None]
        return out.reshape(self.T, -1)


FORMS = [
    dict(portions=[(0, 300)], H=8, G=2, D=128, Dv=128),
    dict(portions=[(0, 1), (0, 129), (0, 64), (5, 9)], H=6, G=3, D=64, Dv=64, PS=16),
    dict(portions=[(0, 260)], H=16, G=2, D=128, Dv=128, chunk=100, cap=5.0, slopes=1, gate=1),
    dict(portions=[(0, 200), (700, 40)], H=4, G=4, D=96, Dv=96, window=130, keep=3, slopes=2, PS=7),
    dict(portions=[(0, 257)], H=16, G=1, D=576, Dv=512, sinks=True, gate=2, alias=True),
    dict(portions=[(300, 33)], H=12, G=1, D=144, Dv=128, window=200, sinks=True, alias=True, PS=32),
    dict(portions=[(0, 150), (20, 31)], H=8, G=4, D=40, Dv=24, prob=True, PS=5),
    dict(portions=[(0, 140)], H=40, G=1, D=32, Dv=256, cap=30.0, gate=1),
    dict(portions=[(1000, 20)], H=8, G=2, D=128, Dv=128, splits=4, sinks=True, gate=1),
    dict(portions=[(900, 7), (0, 5)], H=8, G=2, D=72, Dv=136, splits=7, window=500, keep=130),
    dict(portions=[(700, 3)], H=8, G=2, D=128, Dv=64, splits=3, prob=True),
    dict(portions=[(0, 300)], H=8, G=8, D=128, Dv=128, q_gain=30.0),                 # sharp rows: references move late
    dict(portions=[(0, 150), (400, 60)], H=8, G=2, D=128, Dv=128, window=77, keep=5, slopes=2, cap=8.0, PS=24),
    dict(portions=[(0, 200)], H=8, G=4, D=64, Dv=80, prob=True, slopes=1, cap=20.0, PS=128),
]


@pytest.mark.parametrize("form", range(len(FORMS)))
def test_forms(form):
    c = Case(**FORMS[form])
    ref = c.exact()
    old, new = c.run(True), c.run(False)
    top = np.abs(ref).max()
    worst_old, worst_new = np.abs(old - ref).max(), np.abs(new - ref).max()
    rms_old, rms_new = (np.sqrt(np.mean((x - ref) ** 2)) for x in (old, new))
    print(f"form {form}: max {worst_old:.2e} -> {worst_new:.2e}, rms {rms_old:.2e} -> {rms_new:.2e}, top {top:.2f}")
    assert worst_new <= 2 * worst_old + 2 * 2.0 ** -23 * top
    assert rms_new <= 1.5 * rms_old + 2.0 ** -24 * top


DECODE = [
    dict(H=16, G=4, D=128, Dv=128, window=90, gate=1),
    dict(H=16, G=1, D=576, Dv=512, alias=True, sinks=True),
    dict(H=8, G=8, D=64, Dv=80, slopes=1, cap=20.0, PS=7),
    dict(H=40, G=1, D=40, Dv=256, chunk=100, gate=2, PS=16),
    dict(H=6, G=2, D=100, Dv=128),                               # rows that the copies cannot fetch: the float32 kernel
]


@pytest.mark.parametrize("splits", [1, 2, 8, 64])
@pytest.mark.parametrize("form", range(len(DECODE)))
def test_decoding(form, splits):
    """one query per request, over contexts that end at and beside a tile of keys: the bounds of the portions above"""
    c = Case([(p, 1) for p in (0, 59, 126, 127, 128, 300, 1030)], splits=splits, single=2, **DECODE[form])
    ref = c.exact()
    old, new = c.run(True), c.run(False)
    top = np.abs(ref).max()
    assert np.abs(new - ref).max() <= 2 * np.abs(old - ref).max() + 2 * 2.0 ** -23 * top


def test_late_maximum():
    """one key far back beats everything behind it by hundreds: sums and outputs kept so far must vanish, not overflow"""
    c = Case([(0, 400)], 8, 2, 128, 128, seed=3)
    for at in (3, 399):
        pg, r = c.table[0][at // 64], at % 64
        q = c.q[399, 4:].reshape(8, 128)
        for g in range(2):
            c.k[pg, g, r] = bf16(40.0 * np.sign(q[4 * g:4 * g + 4].sum(0)))
        ref, new = c.exact(), c.run(False)
        assert np.abs(new - ref).max() <= 2 * np.abs(c.run(True) - ref).max() + 1e-6


def test_non_finite_rows_stay_outside():
    """stale rows behind a sequence's end and rows before its window never touch an output"""
    c = Case([(0, 100), (500, 30)], 8, 2, 128, 128, window=64, seed=4)
    clean = c.run(False)
    used = np.zeros((c.k.shape[0], c.PS), bool)
    for s, (p, n) in enumerate(c.portions):
        j = np.arange(max(0, p - 63), p + n)
        used[c.table[s][j // c.PS], j % c.PS] = True
    for arr in (c.k, c.v):
        arr.transpose(0, 2, 1, 3)[~used] = np.nan
    assert (c.run(False) == clean).all()


def test_nan_query_stays_in_its_row():
    c = Case([(0, 90)], 8, 2, 64, 64, seed=5)
    clean = c.run(False)
    c.q[40] = np.nan
    out = c.run(False)
    keep = np.arange(90) != 40
    assert (out[keep] == clean[keep]).all() and np.isnan(out[40]).all()


@pytest.mark.parametrize("Dv", [8, 72, 136, 264])
@pytest.mark.parametrize("gate", [0, 1])
def test_value_rows_off_the_chunks(Dv, gate):
    """lanes beyond the value row skip their stores between one load of the accumulators and the next"""
    c = Case([(0, 130), (140, 1)], 24, 1, 64, Dv, gate=gate, seed=6)
    ref, old, new = c.exact(), c.run(True), c.run(False)
    assert np.abs(new - ref).max() <= 2 * np.abs(old - ref).max() + 2 * 2.0 ** -23 * np.abs(ref).max()


INFINITE = [
    dict(portions=[(0, 150)], H=8, G=2, D=64, Dv=64),
    dict(portions=[(0, 150), (200, 9)], H=8, G=2, D=128, Dv=136, cap=5.0, slopes=1, gate=1, window=90),
    dict(portions=[(0, 150)], H=16, G=2, D=72, Dv=64, prob=True, PS=5),
    dict(portions=[(140, 10)], H=8, G=2, D=64, Dv=64, splits=2, sinks=True),
    dict(portions=[(59, 1), (127, 1), (300, 1)], H=16, G=2, D=128, Dv=128, single=2),
]


@pytest.mark.parametrize("where", ["query", "key", "value"])
@pytest.mark.parametrize("form", range(len(INFINITE)))
def test_infinities_follow_float32(form, where):
    """An infinity in a query, key or value row gives what the float32 kernel gives: an infinite score is a weight of 0 (or a cap, or 0
    and 1 under the sigmoid) or makes its row NaN, an infinite value with a weight is that infinity.  Where that is finite both
    are within the sums' float32 error of each other."""
    c = Case(seed=8, **INFINITE[form])
    rng = np.random.default_rng(form)
    if where == "query":                                 # a dimension in which the first half of the groups have keys of one sign
        c.k[..., 5] = bf16(np.abs(c.k[..., 5]) + 0.01)
        q = c.q[:, 4:].reshape(c.T, c.H, c.D)
        q[::3, ::2, 5], q[1::3, 1::2, 5] = np.inf, -np.inf
        c.q[:, 4:] = q.reshape(c.T, -1)
        c.q[:, 4:][:, ::7] = bf16(c.q[:, 4:][:, ::7])    # elements whose smaller terms are 0
    rows = [(0, j) for j in (2, 31, 57)]
    for n, (s, j) in enumerate(rows):
        pg, r = c.table[s][j // c.PS], j % c.PS
        if where == "key":
            c.k[pg, n % c.G, r, 3] = np.inf if n % 2 else -np.inf
        if where == "value":
            c.v[pg, :, r, 5 * n:5 * n + 9] = np.inf if n % 2 else -np.inf
    new, c.single = c.run(False), 0                      # (the float32 kernel for one query per tile writes 0 for a NaN row)
    old = c.run(True)
    assert (np.isnan(old) == np.isnan(new)).all()
    assert not np.isfinite(old).all() or where == "query" or c.prob or c.cap
    inf = np.isinf(old)
    assert (inf == np.isinf(new)).all() and (np.sign(old[inf]) == np.sign(new[inf])).all()
    fin = np.isfinite(old)
    assert fin.any() and np.abs(old[fin] - new[fin]).max() <= 2.0 ** -18 * (1 + np.abs(old[fin]).max())
