"""Row kernels of the token-major models in the forms that many rows take: a causal convolution of several rows per thread, the
weighted sum of expert rows by four elements, router logits by pairs of rows, rotary angles shared by a token's heads."""
import numpy as np
import pytest

import pygpukit_b200 as gk
from pygpukit_b200._lib import api

pytestmark = pytest.mark.gpu


def f32(a):
    return gk.from_numpy(np.ascontiguousarray(a, np.float32))


def i32(a):
    return gk.from_numpy(np.ascontiguousarray(a, np.int32))


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
@pytest.mark.parametrize("rows,twice", [((256,), False), ((1, 258, 2, 3), True), ((130, 131), True), ((5, 1, 1, 300), False)])
def test_convolution_over_many_rows_equals_portions(rows, twice, taps, width=300):
    """one launch of 256 rows and more against the same rows in launches of fewer (the kernel of a row per block): the same bits in
    rows and rings, sequences that start, continue and end anywhere in a thread's four rows"""
    W, S = width, len(rows)
    rng = np.random.default_rng(sum(rows) + taps)
    ring, first = max(1, taps - 1), [0 if s % 2 == 0 else 7 for s in range(S)]
    h, w = rng.standard_normal((sum(rows), W)), f32(rng.standard_normal((W, taps)))
    start = rng.standard_normal((S, (2 if twice else 1) * ring * W)).astype(np.float32)
    at = np.concatenate([[0], np.cumsum(rows)])

    def run(parts):
        state, steps, got = f32(start), [0] * S, [[] for _ in rows]
        for part in parts:                                       # [(sequence, first, end)]
            x = np.concatenate([h[at[s] + lo:at[s] + hi] for s, lo, hi in part])
            slot = np.concatenate([[s] * (hi - lo) for s, lo, hi in part])
            pos = np.concatenate([first[s] + np.arange(lo, hi) for s, lo, hi in part])
            par = np.concatenate([[steps[s] & 1] * (hi - lo) for s, lo, hi in part])
            seqs, row = [], 0
            for s, lo, hi in part:
                seqs.append((row, hi - lo, s, first[s] + lo))
                row += hi - lo
            xd, u, sl, ps, pr, sq = f32(x), gk.zeros(x.shape, gk.float32), i32(slot), i32(pos), i32(par), i32(seqs)
            api.causal_conv_rows_f32(xd.device_ptr, u.device_ptr, w.device_ptr, state.device_ptr, sl.device_ptr, ps.device_ptr,
                                     pr.device_ptr if twice else None, len(x), W, taps, None)
            if not twice:
                api.causal_conv_state_f32(xd.device_ptr, state.device_ptr, sq.device_ptr, len(seqs), W, taps, None)
            out, row = u.to_numpy(), 0
            for s, lo, hi in part:
                got[s].append(out[row:row + hi - lo])
                row += hi - lo
                steps[s] += 1
        return np.concatenate([np.concatenate(g) for g in got])

    whole = run([[(s, 0, n) for s, n in enumerate(rows)]])
    cut = run([[(s, lo, min(lo + 100, n))] for s, n in enumerate(rows) for lo in range(0, n, 100)])
    assert np.array_equal(whole, cut)


@pytest.mark.parametrize("top,W", [(1, 4), (4, 2048), (8, 516), (9, 64), (3, 30), (64, 12)])
def test_weighted_sum_of_expert_rows(top, W):
    rng = np.random.default_rng(top + W)
    T = 37
    parts, own, shared = (rng.standard_normal((n, W)).astype(np.float32) for n in (T * top, T, T))
    wt = rng.random((T, top)).astype(np.float32)
    inv = rng.permutation(T * top).reshape(T, top)
    mat = np.where(rng.random((T, top)) < 0.2, -1, 0)
    gate = rng.standard_normal((T, 3)).astype(np.float32)
    keep = [f32(parts), i32(inv), i32(mat), f32(wt), f32(own), f32(shared), f32(gate)]
    out = gk.from_numpy(np.full((T, W), 7.0, np.float32))
    p = [k.device_ptr for k in keep]
    api.moe_combine_rows_f32(p[0], p[1], p[2], p[3], top, p[4], p[5], p[6], 3, 1, out.device_ptr, T, W, None)
    x = np.where((mat < 0)[..., None], own[:, None].astype(np.float64), parts.astype(np.float64)[inv])
    terms = np.concatenate([wt[..., None].astype(np.float64) * x, (shared / (1 + np.exp(-gate[:, 1:2].astype(np.float64))))[:, None]], 1)
    assert (np.abs(out.to_numpy() - terms.sum(1)) <= 2.0 ** -23 * (top + 4) * np.abs(terms).sum(1) + 1e-30).all()


@pytest.mark.parametrize("M,N,K", [(9, 1, 32), (10, 8, 33), (17, 9, 100), (300, 16, 2048), (2001, 64, 31), (1000, 63, 520)])
def test_router_logits(M, N, K):
    rng = np.random.default_rng(M + N)
    A, W = rng.standard_normal((M, K + 1)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    a, w, c = f32(A), f32(W), gk.from_numpy(np.full((M, N + 1), 7.0, np.float32))
    api.gemm_rows_f32(a.device_ptr, K + 1, None, w.device_ptr, 0, 0, c.device_ptr, N + 1, M, N, K, None, 1, M, 0, 1.0, 0.0, None)
    x, y = A[:, :K].astype(np.float64), W.astype(np.float64)
    out = c.to_numpy()
    assert (np.abs(out[:, :N] - x @ y.T) <= 2.0 ** -24 * (K / 32 + 6) * (np.abs(x) @ np.abs(y).T)).all()
    assert (out[:, N:] == 7.0).all()


@pytest.mark.parametrize("H,D,rot", [(1, 16400, 16400), (9, 8200, 8194), (4, 64, 0), (2, 96, 50), (9, 96, 50), (33, 64, 64)])
def test_turned_heads_of_any_length(H, D, rot):
    """heads with more pairs than the kernel's table of angles holds: silu and turn of q and k in float32 on float64 angles, two
    products and a sum of values of about 1 and the table's roundings"""
    T, Dv = 5, 24
    rng = np.random.default_rng(D + rot)
    ld = 2 * H * D + H * Dv
    x = rng.standard_normal((T, ld)).astype(np.float32)
    pos = np.array([0, 1, 77, 4095, 100000])
    freq = 10000.0 ** (-np.arange(max(1, rot // 2)) / max(1, rot // 2))
    p, fr, ps = f32(x), gk.from_numpy(freq), i32(pos)
    api.seq_linear_prep(p.device_ptr, ld, T, H, D, Dv, 0, H * D, 2 * H * D, 1, rot, fr.device_ptr, 0.25, ps.device_ptr, None)
    s = x.astype(np.float64) / (1 + np.exp(-x.astype(np.float64)))
    qk = s[:, :2 * H * D].reshape(T, 2 * H, D).copy()
    h = rot // 2
    a = (pos[:, None] * freq[None, :h])[:, None]
    lo, hi = qk[..., :h].copy(), qk[..., h:rot].copy()
    qk[..., :h], qk[..., h:rot] = lo * np.cos(a) - hi * np.sin(a), hi * np.cos(a) + lo * np.sin(a)
    qk[:, H:] *= 0.25
    ref = np.concatenate([qk.reshape(T, -1), s[:, 2 * H * D:]], 1)
    assert np.abs(p.to_numpy() - ref).max() <= 2.0 ** -20 * (1 + np.abs(s).max())


@pytest.mark.parametrize("lens,heads,dim,vdim", [([128], 2, 128, 128), ([129, 1, 300], 2, 128, 72), ([70, 257], 3, 72, 128), ([640], 20, 64, 64), ([33, 127], 4, 128, 64)])
@pytest.mark.parametrize("start", [0, 9])
def test_linear_attention_chunks_against_float64(lens, heads, dim, vdim, start):
    """Chunks of 128 tokens: ragged sequences that end inside, on and behind a chunk's edge, heads that do not fill a tile, states carried in and
    from one segment to the next.  Operands keep 24 bits and sums are float32, so errors stay within a few 2^-24 of the sums of magnitudes."""
    rng = np.random.default_rng(sum(lens) + dim)
    T, S, ld = sum(lens), len(lens), 2 * heads * dim + heads * vdim + 4
    proj = rng.standard_normal((T, ld)).astype(np.float32)
    decay = (1 - 2.0 ** -np.linspace(3, 9, heads)).astype(np.float32)
    state = rng.standard_normal((S, heads, dim, vdim)).astype(np.float32)
    rows = np.cumsum([0] + lens)
    seqs = np.array([(rows[i], n, i, start) for i, n in enumerate(lens)], np.int32)
    k_off, v_off, chunks = heads * dim, 2 * heads * dim, -(-max(lens) // 32)
    gp, gs, gd, gq = gk.from_numpy(proj), gk.from_numpy(state), gk.from_numpy(decay), gk.from_numpy(seqs)
    out, ws = gk.zeros((T, heads * vdim), gk.float32), gk.zeros((chunks * S * heads * dim * vdim,), gk.float32)
    for c0, n in ((0, 5), (5, chunks - 5)) if chunks > 5 else ((0, chunks),):
        api.seq_linear_attention_chunks(gp.device_ptr, ld, 0, k_off, v_off, out.device_ptr, heads * vdim, gs.device_ptr, gd.device_ptr, gq.device_ptr, S,
                                        heads, dim, vdim, c0, n, ws.device_ptr, None)
    got, after = out.to_numpy().astype(np.float64), gs.to_numpy().astype(np.float64)
    for i, n in enumerate(lens):
        x = proj[rows[i]:rows[i + 1]].astype(np.float64)
        t = np.arange(n)
        for h in range(heads):
            q, k, v = x[:, h * dim:(h + 1) * dim], x[:, k_off + h * dim:k_off + (h + 1) * dim], x[:, v_off + h * vdim:v_off + (h + 1) * vdim]
            a, s0 = float(decay[h]), state[i, h].astype(np.float64) * (start > 0)
            w = np.where(t[:, None] >= t[None], a ** np.maximum(t[:, None] - t[None], 0), 0.0)
            fall, rest = (a ** (t + 1.0))[:, None], (a ** (n - 1.0 - t))[:, None]
            ref, size = (q @ k.T * w) @ v + fall * (q @ s0), (np.abs(q) @ np.abs(k).T * w) @ np.abs(v) + fall * (np.abs(q) @ np.abs(s0))
            sref, ssize = a ** n * s0 + (k * rest).T @ v, a ** n * np.abs(s0) + (np.abs(k) * rest).T @ np.abs(v)
            assert (np.abs(got[rows[i]:rows[i + 1], h * vdim:(h + 1) * vdim] - ref) <= 64 * 2.0 ** -24 * size).all()
            assert (np.abs(after[i, h] - sref) <= 64 * 2.0 ** -24 * ssize).all()


def test_linear_attention_chunks_with_an_infinite_value():
    """float32 semantics: the outputs that see the value are infinite or NaN, all others are untouched."""
    rng = np.random.default_rng(3)
    T, heads, dim, vdim = 300, 2, 128, 64
    ld = 2 * heads * dim + heads * vdim
    proj = np.abs(rng.standard_normal((T, ld))).astype(np.float32)
    decay, seqs = np.full(heads, 0.99, np.float32), np.array([(0, T, 0, 0)], np.int32)

    def run(p):
        bufs = [gk.from_numpy(p), gk.zeros((1, heads, dim, vdim), gk.float32), gk.from_numpy(decay), gk.from_numpy(seqs),
                gk.zeros((T, heads * vdim), gk.float32), gk.zeros((10 * heads * dim * vdim,), gk.float32)]
        x, s, d, q, o, w = (b.device_ptr for b in bufs)
        api.seq_linear_attention_chunks(x, ld, 0, heads * dim, 2 * heads * dim, o, heads * vdim, s, d, q, 1, heads, dim, vdim, 0, 10, w, None)
        return bufs[4].to_numpy()

    a = run(proj)
    proj[150, 2 * heads * dim + 7] = np.inf
    b = run(proj)
    assert np.isposinf(b[150:, 7]).all()
    keep = np.ones_like(a, bool)
    keep[150:, 7] = False
    assert np.isfinite(b[keep]).all() and np.abs(b - a)[keep].max() <= 1e-5 * np.abs(a).max()


_HELD = []


def _held(a):
    """the address of an operand that lives until the next test"""
    _HELD.append(a)
    return a.device_ptr


@pytest.fixture(autouse=True)
def _let_go():
    yield
    gk.synchronize()
    _HELD.clear()


def _close(got, ref, terms):
    """float32 arithmetic of a row kernel: sums in some order (a block's: up to 20 additions in a row beside the elements of a thread) and a
    handful of roundings behind them, of magnitudes `terms`"""
    assert (np.abs(got - ref) <= 2.0 ** -24 * 48 * (np.abs(terms) + 1.0)).all()


@pytest.mark.parametrize("W", [1, 63, 256, 260, 2048, 4095, 4096, 4097, 4100, 8192, 8193, 8196])
@pytest.mark.parametrize("rows", [1, 5])
def test_norms_of_rows_of_any_width(rows, W):
    """the forms by width (two and four groups of four per thread, shared memory beyond) and by alignment"""
    rng = np.random.default_rng(W)
    x, y, d = (rng.standard_normal((rows, W)).astype(np.float32) for _ in range(3))
    w, g, b = (rng.standard_normal(W).astype(np.float32) for _ in range(3))
    X, Y, D = (v.astype(np.float64) for v in (x, y, d))
    rms = lambda v, k: v / np.sqrt((v * v).mean(1, keepdims=True) + 1e-5) * k
    xs, out = f32(x), f32(y)
    api.rms_norm_rows_f32(xs.device_ptr, None, _held(f32(d)), xs.device_ptr, _held(f32(w)), 0.5, 1e-5, out.device_ptr, rows, W, 1, None)
    _close(xs.to_numpy(), X + D, X)
    _close(out.to_numpy(), Y + rms(X + D, 0.5 + w), 4 * (np.abs(Y) + np.abs(rms(X + D, 0.5 + w))))
    xs, h = f32(x), gk.from_numpy(np.full((rows, W), 7.0, np.float32))
    api.rms_norm_seam_f32(_held(f32(y)), _held(f32(w)), 1.0, xs.device_ptr, _held(f32(d)), _held(f32(g)), 0.0, 1e-5, h.device_ptr, rows, W, None)
    s = X + rms(Y, 1.0 + w) + D
    _close(xs.to_numpy(), s, 8 * np.abs(rms(Y, 1.0 + w)) + np.abs(X))
    _close(h.to_numpy(), rms(s, g), 40 * np.abs(rms(s, g)) + 8)
    top = 3
    parts, inv, wt = rng.standard_normal((rows * top, W)).astype(np.float32), rng.permutation(rows * top).reshape(rows, top), rng.random((rows, top)).astype(np.float32)
    out = f32(y)
    api.combine_layernorm_f32(_held(f32(x)), None, _held(f32(parts)), _held(i32(inv)), _held(f32(wt)), top, _held(f32(g)), _held(f32(b)),
                              1e-5, out.device_ptr, rows, W, 1, None)
    s = X + (wt[..., None].astype(np.float64) * parts.astype(np.float64)[inv]).sum(1)
    c = s - s.mean(1, keepdims=True)
    n = c / np.sqrt((c * c).mean(1, keepdims=True) + 1e-5)
    if W > 1:
        _close(out.to_numpy(), Y + n * g + b, 16 * (np.abs(n * g) + np.abs(g)) + np.abs(Y) + np.abs(b))
    table, toks = rng.standard_normal((9, W)).astype(np.float32), rng.integers(0, 9, rows)
    xs, keep = f32(x), f32(x)
    api.embed_norm_rows_f32(_held(f32(table)), 0, _held(i32(toks)), _held(f32(w)), 1.0, 1e-5, xs.device_ptr, keep.device_ptr, rows, W, 9, None)
    ref = rms(table.astype(np.float64)[toks], 1.0 + w)
    _close(xs.to_numpy(), ref, 4 * ref)
    assert np.array_equal(xs.to_numpy(), keep.to_numpy())


@pytest.mark.parametrize("H,G,D,Dv,pad", [(1, 1, 128, 128, 0), (32, 4, 128, 64, 4), (45, 9, 96, 100, 0), (6, 2, 4, 8, 1), (4, 2, 132, 128, 0)])
@pytest.mark.parametrize("T", [3, 400])
def test_heads_and_cache_rows_of_a_projection(H, G, D, Dv, pad, T):
    """several heads of a warp, heads that leave lanes idle, rows off 16-byte boundaries and heads too long for a lane's four elements; values recorded
    and mixed.  Queries and the float32 cache against float64."""
    rng = np.random.default_rng(H * D + T)
    PS, pages = 16, T // 16 + 1
    ld = (H + G) * D + G * Dv + pad
    x = rng.standard_normal((T, ld)).astype(np.float32)
    qw, kw = (rng.standard_normal(D).astype(np.float32) for _ in range(2))
    first = rng.standard_normal((T, G * Dv)).astype(np.float32)
    table = rng.permutation(pages).astype(np.int32)
    X = x.astype(np.float64)
    qk = X[:, :(H + G) * D].reshape(T, H + G, D)
    qk = qk / np.sqrt((qk * qk).mean(2, keepdims=True) + 1e-6) * np.where(np.arange(H + G)[:, None] < H, qw, kw)
    for mode in (0, 1, 2):
        p, kc, vc, vf = f32(x), gk.zeros((pages * G * PS * D,), gk.float32), gk.zeros((pages * G * PS * Dv,), gk.float32), f32(first)
        api.seq_mixer_prep(p.device_ptr, ld, T, H, G, D, Dv, _held(f32(qw)), _held(f32(kw)), 1e-6, mode, 0.25, vf.device_ptr, kc.device_ptr,
                           vc.device_ptr, 0, _held(i32(table)), pages, PS, _held(i32(np.zeros(T))), _held(i32(np.arange(T))), None)
        v = X[:, (H + G) * D:(H + G) * D + G * Dv]
        if mode == 2:
            v = 0.75 * v + 0.25 * first.astype(np.float64)
        rows = lambda c, n: c.to_numpy().reshape(pages, G, PS, n)[table].transpose(0, 2, 1, 3).reshape(pages * PS, G, n)[:T]
        got = p.to_numpy()
        _close(got[:, :H * D], qk[:, :H].reshape(T, -1), 4 * qk[:, :H].reshape(T, -1))
        _close(rows(kc, D), qk[:, H:], 4 * qk[:, H:])
        _close(rows(vc, Dv), v.reshape(T, G, Dv), 4 * v.reshape(T, G, Dv))
        assert np.array_equal(got[:, H * D:], x[:, H * D:])
        assert mode != 1 or np.array_equal(vf.to_numpy(), x[:, (H + G) * D:(H + G) * D + G * Dv])


@pytest.mark.parametrize("H,G,D,pad", [(4, 2, 64, 0), (16, 8, 128, 3), (32, 4, 128, 0), (33, 2, 128, 0), (3, 1, 30, 0)])
def test_whole_projection_norm(H, G, D, pad):
    rng = np.random.default_rng(H * D)
    T, PS, pages, off = 9, 4, 3, H * D + pad
    ld = off + G * D + pad
    x = rng.standard_normal((T, ld)).astype(np.float32)
    qb, qw = (rng.standard_normal(H * D).astype(np.float32) for _ in range(2))
    kb, kw = (rng.standard_normal(G * D).astype(np.float32) for _ in range(2))
    p, kc, vc = f32(x), gk.zeros((pages * G * PS * D,), gk.float32), gk.zeros((pages * G * PS * D,), gk.float32)
    api.seq_mixer_prep_all(p.device_ptr, ld, T, H, G, D, off, _held(f32(qb)), _held(f32(kb)), _held(f32(qw)), _held(f32(kw)), 1.0, 1e-6,
                           kc.device_ptr, vc.device_ptr, 0, _held(i32(np.arange(pages))), pages, PS, _held(i32(np.zeros(T))), _held(i32(np.arange(T))), None)
    q, k = x[:, :H * D].astype(np.float64) + qb, x[:, off:off + G * D].astype(np.float64) + kb
    rms = lambda v: v / np.sqrt((v * v).mean(1, keepdims=True) + 1e-6)
    rows = lambda c: c.to_numpy().reshape(pages, G, PS, D).transpose(0, 2, 1, 3).reshape(pages * PS, G * D)[:T]
    _close(p.to_numpy()[:, :H * D], rms(q) * (1.0 + qw), 4 * np.abs(rms(q)) * (1 + np.abs(qw)))
    _close(rows(kc), rms(k) * (1.0 + kw), 4 * np.abs(rms(k)) * (1 + np.abs(kw)))
    _close(rows(vc), k, 2 * np.abs(k))


@pytest.mark.parametrize("qr,rank,rot,turn,pad", [(768, 512, 64, 64, 0), (0, 256, 64, 32, 1), (2052, 512, 8, 8, 0), (512, 2100, 64, 64, 0), (30, 18, 6, 4, 0), (64, 64, 520, 516, 0)])
def test_latents_and_their_cache_rows(qr, rank, rot, turn, pad):
    rng = np.random.default_rng(qr + rank)
    T, PS, pages = 9, 4, 3
    ld = qr + rank + rot + pad
    x = rng.standard_normal((T, ld)).astype(np.float32)
    qw, cw = rng.standard_normal(max(1, qr)).astype(np.float32), rng.standard_normal(rank).astype(np.float32)
    freq, pos = 10000.0 ** (-np.arange(turn // 2) / (turn // 2)), np.arange(T)
    p, kc = f32(x), gk.zeros((pages * PS * (rank + rot),), gk.float32)
    api.seq_latent_prep(p.device_ptr, ld, T, qr, qr, rank, rot, turn, _held(f32(qw)) if qr else None, _held(f32(cw)), 1.0, 1e-6, _held(gk.from_numpy(freq)),
                        kc.device_ptr, 0, _held(i32(np.arange(pages))), pages, PS, _held(i32(np.zeros(T))), _held(i32(pos)), None)
    X = x.astype(np.float64)
    rms = lambda v: v / np.sqrt((v * v).mean(1, keepdims=True) + 1e-6)
    q, c, r = X[:, :qr], rms(X[:, qr:qr + rank]) * (1.0 + cw), X[:, qr + rank:qr + rank + rot].copy()
    a = pos[:, None] * freq
    u, v = r[:, 0:turn:2].copy(), r[:, 1:turn:2].copy()
    r[:, 0:turn:2], r[:, 1:turn:2] = u * np.cos(a) - v * np.sin(a), v * np.cos(a) + u * np.sin(a)
    got, rows = p.to_numpy(), kc.to_numpy().reshape(pages * PS, rank + rot)[:T]
    if qr:
        _close(got[:, :qr], rms(q) * (1.0 + qw), 4 * np.abs(rms(q)) * (1 + np.abs(qw)))
    _close(rows, np.concatenate([c, r], 1), 4 * np.abs(np.concatenate([c, np.abs(r) + 1], 1)))
    assert np.array_equal(got[:, qr:], x[:, qr:])


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (2000, 4, 18), (37, 8, 513), (4100, 2, 64)])
def test_rows_of_every_expert(T, top, E):
    rng = np.random.default_rng(T)
    idx = rng.integers(0, E, (T, top)).astype(np.int32)
    counts, rank = np.bincount(idx.ravel(), minlength=E), np.zeros(T * top, np.int64)
    for e in range(E):
        m = idx.ravel() == e
        rank[m] = rng.permutation(m.sum())
    cd, off, perm, inv = i32(counts), i32(np.zeros(E + 1)), i32(np.zeros(T * top)), i32(np.zeros(T * top))
    api.moe_row_lists(cd.device_ptr, off.device_ptr, _held(i32(idx)), _held(i32(rank)), perm.device_ptr, inv.device_ptr, E, T, top, None)
    first = np.concatenate([[0], np.cumsum(counts)])
    row = first[idx.ravel()] + rank
    assert np.array_equal(off.to_numpy(), first) and np.array_equal(inv.to_numpy(), row) and (cd.to_numpy() == 0).all()
    assert np.array_equal(perm.to_numpy()[row], np.arange(T * top) // top)


@pytest.mark.parametrize("taps", [3, 4])
def test_convolution_of_single_columns(taps):
    """rows whose width leaves no 16-byte boundaries"""
    test_convolution_over_many_rows_equals_portions((1, 258, 2, 3), True, taps, width=301)


@pytest.mark.parametrize("H,Dv,pad", [(16, 128, 0), (3, 7, 1), (33, 128, 0), (64, 128, 4), (65, 128, 0)])
@pytest.mark.parametrize("act", [0, 1, 2])
def test_output_norm_and_gate_over_all_heads(H, Dv, pad, act):
    rng = np.random.default_rng(H + Dv)
    T, n = 5, H * Dv
    o, g, w = rng.standard_normal((T, n + pad)).astype(np.float32), rng.standard_normal((T, n + 2 * pad)).astype(np.float32), rng.standard_normal(n).astype(np.float32)
    od = f32(o)
    api.seq_linear_finish(od.device_ptr, n + pad, _held(f32(g)), n + 2 * pad, pad, _held(f32(w)), T, H, Dv, 0, act, 1e-5, 0.5, None)
    x, z = o[:, :n].astype(np.float64), g[:, pad:pad + n].astype(np.float64)
    ref = x / np.sqrt((x * x).mean(1, keepdims=True) + 1e-5) * w * 0.5 * (1.0 if act == 0 else (1 if act == 1 else z) / (1 + np.exp(-z)))
    _close(od.to_numpy()[:, :n], ref, 4 * ref)
    assert np.array_equal(od.to_numpy()[:, n:], o[:, n:])
