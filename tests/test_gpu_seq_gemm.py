"""The many-row products of the token-major family at the sizes where their tiles end: row counts around the tile heights and
the MMA's granularity, columns and k that are no multiple of a tile, k cut over a cluster, every epilogue, row gathers, groups
of unequal length (empty, one row, several tiles) and batches -- against float64 products of the bfloat16-rounded operands.

Tolerance: a product of K bfloat16 pairs is exact per pair; the sums are formed in float32 in blocks of 16, at most K / 16 + 8
roundings of half a unit or truncations of one, so |error| <= (K / 16 + 8) 2^-23 sum |a w|.  An activation f changes that by its
slope (at most 2 here, for pairs times the other factor), and adds a few units of its own value."""
import ctypes as C

import numpy as np
import pytest

import pygpukit_b200 as gk
from pygpukit_b200 import llm
from pygpukit_b200._lib import api

pytestmark = pytest.mark.gpu


def bf16(a):
    u = np.ascontiguousarray(a, np.float32).view(np.uint32)
    return (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32)


def dev_w(a):
    a = np.ascontiguousarray(a, np.float32)
    return gk.from_numpy((a.view(np.uint32) >> 16).astype(np.uint16).reshape(a.shape))


def operands(seed, M, N, K, groups=1):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((M, K)).astype(np.float32)
    W = bf16(rng.standard_normal((groups, N, K)).astype(np.float32) / np.sqrt(K))
    return A, W


def product(A, W):
    a, w = bf16(A).astype(np.float64), W.astype(np.float64)
    return a @ w.T, (K_ROUND(A.shape[1]) * (np.abs(a) @ np.abs(w).T))


def K_ROUND(K):
    return (K / 16 + 8) * 2.0 ** -23


def no_wait_error():
    v = C.c_int(7)
    api.gemm_rows_wait_error(C.byref(v))
    assert v.value == 0


@pytest.mark.parametrize("M,N,K", [(9, 128, 64), (16, 130, 72), (17, 7, 128), (33, 257, 136), (64, 2048, 2048), (100, 96, 4096), (127, 129, 520),
                                   (255, 384, 192), (256, 128, 64), (257, 640, 320), (300, 1000, 1000), (513, 2049, 264), (2000, 272, 128)])
def test_rows(M, N, K):
    A, W = operands(M + N, M, N, K)
    ref, tol = product(A, W[0])
    a, w = gk.from_numpy(A), dev_w(W[0])
    c = gk.from_numpy(np.full((M, N + 3), 7.0, np.float32))
    api.gemm_rows_f32(a.device_ptr, K, None, w.device_ptr, 2, 0, c.device_ptr, N + 3, M, N, K, None, 1, M, 0, 1.0, 0.0, None)
    out = c.to_numpy()
    assert (np.abs(out[:, :N] - ref) <= tol + 1e-6).all()
    assert (out[:, N:] == 7.0).all()
    no_wait_error()


def gelu_tanh(z):
    return 0.5 * z * (1 + np.tanh(np.sqrt(2 / np.pi) * (z + 0.044715 * z ** 3)))


def sigmoid(z):
    return 1 / (1 + np.exp(-z))


@pytest.mark.parametrize("M,F,K", [(20, 66, 80), (130, 131, 256), (48, 64, 2048)])
@pytest.mark.parametrize("epi", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_epilogues(M, F, K, epi):
    from math import erf
    N = 2 * F if epi in (1, 3, 7) else F
    A, W = operands(M + epi, M, N, K)
    z, tol = product(A, W[0])
    rng = np.random.default_rng(epi)
    g, u = (z[:, 0::2], z[:, 1::2]) if epi in (1, 3, 7) else (z, None)
    old = rng.standard_normal((M, F)).astype(np.float32)
    colv = rng.standard_normal(F).astype(np.float32)
    table = rng.standard_normal((11, F + 5)).astype(np.float32)
    rows = rng.integers(0, 11, M).astype(np.int32)
    gate = rng.standard_normal((M, F + 2)).astype(np.float32)
    p0, p1, aux = 0.0, 0.0, (None, 0, None, 0, 0)
    if epi == 1:
        ref = g * sigmoid(g) * u
    elif epi == 2:
        p0, p1 = 1.3, 2.0
        ref = 2.0 * np.tanh(1.3 * z / 2.0)
    elif epi == 3:
        p0, p1 = 1.702, 0.9
        gg, uu = np.minimum(g, 0.9), np.clip(u, -0.9, 0.9)
        ref = gg * sigmoid(1.702 * gg) * (uu + 1)
    elif epi == 4:
        ref = old + colv * z
    elif epi == 5:
        ref = gelu_tanh(z) * table[rows, 3:3 + F]
    elif epi == 6:
        ref = np.maximum(z, 0) ** 2
    elif epi == 7:
        ref = gelu_tanh(g) * u
    elif epi == 8:
        ref = 0.5 * z * (1 + np.vectorize(erf)(z / np.sqrt(2)))
    elif epi == 9:
        ref = gelu_tanh(z)
    else:
        ref = z * sigmoid(gate[:, 1:1 + F])
    a, w, c = gk.from_numpy(A), dev_w(W[0]), gk.from_numpy(old)
    dt, dr, dg, dc = gk.from_numpy(table), gk.from_numpy(rows), gk.from_numpy(gate), gk.from_numpy(colv)
    if epi == 5:
        aux = (dt.device_ptr, 0, dr.device_ptr, F + 5, 3)
    if epi == 10:
        aux = (dg.device_ptr, 0, None, F + 2, 1)
    api.gemm_seq_f32(a.device_ptr, K, 0, w.device_ptr, 2, 0, c.device_ptr, F, 0, M, N, K, 1, epi, p0, p1, dc.device_ptr, aux[0], aux[1], aux[2],
                     aux[3], aux[4], 0, None)
    t = tol if epi not in (1, 3, 7) else np.maximum(tol[:, 0::2], tol[:, 1::2])
    slope = 4.0 * (1.0 + (np.abs(u) + np.abs(g) if u is not None else np.abs(z)) + np.abs(table[rows, 3:3 + F]) + np.abs(colv))
    assert (np.abs(c.to_numpy() - ref) <= slope * t + 1e-5 * (1 + np.abs(ref))).all()
    no_wait_error()


@pytest.mark.parametrize("counts,N,K", [([30, 0, 70, 1, 9], 130, 72), ([300, 16, 0, 17, 257, 1], 256, 128), ([0, 0, 5], 64, 200),
                                        ([1] * 40, 96, 64), ([0] * 7, 96, 64), ([3, 129] * 20, 64, 96)])
@pytest.mark.parametrize("extra", [0, 50])
def test_groups(counts, N, K, extra):
    E, R = len(counts), sum(counts)
    T = max(R, 8)
    A, W = operands(R + N, T, N, K, E)
    rng = np.random.default_rng(R)
    src = rng.integers(0, T, R + extra).astype(np.int32)
    src[R:] = 1 << 30                                    # rows behind the last group name nothing
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    a, w, o, s = gk.from_numpy(A), dev_w(W), gk.from_numpy(off), gk.from_numpy(src if len(src) else np.zeros(1, np.int32))
    c = gk.from_numpy(np.full((R + extra + 1, N), 7.0, np.float32))
    lin = llm.LinearRows(w)
    lin.forward_grouped(a.device_ptr, K, c.device_ptr, N, s.device_ptr, o.device_ptr, max(counts + [1]), R + extra)
    out = c.to_numpy()
    grp = np.repeat(np.arange(E), counts)
    for e in range(E):
        if counts[e]:
            ref, tol = product(A[src[:R]][grp == e], W[e])
            assert (np.abs(out[:R][grp == e] - ref) <= tol + 1e-6).all()
    assert (out[R:] == 7.0).all()
    no_wait_error()


@pytest.mark.parametrize("M,H,N,K,pad", [(40, 3, 96, 64, 0), (70, 5, 512, 128, 8), (260, 2, 130, 72, 4), (33, 4, 64, 128, 3)])
def test_batches(M, H, N, K, pad):
    """products on slices of the same rows, K + pad columns apart (pad 3: off the 16-byte grid)"""
    rng = np.random.default_rng(M)
    A = rng.standard_normal((M, H * (K + pad))).astype(np.float32)
    W = bf16(rng.standard_normal((H, N, K)).astype(np.float32) / np.sqrt(K))
    a, w, c = gk.from_numpy(A), dev_w(W), gk.zeros((M, H * (N + 1)), gk.float32)
    api.gemm_seq_f32(a.device_ptr, H * (K + pad), K + pad, w.device_ptr, 2, N * K, c.device_ptr, H * (N + 1), N + 1, M, N, K, H, 0, 0.0, 0.0, None,
                     None, 0, None, 0, 0, 0, None)
    out = c.to_numpy().reshape(M, H, N + 1)
    for h in range(H):
        ref, tol = product(A[:, h * (K + pad):h * (K + pad) + K], W[h])
        assert (np.abs(out[:, h, :N] - ref) <= tol + 1e-6).all()
    no_wait_error()


def test_nan_stays_in_its_row_and_batch():
    """a batch's k tail reads nothing of the next batch's columns"""
    M, H, N, K = 20, 2, 64, 72
    A = np.ones((M, H * K), np.float32)
    A[:, K:] = np.nan
    W = np.ones((H, N, K), np.float32)
    a, w, c = gk.from_numpy(A), dev_w(W), gk.zeros((M, H * N), gk.float32)
    api.gemm_seq_f32(a.device_ptr, H * K, K, w.device_ptr, 2, N * K, c.device_ptr, H * N, N, M, N, K, H, 0, 0.0, 0.0, None, None, 0, None, 0, 0, 0, None)
    out = c.to_numpy()
    assert (out[:, :N] == K).all() and np.isnan(out[:, N:]).all()


def test_captured_and_replayed():
    """work memory is part of a captured graph; replays follow new inputs"""
    M, N, K = 50, 256, 512
    A, W = operands(5, M, N, K)
    a, w, c = gk.from_numpy(A), dev_w(W[0]), gk.zeros((M, N), gk.float32)
    from pygpukit_b200.core.stream import CudaGraph, Stream
    st, g = Stream(), CudaGraph()
    lin = llm.LinearRows(w)
    with g.capture(st):
        lin.forward(a.device_ptr, K, M, c.device_ptr, N)
        lin.forward(a.device_ptr, K, M, c.device_ptr, N)
    for _ in range(3):
        a.copy_from_numpy(A)
        g.replay(st)
        st.synchronize()
        ref, tol = product(A, W[0])
        assert (np.abs(c.to_numpy() - ref) <= tol + 1e-6).all()
        A = A[::-1].copy()


# ---------------------------------------------------------------- at most 16 rows: the rounding in the kernel
@pytest.mark.parametrize("M", [1, 3, 8, 12, 16])
@pytest.mark.parametrize("N,K", [(128, 64), (130, 72), (7, 200), (2048, 2048), (300, 1000), (96, 8192), (20000, 128)])
def test_few_rows(M, N, K):
    A, W = operands(M + N, M + 3, N, K)
    rows = np.random.default_rng(M).permutation(M + 3)[:M].astype(np.int32)
    ref, tol = product(A[rows], W[0])
    lda = K + (1 if M == 3 else 0)                       # rows off the 16-byte grid
    wide = np.zeros((M + 3, lda), np.float32)
    wide[:, :K] = A
    a, w, r = gk.from_numpy(wide), dev_w(W[0]), gk.from_numpy(rows)
    c = gk.from_numpy(np.full((M, N + 1), 7.0, np.float32))
    if M <= 8:
        api.gemm_few_rows_f32(a.device_ptr, lda, r.device_ptr, w.device_ptr, 2, 0, c.device_ptr, N + 1, M, N, K, None, min(M, max(1, 40960 // K)), 0, 1.0,
                              0.0, None)
    else:
        api.gemm_rows_f32(a.device_ptr, lda, r.device_ptr, w.device_ptr, 2, 0, c.device_ptr, N + 1, M, N, K, None, 1, M, 0, 1.0, 0.0, None)
    out = c.to_numpy()
    assert (np.abs(out[:, :N] - ref) <= tol + 1e-6).all()
    assert (out[:, N:] == 7.0).all()
    no_wait_error()


@pytest.mark.parametrize("groups,per", [([0], 1), ([2, 0, -1, 2, 4], 1), ([-1, -1], 1), ([3, 1], 4), (list(range(5)) * 9, 1)])
@pytest.mark.parametrize("epi", [0, 1, 6])
def test_few_rows_with_their_own_matrices(groups, per, epi):
    E, N, K, M = 5, 140, 136, len(groups) * per
    A, W = operands(M, M, N, K, E)
    grp = np.repeat(groups, per).astype(np.int32)
    cols = N // 2 if epi == 1 else N
    a, w, g = gk.from_numpy(A), dev_w(W), gk.from_numpy(grp)
    c = gk.from_numpy(np.full((M, cols), 7.0, np.float32))
    api.gemm_few_rows_f32(a.device_ptr, K, None, w.device_ptr, 2, N * K, c.device_ptr, cols, M, N, K, g.device_ptr, per, epi, 1.0, 0.0, None)
    out = c.to_numpy()
    for m in range(M):
        if grp[m] < 0:
            assert (out[m] == 7.0).all()
            continue
        z, tol = product(A[m:m + 1], W[grp[m]])
        z, tol = z[0], tol[0]
        if epi == 1:
            u = z[1::2]
            z = z[0::2] * sigmoid(z[0::2]) * u
            tol = 2.0 * (1.0 + np.abs(u) + np.abs(z)) * np.maximum(tol[0::2], tol[1::2])
        if epi == 6:
            tol = 2.0 * (np.maximum(z, 0) + tol) * tol
            z = np.maximum(z, 0) ** 2
        assert (np.abs(out[m] - z) <= tol + 1e-6).all()
    no_wait_error()


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("epi", [0, 4, 10])
def test_few_rows_batches(M, epi):
    H, N, K = 6, 200, 72
    A, W = operands(M, M, N, H * K)
    W = bf16(np.random.default_rng(1).standard_normal((H, N, K)).astype(np.float32) / np.sqrt(K))
    old = np.random.default_rng(2).standard_normal((M, H * N)).astype(np.float32)
    gate = np.random.default_rng(3).standard_normal((M, H * N)).astype(np.float32)
    cs = np.random.default_rng(4).standard_normal(N).astype(np.float32)
    a, w, c, g, s = gk.from_numpy(A), dev_w(W), gk.from_numpy(old), gk.from_numpy(gate), gk.from_numpy(cs)
    aux = (g.device_ptr, 0, None, H * N, 0) if epi == 10 else (None, 0, None, 0, 0)
    api.gemm_seq_f32(a.device_ptr, H * K, K, w.device_ptr, 2, N * K, c.device_ptr, H * N, N, M, N, K, H, epi, 0.0, 0.0, s.device_ptr, aux[0], aux[1],
                     aux[2], aux[3], aux[4], M, None)
    out = c.to_numpy()
    for h in range(H):
        z, tol = product(A[:, h * K:(h + 1) * K], W[h])
        sl = slice(h * N, (h + 1) * N)
        if epi == 4:
            z, tol = old[:, sl] + cs * z, tol * np.abs(cs)
        if epi == 10:
            z = z * sigmoid(gate[:, sl])
        assert (np.abs(out[:, sl] - z) <= tol + 1e-6).all()
    no_wait_error()


@pytest.mark.parametrize("M", [24, 40, 200])
@pytest.mark.parametrize("N,K", [(140, 1024), (1090, 2056), (2, 4096)])
@pytest.mark.parametrize("epi", [1, 4])
def test_rows_beyond_n_with_shared_k(M, N, K, epi):
    """k shared by a cluster and a last column tile that is not full: lanes beyond N skip their stores, and the block still meets the
    others at the closing barrier as whole warps"""
    A, W = operands(M + N, M, N, K)
    z, tol = product(A, W[0])
    cols = N // 2 if epi == 1 else N
    old = np.random.default_rng(1).standard_normal((M, cols)).astype(np.float32)
    cs = np.random.default_rng(2).standard_normal(N).astype(np.float32)
    a, w, c, s = gk.from_numpy(A), dev_w(W[0]), gk.from_numpy(old), gk.from_numpy(cs)
    api.gemm_seq_f32(a.device_ptr, K, 0, w.device_ptr, 2, 0, c.device_ptr, cols, 0, M, N, K, 1, epi, 0.0, 0.0, s.device_ptr, None, 0, None, 0, 0, 0, None)
    if epi == 1:
        g, u = z[:, 0::2], z[:, 1::2]
        ref = g * sigmoid(g) * u
        tol = 2.0 * (1.0 + np.abs(u) + np.abs(g)) * np.maximum(tol[:, 0::2], tol[:, 1::2])
    else:
        ref, tol = old + cs * z, tol * np.abs(cs)
    assert (np.abs(c.to_numpy() - ref) <= tol + 1e-6 * (1 + np.abs(ref))).all()
    no_wait_error()


@pytest.fixture
def programmatic_launch():
    api.set_pdl(1)
    yield
    api.set_pdl(0)


def chain(ws, x, bufs, rows):
    """x -> w0 -> w1 -> ... and back into x's shape, every product reading what the one before wrote"""
    for _ in range(2):
        src, k = x, ws[0].shape[1]
        for w, b in zip(ws, bufs):
            llm.LinearRows(w).forward(src.device_ptr, k, rows, b.device_ptr, w.shape[0])
            src, k = b, w.shape[0]
    return src


@pytest.mark.parametrize("rows", [8, 16, 17, 60, 300, 1500])
def test_chained_products_under_programmatic_launch(rows, programmatic_launch):
    """the activations' rounding lets its dependents start early, clusters carry the launch attribute, work memory goes from product to
    product: the bits are those of plain launches, eagerly and in a replayed graph"""
    from pygpukit_b200.core.stream import CudaGraph, Stream
    sizes = [512, 2048, 648, 1536, 520, 512]             # every product on tcgen05
    rng = np.random.default_rng(rows)
    ws = [dev_w(bf16(rng.standard_normal((n, k)) / np.sqrt(k))) for k, n in zip(sizes, sizes[1:])]
    x = gk.from_numpy(rng.standard_normal((rows, sizes[0])).astype(np.float32))

    def buffers():
        return [gk.zeros((rows, n), gk.float32) for n in sizes[1:]]

    api.set_pdl(0)
    plain = buffers()
    chain(ws, x, plain, rows)
    ref = [b.to_numpy() for b in plain]
    api.set_pdl(1)
    for _ in range(5):
        got = buffers()
        chain(ws, x, got, rows)
        assert all((a == b.to_numpy()).all() for a, b in zip(ref, got))
    st, g, got = Stream(), CudaGraph(), buffers()
    with g.capture(st):
        chain(ws, x, got, rows)
    for _ in range(3):
        for b in got:
            b.copy_from_numpy(np.zeros(b.shape, np.float32))
        g.replay(st)
        st.synchronize()
        assert all((a == b.to_numpy()).all() for a, b in zip(ref, got))
    assert np.isfinite(ref[-1]).all() and np.abs(ref[-1]).max() > 0
    no_wait_error()


@pytest.mark.parametrize("M,N,K", [(17, 7, 648), (33, 257, 520), (64, 128, 456), (128, 129, 392), (129, 1023, 1032), (257, 640, 448), (272, 384, 1000), (1999, 272, 456)])
def test_rows_of_longer_k(M, N, K):
    """the tile heights, column tails and k tails of test_rows where the product runs on tcgen05"""
    test_rows(M, N, K)


@pytest.mark.parametrize("counts,N,K", [([30, 0, 70, 1, 9], 130, 712), ([300, 16, 0, 17, 257, 1], 256, 640), ([0, 0, 5], 64, 584),
                                        ([1] * 40, 96, 640), ([0] * 7, 96, 640), ([3, 129] * 20, 64, 520)])
@pytest.mark.parametrize("extra", [0, 50])
def test_groups_of_longer_k(counts, N, K, extra):
    test_groups(counts, N, K, extra)


@pytest.mark.parametrize("M,H,N,K,pad", [(40, 3, 96, 512, 0), (70, 5, 512, 384, 8), (260, 2, 130, 456, 4), (33, 4, 64, 520, 3)])
def test_batches_of_longer_k(M, H, N, K, pad):
    test_batches(M, H, N, K, pad)


@pytest.mark.parametrize("M,N,K", [(20, 128, 312), (20, 128, 352), (500, 2048, 216), (500, 2048, 240), (4, 4096, 1016), (4, 4096, 1024), (2, 4096, 2048)])
def test_both_sides_of_the_lines(M, N, K):
    """sizes just below and above the lines between the two forms: the same product"""
    A, W = operands(M + K, M, N, K)
    ref, tol = product(A, W[0])
    a, w, c = gk.from_numpy(A), dev_w(W[0]), gk.zeros((M, N), gk.float32)
    llm.LinearRows(w).forward(a.device_ptr, K, M, c.device_ptr, N)
    assert (np.abs(c.to_numpy() - ref) <= tol + 1e-6).all()
    no_wait_error()


def free_bytes():
    f, t = C.c_size_t(), C.c_size_t()
    api.mem_info(C.byref(f), C.byref(t))
    return f.value


def test_idle_work_memory_goes_back():
    """256 MB of rounded rows that a captured product allocates, and as many of plain ones: with the device again once they are idle"""
    from pygpukit_b200.core.stream import CudaGraph, Stream
    M, N, K = 1 << 16, 256, 2048
    a, w, c = gk.zeros((M, K), gk.float32), dev_w(np.ones((N, K))), gk.zeros((M, N), gk.float32)
    lin, st = llm.LinearRows(w), Stream()

    def captured():
        g = CudaGraph()
        with g.capture(st):
            lin.forward(a.device_ptr, K, M, c.device_ptr, N)
        g.replay(st)
        st.synchronize()
        return g

    def plain():
        lin.forward(a.device_ptr, K, M, c.device_ptr, N)
        api.device_sync()

    for make in (captured, plain):
        keep = make()                                    # (whatever the first one keeps for good)
        del keep
        api.mem_trim()
        before = free_bytes()
        keep = make()
        assert before - free_bytes() >= 200 << 20
        del keep
        api.mem_trim()
        assert before - free_bytes() <= 32 << 20
    plain()
    assert (c.to_numpy() == 0).all()


@pytest.mark.parametrize("M", [1, 8, 40, 300])
def test_products_see_weights_and_rows_written_by_the_launch_before(M):
    """Launches are brought to the SMs while the one before drains: weights and activations that the kernel just before has written are
    the ones that the product reads, in every form (streaming GEMV, few rows, many rows), call after call without a wait."""
    K, N, rounds = 1024, 2048, 6
    rng = np.random.default_rng(M)
    W = [gk.from_numpy(rng.standard_normal((N, K)).astype(np.float32)) for _ in range(rounds)]
    X = [gk.from_numpy(rng.standard_normal((M, K)).astype(np.float32)) for _ in range(rounds)]

    def run(wait):
        w, x, xb = gk.zeros((N, K), gk.bfloat16), gk.zeros((M, K), gk.float32), gk.zeros((M, K), gk.bfloat16)
        rows, gemv = [gk.zeros((M, N), gk.float32) for _ in range(rounds)], [gk.zeros((M, N), gk.bfloat16) for _ in range(rounds)]
        layer = llm.LinearRows(w)
        for i in range(rounds):
            api.cast(X[i].device_ptr, x.device_ptr, M * K, 0, 0, None)
            api.cast(W[i].device_ptr, w.device_ptr, N * K, 0, 2, None)
            if wait:
                api.device_sync()
            layer.forward(x.device_ptr, K, M, rows[i].device_ptr, N)
            if M <= 8:
                api.cast(X[i].device_ptr, xb.device_ptr, M * K, 0, 2, None)
                api.cast(W[rounds - 1 - i].device_ptr, w.device_ptr, N * K, 0, 2, None)
                if wait:
                    api.device_sync()
                api.gemv_bf16(xb.device_ptr, w.device_ptr, gemv[i].device_ptr, M, K, N, None)
        return [a.to_numpy() for a in rows + gemv]

    for a, b in zip(run(True), run(False)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("M,N,K", [(17, 200, 520), (31, 129, 72), (32, 2048, 2048), (33, 130, 456), (64, 2048, 2048), (65, 2056, 2048), (255, 72, 1000), (256, 512, 1024),
                                   (257, 512, 1024), (128, 24, 8192)])
def test_blocks_of_few_rows(M, N, K):
    """accumulators of 32 rows, blocks of them whose last one is not full, k cut over a cluster, and sizes beside the line to the product of many rows"""
    test_rows(M, N, K)


# rows of few (17, 200 x 512), of tcgen05 (600, 300 x 2048, cut k and not), of the tiles (short k, k no multiple of 8, unaligned rows)
@pytest.mark.parametrize("M,N,K,batch,pad", [(17, 136, 520, 1, 0), (200, 512, 256, 2, 4), (600, 1034, 512, 1, 8), (300, 128, 2048, 3, 8), (300, 130, 2048, 1, 3),
                                             (70, 64, 40, 2, 0), (70, 66, 44, 1, 1), (40, 64, 203, 1, 0)])
@pytest.mark.parametrize("epi", [0, 1, 3, 5, 6, 8, 10])
def test_bfloat16_rows_between_products(M, N, K, batch, pad, epi):
    """rows of A as the product would round them, and C rounded as the next product would: the bits of float32 rows"""
    A, W = operands(M + N, M, N, K * 1, batch)
    lda, F = K + pad, N // 2 if epi in (1, 3, 7) else N
    A = np.pad(A, ((0, 0), (0, pad)))
    rng = np.random.default_rng(5)
    table = gk.from_numpy(rng.standard_normal((M, F * batch + 3)).astype(np.float32))
    rows = gk.from_numpy(np.arange(M, dtype=np.int32))
    a32, a16, w = gk.from_numpy(A), dev_w(bf16(A)), dev_w(W)

    def run(x16, out16):
        c = gk.from_numpy(np.zeros((M, F * batch + 2), np.uint16 if out16 else np.float32))
        api.gemm_seq_f32((a16 if x16 else a32).device_ptr, lda, 0, w.device_ptr, 2 + 16 * x16 + 32 * out16, N * K if batch > 1 else 0, c.device_ptr,
                         F * batch + 2, F if batch > 1 else 0, M, N, K, batch, epi, 1.5, 2.0, None, table.device_ptr, 0, rows.device_ptr, F * batch + 3, 1, 0, None)
        return c.to_numpy()

    want = run(0, 0)
    assert np.array_equal(run(1, 0), want)
    assert np.array_equal(run(0, 1), bf16(want).view(np.uint32) >> 16) and np.array_equal(run(1, 1), bf16(want).view(np.uint32) >> 16)
    no_wait_error()


@pytest.mark.parametrize("counts,N,K", [([30, 0, 70, 1, 9], 130, 72), ([300, 16, 0, 17, 257, 1], 256, 128), ([700, 3, 254, 130], 384, 1032), ([0, 0, 5], 64, 200),
                                        ([1] * 40, 96, 2048), ([3, 129] * 20, 64, 97)])
@pytest.mark.parametrize("gather", [False, True])
def test_bfloat16_rows_of_groups(counts, N, K, gather):
    E, R = len(counts), sum(counts)
    A, W = operands(R + N, R, N, K, E)
    off, src = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32), np.random.default_rng(R).integers(0, R, R + 9).astype(np.int32)
    src[R:] = 1 << 30                                    # rows behind the last group name nothing
    a32, a16, w, o, s = gk.from_numpy(A), dev_w(bf16(A)), dev_w(W), gk.from_numpy(off), gk.from_numpy(src)
    lin = llm.LinearRows(w, epilogue=1)

    def run(x16, out16):
        c = gk.from_numpy(np.zeros((R, N // 2), np.uint16 if out16 else np.float32))
        lin.forward_grouped((a16 if x16 else a32).device_ptr, K, c.device_ptr, N // 2, s.device_ptr if gather else None, o.device_ptr, max(counts),
                            R + (9 if gather else 0), x16=x16, out16=out16)
        return c.to_numpy()

    want = run(0, 0)
    assert np.array_equal(run(1, 0), want)
    assert np.array_equal(run(0, 1), bf16(want).view(np.uint32) >> 16) and np.array_equal(run(1, 1), bf16(want).view(np.uint32) >> 16)
    no_wait_error()


@pytest.mark.parametrize("M,N,K", [(1, 2000, 2050), (2, 900, 3001), (4, 1024, 746), (7, 514, 1007), (8, 130, 843), (8, 6000, 1004), (9, 64, 161), (17, 300, 163), (33, 130, 1001),
                                   (200, 70, 167), (300, 515, 514), (1000, 256, 1002)])
@pytest.mark.parametrize("off", [0, 1, 2])
def test_matrices_off_the_boundaries(M, N, K, off):
    """k of any number, matrices from any element on: brought to boundaries first, for one row up; what lies around the matrix is not read into a sum"""
    A, W = operands(M + N, M, N, K)
    ref, tol = product(A, W[0])
    around = np.full(N * K + 16, np.inf, np.float32)
    around[off:off + N * K] = W[0].ravel()
    w, a, c = dev_w(around), gk.from_numpy(np.pad(A, ((0, 0), (0, 1)), constant_values=np.inf)), gk.from_numpy(np.full((M, N), 7.0, np.float32))
    if M <= 8:
        api.gemm_few_rows_f32(a.device_ptr, K + 1, None, w.device_ptr + 2 * off, 2, 0, c.device_ptr, N, M, N, K, None, M, 0, 1.0, 0.0, None)
    else:
        api.gemm_rows_f32(a.device_ptr, K + 1, None, w.device_ptr + 2 * off, 2, 0, c.device_ptr, N, M, N, K, None, 1, M, 0, 1.0, 0.0, None)
    assert (np.abs(c.to_numpy() - ref) <= tol + 1e-6).all()
    no_wait_error()


@pytest.mark.parametrize("M", [3, 20, 300])
def test_batches_off_the_boundaries(M):
    """products side by side whose matrices start anywhere"""
    batch, N, K = 3, 66, 1101
    A, W = operands(M, M, N, K * 1, batch)
    a, w, c = gk.from_numpy(A), dev_w(W), gk.from_numpy(np.zeros((M, batch * N), np.float32))
    api.gemm_seq_f32(a.device_ptr, K, 0, w.device_ptr, 2, N * K, c.device_ptr, batch * N, N, M, N, K, batch, 0, 1.0, 0.0, None, None, 0, None, 0, 0, M if M <= 8 else 0, None)
    for b in range(batch):
        ref, tol = product(A, W[b])
        assert (np.abs(c.to_numpy()[:, b * N:(b + 1) * N] - ref) <= tol + 1e-6).all()
    no_wait_error()


@pytest.mark.parametrize("M,N,K", [(9, 66, 31), (16, 128, 32), (17, 130, 33), (64, 70, 100), (101, 802, 212), (1000, 700, 65), (1025, 1000, 40)])
@pytest.mark.parametrize("epi", [0, 6, 7])
def test_float32_rows_sum_in_the_order_of_k(M, N, K, epi):
    """(more than 64 columns: up to there the router's kernel serves plain products) both tile heights: every sum is the chain of fused multiply-adds over k (float64 products rounded once per step), bit for bit without an activation"""
    A, W = operands(M + N, M, N, K)
    W = W[0] + np.float32(1e-4)
    F = N // 2 if epi == 7 else N
    a, w, c = gk.from_numpy(A), gk.from_numpy(W), gk.from_numpy(np.zeros((M, F), np.float32))
    api.gemm_rows_f32(a.device_ptr, K, None, w.device_ptr, 0, 0, c.device_ptr, F, M, N, K, None, 1, M, epi, 1.0, 0.0, None)
    z = np.zeros((M, N), np.float32)
    for k in range(K):                                   # a float64 product of float32 is exact, its sum with z rounds twice at worst: half a unit in 2^-29 of all cases
        z = (A[:, k:k + 1].astype(np.float64) * W[:, k].astype(np.float64) + z).astype(np.float32)
    got = c.to_numpy()
    if epi == 0:
        assert (got != z).mean() < 1e-4 and np.allclose(got, z, rtol=1e-6, atol=1e-6)
    else:
        z = z.astype(np.float64)
        ref = np.maximum(z, 0) ** 2 if epi == 6 else gelu_tanh(z[:, 0::2]) * z[:, 1::2]
        assert np.allclose(got, ref, rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("M,N,K", [(9, 1, 1), (17, 4, 127), (30, 5, 128), (16, 18, 132), (33, 64, 260), (100, 8, 1023), (12, 17, 2048)])
def test_router_logits_by_fours_and_one_by_one(M, N, K):
    """float32 rows of few columns, k that is and is not a multiple of a lane's four and of a warp's 128; each lane adds ceil(K / 32) + 4 products, five
    more sums join the lanes: so many half units of 2^-24, twice for products rounded into sums"""
    A, W = operands(M + N, M, N, K)
    W = W[0] + np.float32(1e-4)
    a, w, c = gk.from_numpy(A), gk.from_numpy(W), gk.from_numpy(np.zeros((M, N), np.float32))
    api.gemm_rows_f32(a.device_ptr, K, None, w.device_ptr, 0, 0, c.device_ptr, N, M, N, K, None, 1, M, 0, 1.0, 0.0, None)
    ref, tol = A.astype(np.float64) @ W.astype(np.float64).T, (K / 32 + 10) * 2.0 ** -23 * (np.abs(A.astype(np.float64)) @ np.abs(W.astype(np.float64)).T)
    assert (np.abs(c.to_numpy() - ref) <= tol).all()
