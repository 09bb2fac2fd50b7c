"""Mixtures of NVF4 experts over a few dozen tokens: routing with row lists, the experts' products and the weighted sum against the row-by-row
pipeline of the same layer; the fused gate/up product of a dense feed-forward; BF16 products of few columns."""
import numpy as np
import pytest

import pygpukit_b200 as gk
from pygpukit_b200 import llm
from pygpukit_b200._lib import api
from tests.util import f32, rand_bf16

pytestmark = pytest.mark.gpu


def _nvf4(rng, *shape):
    """codes of every value and scales of 2^-9 ... 2^-6, [.., K / 2, N] and [.., K / 32, N] for shape [.., K, N]"""
    *e, K, N = shape
    return (gk.from_numpy(rng.integers(0, 256, (*e, K // 2, N)).astype(np.uint8)),
            gk.from_numpy((rng.integers(0, 32, (*e, K // 32, N)) - 16 & 0x7f).astype(np.uint8) & 0x1f))


def _layer(rng, E, k, H, I, held=None, offset=0):
    cfg = llm.TransformerConfig(vocab_size=64, hidden_size=H, num_layers=1, num_heads=2, num_kv_heads=2, intermediate_size=I, _head_dim=64, norm_eps=1e-6,
                                rope_theta=1e4, tie_word_embeddings=False, num_experts=E, num_experts_per_tok=k, moe_intermediate_size=I)
    n = E if held is None else held
    st = {"format": "nvf4", "gate": _nvf4(rng, n, H, I), "up": _nvf4(rng, n, H, I), "down": _nvf4(rng, n, I, H)}
    return llm.MoELayer(cfg, gk.from_numpy(rand_bf16(rng, (E, H), 0.05)), stacked=st, expert_offset=offset)


@pytest.mark.parametrize("T,E,k,H,I", [(2, 8, 2, 128, 128), (15, 128, 8, 384, 256), (16, 16, 4, 2048, 128), (17, 64, 8, 256, 640), (33, 8, 8, 128, 384),
                                       (64, 512, 16, 256, 128), (64, 8, 2, 1024, 256), (3, 40, 5, 128, 128)])
def test_products_equal_the_row_by_row_pipeline(T, E, k, H, I):
    rng = np.random.default_rng(T * E + H)
    layer = _layer(rng, E, k, H, I)
    x, res = gk.from_numpy(rand_bf16(rng, (T, H))), gk.from_numpy(rand_bf16(rng, (T, H)))
    assert layer._as_products(x)
    for residual in (None, res):
        got = f32(layer.forward(x, residual=residual).to_numpy())
        b = layer._bufs[T]
        w, inv, first, active = (b[n].to_numpy() for n in ("weights", "reverse", "offsets", "active"))
        act = f32(b["act"].to_numpy())
        layer._as_products = lambda x: False
        ref = f32(layer.forward(x, residual=residual).to_numpy())
        del layer._as_products
        # routing: the same weights, rows and offsets, whole
        assert np.array_equal(w, b["weights"].to_numpy()) and np.array_equal(inv, b["reverse"].to_numpy()) and np.array_equal(first, b["offsets"].to_numpy())
        assert active[0] == (np.diff(first) > 0).sum() and np.array_equal(active[1:1 + active[0]], np.flatnonzero(np.diff(first)))
        # products: exact ones in float32, so an activation moves to its BF16 neighbour at most, and an output by what its activations moved
        a = f32(b["act"].to_numpy())
        assert (np.abs(act - a) <= 2.0 ** -6 * np.abs(a) + 2.0 ** -20 * np.abs(a).max()).all()
        assert np.linalg.norm(got - ref) <= 2.0 ** -8 * np.linalg.norm(ref)


@pytest.mark.parametrize("T,E,k,H,I", [(2, 8, 2, 128, 128), (19, 16, 4, 1152, 128)])
@pytest.mark.parametrize("at,res_at", [(1, 0), (0, 1), (4, 3)])
def test_rows_off_16_byte_boundaries_are_taken(T, E, k, H, I, at, res_at):
    """an output and a residual that start `at` elements behind a boundary: the bits of those on one, and nothing beside them is written"""
    rng = np.random.default_rng(T + at)
    layer = _layer(rng, E, k, H, I)
    x, r = gk.from_numpy(rand_bf16(rng, (T, H))), rand_bf16(rng, (T, H))
    room, res = gk.from_numpy(np.zeros(T * H + 16, np.uint16)), gk.from_numpy(np.concatenate([r.reshape(-1)[:8], r.reshape(-1), r.reshape(-1)[:8]])[8 - res_at:])
    view = lambda a, n: gk.GPUArray((T, H), gk.bfloat16, ptr=a.device_ptr + 2 * n, source=a)
    want = layer.forward(x, residual=gk.from_numpy(r)).to_numpy()
    got = layer.forward(x, out=view(room, at), residual=view(res, res_at))
    assert got.device_ptr % 16 == 2 * at and np.array_equal(got.to_numpy(), want)
    room = room.to_numpy()
    assert (room[:at] == 0).all() and (room[at + T * H:] == 0).all()


@pytest.mark.parametrize("offset,held", [(0, 3), (5, 3), (2, 6)])
def test_rows_of_experts_held_elsewhere_are_zeros(offset, held):
    """The rows of the experts that are here have the bits of the whole layer's, the others are zeros."""
    rng = np.random.default_rng(5)
    T, E, k, H, I = 9, 8, 3, 256, 128
    layer = _layer(rng, E, k, H, I)
    x = gk.from_numpy(rand_bf16(rng, (T, H)))
    layer.forward(x)
    b = layer._bufs[T]
    down, first = b["down"].to_numpy().copy(), b["offsets"].to_numpy()
    cut = lambda a: gk.from_numpy(np.ascontiguousarray(a.to_numpy()[offset:offset + held]))
    part = llm.MoELayer(layer.config, layer.gate.weight, stacked={"format": "nvf4", **{n: tuple(cut(a) for a in layer._w[n]) for n in ("gate", "up", "down")}},
                        expert_offset=offset)
    part.forward(x)
    got = part._bufs[T]["down"].to_numpy()
    lo, hi = first[offset], first[offset + held]
    assert np.array_equal(got[lo:hi], down[lo:hi]) and (got[:lo] == 0).all() and (got[hi:] == 0).all()


@pytest.mark.parametrize("M", [5, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("K,I", [(128, 64), (256, 1024), (1920, 320), (4096, 128)])
def test_fused_gate_up_equals_product_and_activation(M, K, I):
    rng = np.random.default_rng(M + K)
    data, scale = _nvf4(rng, K, 2 * I)
    x = gk.from_numpy(rand_bf16(rng, (M, K)))
    gu, two, one = gk.empty((M, 2 * I), gk.bfloat16), gk.empty((M, I), gk.bfloat16), gk.empty((M, I), gk.bfloat16)
    api.gemm_nvf4_bf16_tc(x.device_ptr, data.device_ptr, scale.device_ptr, gu.device_ptr, M, K, 2 * I, 1.0, None, None, None)
    api.swiglu_interleaved8_bf16(gu.device_ptr, two.device_ptr, M, I, None)
    api.gemv_nvf4_swiglu_bf16(x.device_ptr, data.device_ptr, scale.device_ptr, one.device_ptr, M, K, 2 * I, None)
    assert np.array_equal(one.to_numpy(), two.to_numpy())


@pytest.mark.parametrize("bias,residual", [(False, False), (True, True)])
def test_bf16_rows_beyond_a_grid(bias, residual):
    """more blocks of 16 rows than a grid has places for"""
    rng = np.random.default_rng(1)
    M, K, N = 16 * 65535 + 21, 16, 3
    A, B, bb, rr = rand_bf16(rng, (M, K)), rand_bf16(rng, (N, K)), rand_bf16(rng, (N,)), rand_bf16(rng, (M, N))
    a, b, bd, rd, c = (gk.from_numpy(v) for v in (A, B, bb, rr, np.zeros((M, N), np.uint16)))
    api.gemv_bf16_ex(a.device_ptr, b.device_ptr, c.device_ptr, M, K, N, bd.device_ptr if bias else None, rd.device_ptr if residual else None, None)
    x, y = f32(A).astype(np.float64), f32(B).astype(np.float64)
    ref = x @ y.T
    s = ref + bias * f32(bb).astype(np.float64)
    out = s + residual * f32(rr).astype(np.float64)
    # as below: one rounding of the sum, one more behind the bias and one behind the residual
    assert (np.abs(f32(c.to_numpy()) - out) <= 2.0 ** -7 * (np.abs(ref) + np.abs(s) + np.abs(out)) + 2.0 ** -20 * (np.abs(x) @ np.abs(y).T)).all()


@pytest.mark.parametrize("M,K,N", [(5, 16, 1), (15, 3456, 128), (16, 512, 8), (17, 2048, 130), (64, 4096, 33), (64, 48, 4096), (33, 1040, 2048)])
def test_bf16_rows_against_float64(M, K, N):
    """exact products, float32 sums of 32 k and over the 16 warps, one rounding to BF16 (and one more behind the bias)"""
    rng = np.random.default_rng(M + K + N)
    A, B, bias, res = rand_bf16(rng, (M, K)), rand_bf16(rng, (N, K)), rand_bf16(rng, (N,)), rand_bf16(rng, (M, N))
    a, b, bb, rr, c = (gk.from_numpy(v) for v in (A, B, bias, res, np.zeros((M, N), np.uint16)))
    x, y = f32(A).astype(np.float64), f32(B).astype(np.float64)
    ref, size = x @ y.T, np.abs(x) @ np.abs(y).T
    api.gemv_bf16(a.device_ptr, b.device_ptr, c.device_ptr, M, K, N, None)
    assert (np.abs(f32(c.to_numpy()) - ref) <= 2.0 ** -8 * np.abs(ref) + 2.0 ** -20 * size).all()
    api.gemv_bf16_ex(a.device_ptr, b.device_ptr, c.device_ptr, M, K, N, bb.device_ptr, rr.device_ptr, None)
    s = ref + f32(bias).astype(np.float64)
    out = s + f32(res).astype(np.float64)
    assert (np.abs(f32(c.to_numpy()) - out) <= 2.0 ** -7 * (np.abs(ref) + np.abs(s) + np.abs(out)) + 2.0 ** -20 * size).all()


def test_slots_without_a_finite_choice_share_a_row():
    """fewer finite logits than slots: the slots left name expert 0 with weight zero, as in the row-by-row pipeline"""
    rng = np.random.default_rng(3)
    T, E, k, H, I = 40, 8, 4, 128, 128
    layer = _layer(rng, E, k, H, I)
    z = rng.standard_normal((T, E)).astype(np.float32)
    z[:, 2:] = -np.inf
    from tests.util import bf16
    layer.gate.forward = lambda x, out: out.copy_from(logits) if hasattr(out, "copy_from") else api.memcpy_d2d(out.device_ptr, logits.device_ptr, out.nbytes, None)
    logits = gk.from_numpy(bf16(z))
    x = gk.from_numpy(rand_bf16(rng, (T, H)))
    got = f32(layer.forward(x).to_numpy())
    layer._as_products = lambda x: False
    ref = f32(layer.forward(x).to_numpy())
    assert np.isfinite(got).all() and np.linalg.norm(got - ref) <= 2.0 ** -8 * np.linalg.norm(ref)


@pytest.mark.parametrize("E,k", [(1, 1), (8, 8), (128, 8), (129, 32), (512, 6)])
def test_routing_of_unusual_logits(E, k):
    """ties, zeros of either sign, infinities, NaN, values at the limit of what is chosen, and fewer candidates than slots"""
    rng = np.random.default_rng(E)
    for case in range(6):
        z = np.round(rng.standard_normal(E) * 2) / 2 if case else np.full(E, np.nan)
        if case == 1:
            z = np.where(rng.random(E) < 0.5, 0.0, -0.0)
        if case == 2:
            z[rng.random(E) < 0.9] = -np.inf
        if case == 3:
            z[rng.random(E) < 0.5] = np.nan
        if case == 4:
            z = np.where(rng.random(E) < 0.8, -1e30, -9e29)
        bits = (np.asarray(z, np.float32).view(np.uint32) >> 16).astype(np.uint16)
        v = (bits.astype(np.uint32) << 16).view(np.float32)
        left, ids, vals = {e: v[e] for e in range(E) if v[e] > np.float32(-1e30)}, [], []
        for _ in range(k):
            e = min(left, key=lambda i: (-left[i], i)) if left else 0
            ids.append(e)
            vals.append(left.pop(e) if left else np.float32(-1e30))
        zd, wd, idd, rd = gk.from_numpy(bits), gk.from_numpy(np.zeros(k, np.uint16)), gk.from_numpy(np.full(k, -1, np.int32)), gk.from_numpy(np.full(k, -1, np.int32))
        api.moe_route_t1(zd.device_ptr, wd.device_ptr, idd.device_ptr, rd.device_ptr, E, k, None)
        assert idd.to_numpy().tolist() == ids and rd.to_numpy().tolist() == ids
        ex = np.exp(np.asarray(vals, np.float64) - max(vals))
        assert np.abs((wd.to_numpy().astype(np.uint32) << 16).view(np.float32) - ex / ex.sum()).max() <= 2.0 ** -8
