"""The work that is measured when this package's speed is compared between two of its states: layers of quantised decoders
(decoding one token or a batch, and prompts) and layers of the token-major family (prompts and decoding), through the calls
that a program makes.  Sizes are those of the named configurations (`llm.config.named_config`) and of the layered benchmark
(`scripts/bench_layered.py`); `draw` spreads them over the ranges around those, odd ones among them.

Every case returns whole outputs: a layer's rows, the cache rows it wrote, a model's logits.  `exact` restates the same
mathematics in float64 on the same inputs, which come from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pygpukit_b200 import llm
from pygpukit_b200.core.array import GPUArray
from pygpukit_b200.core.dtypes import bfloat16, float32, uint8
from pygpukit_b200.llm.models.layered import StepContext

DEV = "cuda"
F64 = torch.float64
VOCAB = 32768                       # the layered benchmark's vocabulary


# ---------------------------------------------------------------------------------------------------- the cases
def listed() -> list[dict]:
    return [
        # the fused q/k/v projection of an 8B decoder, one decoded token: the smallest call, latency counts
        dict(name="linear_fp8_m1", kind="linear_fp8", rows=1, k=4096, n=6144),
        # the feed-forward of a 70B decoder in NVF4, one decoded token: most of the bytes of the headline decode step
        dict(name="mlp_nvf4_m1", kind="mlp_nvf4", rows=1, hidden=8192, inter=28672),
        # the feed-forward of an 8B decoder in FP8, 64 sequences decoding together
        dict(name="mlp_fp8_m64", kind="mlp_fp8", rows=64, hidden=4096, inter=14336),
        # the attention layer of an 8B decoder (projections in FP8), one token over a context of 4096
        dict(name="attn_decode_4k", kind="attn_decode", seqs=1, ctx=4096, heads=32, kv_heads=8, hidden=4096, qk_norm=True),
        # a mixture-of-experts feed-forward with 128 NVF4 experts, eight chosen, one decoded token
        dict(name="moe_nvf4_t1", kind="moe_nvf4", tokens=1, hidden=2048, inter=768, experts=128, top=8),
        # a prompt through one layer of an FP8 decoder and its final norm and head, on the fixed cache
        dict(name="prompt_fp8_512", kind="prompt_fp8", tokens=512, hidden=4096, inter=14336, heads=32, kv_heads=8),
        # a fused projection of the token-major family over the rows of a prompt
        dict(name="rows_bf16_2000", kind="rows", dtype="bfloat16", rows=2000, k=2048, n=9216, epilogue=0),
        # a prompt through a chunked, gated attention layer with a tanh cap (grouped heads)
        dict(name="attn_prompt_2000", kind="attn_prompt", tokens=2000, requests=1, width=2048, heads=32, kv_heads=4, dim=128,
             chunk=1024, softcap=50.0),
        # a prompt through a latent attention layer
        dict(name="latent_prompt_2000", kind="latent_prompt", tokens=2000, requests=1, width=2048, heads=16, dim=128, rot=64,
             kv_rank=512, q_rank=768),
        # a prompt through a linear attention layer with a state per sequence
        dict(name="linear_prompt_2000", kind="linear_prompt", tokens=2000, requests=1, width=2048, heads=16, dim=128, vdim=128,
             taps=4),
        # the rows of a prompt through a mixture of experts with a gated shared one
        dict(name="experts_prompt_2000", kind="experts", tokens=2000, width=2048, experts=16, identity=2, top=4, ff=2048,
             shared_ff=2048),
        # a whole decode step of eight requests: latent and windowed attention, dense feed-forwards, logits
        dict(name="decode_step_8", kind="decode_step", requests=8, ctx=2000, width=2048, heads=16, kv_heads=4, dim=128,
             window=1024, rot=64, kv_rank=512, q_rank=768, ff=8192, side=256, times=2),
    ]


def _log(rng, lo: int, hi: int, step: int = 1) -> int:
    """a multiple of `step` in lo .. hi, spread over its logarithm"""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng) -> dict:
    kind = rng.choice(["linear_fp8", "mlp_nvf4", "mlp_fp8", "attn_decode", "moe_nvf4", "prompt_fp8", "rows", "rows", "attn_prompt",
                       "latent_prompt", "linear_prompt", "experts", "decode_step"])
    if kind == "linear_fp8":
        return dict(kind=kind, rows=_log(rng, 1, 64), k=_log(rng, 1024, 14336, 128), n=_log(rng, 1024, 14336, 128))
    if kind == "mlp_nvf4":
        return dict(kind=kind, rows=_log(rng, 1, 32), hidden=_log(rng, 1024, 8192, 128), inter=_log(rng, 1024, 28672, 128))
    if kind == "mlp_fp8":
        return dict(kind=kind, rows=_log(rng, 1, 64), hidden=_log(rng, 1024, 8192, 128), inter=_log(rng, 1024, 14336, 128))
    if kind == "attn_decode":
        seqs = _log(rng, 1, 32)
        heads, kv = rng.choice([(32, 8), (64, 8), (32, 4)])
        return dict(kind=kind, seqs=seqs, ctx=_log(rng, 100, 262144 // seqs if seqs > 8 else 32768), heads=heads, kv_heads=kv,
                    hidden=rng.choice([2048, 4096, 8192]), qk_norm=rng.random() < 0.5)
    if kind == "moe_nvf4":
        return dict(kind=kind, tokens=_log(rng, 1, 64), hidden=_log(rng, 1024, 4096, 128), inter=_log(rng, 512, 2048, 128),
                    experts=rng.choice([8, 16, 64, 128]), top=rng.choice([2, 4, 8]))
    if kind == "prompt_fp8":
        heads, kv = rng.choice([(32, 8), (16, 8), (32, 4)])
        return dict(kind=kind, tokens=_log(rng, 16, 512), hidden=rng.choice([2048, 4096]), inter=_log(rng, 2048, 12288, 128), heads=heads,
                    kv_heads=kv)
    if kind == "rows":
        if rng.random() < 0.2:               # the mode that keeps everything in float32
            return dict(kind=kind, dtype="float32", rows=_log(rng, 1, 1000), k=_log(rng, 200, 2048), n=_log(rng, 200, 3000, 2),
                        epilogue=rng.choice([0, 1, 6]))
        return dict(kind=kind, dtype="bfloat16", rows=_log(rng, 1, 4096), k=_log(rng, 256, 4096, rng.choice([1, 2, 8, 64])),
                    n=_log(rng, 256, 6144, rng.choice([2, 16, 128])), epilogue=rng.choice([0, 0, 1, 6, 7, 9]))
    if kind == "attn_prompt":
        heads, kv = rng.choice([(32, 4), (32, 8), (16, 4), (16, 16), (12, 3)])
        return dict(kind=kind, tokens=_log(rng, 20, 2000), requests=rng.choice([1, 1, 2, 3, 7]), width=rng.choice([1024, 2048]), heads=heads,
                    kv_heads=kv, dim=rng.choice([128, 128, 64, 96]), chunk=rng.choice([0, 256, 1000, 1024, 2048]),
                    softcap=rng.choice([0.0, 50.0]))
    if kind == "latent_prompt":
        return dict(kind=kind, tokens=_log(rng, 20, 2000), requests=rng.choice([1, 1, 2, 5]), width=rng.choice([1024, 2048]),
                    heads=rng.choice([8, 12, 16]), dim=128, rot=64, kv_rank=rng.choice([512, 256]), q_rank=rng.choice([512, 768]))
    if kind == "linear_prompt":
        return dict(kind=kind, tokens=_log(rng, 20, 2000), requests=rng.choice([1, 1, 2, 5]), width=rng.choice([1024, 2048]),
                    heads=rng.choice([8, 16]), dim=rng.choice([64, 128]), vdim=rng.choice([64, 128]), taps=4)
    if kind == "experts":
        experts = rng.choice([8, 16, 64, 128])
        return dict(kind=kind, tokens=_log(rng, 9, 2000), width=_log(rng, 512, 2048, 64), experts=experts, identity=rng.choice([0, 2]),
                    top=rng.choice([2, 4, 6]), ff=_log(rng, 256, 1536, 32), shared_ff=rng.choice([0, 512, 1000]))
    return dict(kind="decode_step", requests=_log(rng, 1, 24), ctx=_log(rng, 60, 3000), width=rng.choice([1024, 2048]), heads=16,
                kv_heads=rng.choice([4, 8]), dim=128, window=rng.choice([512, 1024]), rot=64, kv_rank=512, q_rank=768,
                ff=_log(rng, 2048, 8192, 128), side=256, times=rng.choice([1, 2]))


# ---------------------------------------------------------------------------------------------------- small helpers
_DT = {torch.bfloat16: bfloat16, torch.float32: float32, torch.uint8: uint8}


def _arr(t: torch.Tensor) -> GPUArray:
    """a torch tensor's memory as the package's array type"""
    return GPUArray(tuple(t.shape), _DT[t.dtype], ptr=t.data_ptr(), source=t)


class _Mem:
    def __init__(self, ptr, shape, typestr, owner):
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (ptr, False), "version": 3}
        self.owner = owner


def _view(a: GPUArray) -> torch.Tensor:
    """a package array's memory as a torch tensor"""
    if a.dtype.name == "bfloat16":
        return torch.as_tensor(_Mem(a.device_ptr, a.shape, "<i2", a), device=DEV).view(torch.bfloat16)
    return torch.as_tensor(_Mem(a.device_ptr, a.shape, "<f4", a), device=DEV)


class _Gen:
    """tensors of one case, in the order in which they are asked for"""

    def __init__(self, seed: int):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 7919 + 13)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.g, device=DEV) * std).to(dtype)

    def mat(self, *shape, gain=1.0, dtype=torch.bfloat16):
        return self.normal(*shape, std=gain / math.sqrt(shape[-1]), dtype=dtype)

    def around(self, c, n, spread=0.1, dtype=torch.float32):
        return (c + spread * torch.randn(n, generator=self.g, device=DEV)).to(dtype)

    def tokens(self, n, vocab=VOCAB):
        return torch.randint(0, vocab, (n,), generator=self.g, device=DEV).tolist()

    def fp8(self, n, k, gain=1.0):
        """E4M3 codes [n, k] with one bfloat16 scale per 128 x 128 block (largest magnitude on 448)"""
        w = torch.randn(n // 128, 128, k // 128, 128, generator=self.g, device=DEV) * (gain / math.sqrt(k))
        s = (w.abs().amax((1, 3)) / 448.0).to(torch.bfloat16)
        q = (w / s.float()[:, None, :, None]).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn)
        return q.reshape(n, k).view(torch.uint8), s

    def nvf4(self, k, n):
        """E2M1 codes [k / 2, n] (low nibble: even k) distributed like a normal block over its maximum, and one scale code per
        32 k: scales of 2^-7 (1 + m / 8)"""
        z = torch.special.ndtri((torch.arange(256, device=DEV, dtype=F64) + 0.5) / 256) * (6.0 / 2.4)
        code = (z.abs()[:, None] - _E2M1[None, :8].abs()).abs().argmin(1) + 8 * (z < 0)
        pair = (code[:, None] + 16 * code[None, :]).reshape(-1).to(torch.uint8)
        r = torch.randint(0, 65536, (k // 2 * n,), generator=self.g, device=DEV, dtype=torch.int32)
        data = pair.index_select(0, r).view(k // 2, n)
        scale = torch.randint(0, 8, (k // 32, n), generator=self.g, device=DEV, dtype=torch.uint8)
        return data, scale


_E2M1 = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0], dtype=F64,
                     device=DEV if torch.cuda.is_available() else "cpu")


def _fp8_f64(w, s) -> torch.Tensor:
    n, k = w.shape
    v = w.view(torch.float8_e4m3fn).to(torch.float32).to(F64).view(n // 128, 128, k // 128, 128)
    return (v * s.to(F64)[:, None, :, None]).reshape(n, k)


def _nvf4_times(x64, data, scale) -> torch.Tensor:
    """x [m, k] times the dequantised [k, n], a range of columns at a time"""
    k, n = 2 * data.shape[0], data.shape[1]
    out = []
    for c in range(0, n, 4096):
        d = data[:, c:c + 4096]
        m = d.shape[1]
        v = torch.stack([_E2M1[(d & 15).long()], _E2M1[(d >> 4).long()]], 1).view(k // 32, 32, m)
        s = torch.ldexp(torch.ones((), dtype=F64, device=DEV), torch.tensor(-7, device=DEV)) * (1.0 + (scale[:, c:c + 4096] & 7).to(F64) / 8)
        out.append(x64 @ (v * s[:, None, :]).view(k, m))
    return torch.cat(out, 1)


def _silu(z):
    return z * torch.sigmoid(z)


def _rms(x, w, eps, offset=0.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * (offset + w)


def _layer_norm(x, w, eps):
    mu = x.mean(-1, keepdim=True)
    return (x - mu) / torch.sqrt(((x - mu) ** 2).mean(-1, keepdim=True) + eps) * w


def _rope_half(x, pos, theta):
    """x [t, heads, d]: element i pairs with i + d / 2"""
    h = x.shape[-1] // 2
    f = (theta ** (-torch.arange(0, h, dtype=F64, device=DEV) / h))
    a = pos.to(F64)[:, None] * f
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    return torch.cat([x[..., :h] * c - x[..., h:] * s, x[..., h:] * c + x[..., :h] * s], -1)


def _rope_pairs(x, pos, base):
    """x [t, ..., d]: element 2i pairs with 2i + 1"""
    h = x.shape[-1] // 2
    a = pos.to(F64)[:, None] * base ** (-torch.arange(0, h, dtype=F64, device=DEV) / h)
    a = a.reshape((a.shape[0],) + (1,) * (x.ndim - 2) + (h,))
    c, s = torch.cos(a), torch.sin(a)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).reshape(x.shape)


def _split(total: int, parts: int) -> list[int]:
    """unequal portions of a ragged batch"""
    parts = min(parts, total)
    w = [i + 1 for i in range(parts)]
    n = [max(1, total * v // sum(w)) for v in w]
    n[-1] += total - sum(n)
    return n


def _requests(tokens: list[int], parts: int) -> list[list[int]]:
    out, at = [], 0
    for n in _split(len(tokens), parts):
        out.append(tokens[at:at + n])
        at += n
    return out


def _prompt_state(model, cfg, requests):
    model.init_cache(max_tokens=sum(len(r) for r in requests) + 64 * len(requests), slots=max(8, len(requests)))
    return dict(model=model, entries=[(i, r, [len(r) - 1]) for i, r in enumerate(requests)], end=list(range(len(requests))),
                rows=sum(len(r) for r in requests))


def _run_prompt(s):
    out, n = s["model"].step_device(s["entries"], end=s["end"])
    return {"logits": _view(out)[:n], "rows": _view(s["model"]._buf.x)[:s["rows"]]}


# ---------------------------------------------------------------------------------------------------- inputs
def _make(case: dict, seed: int) -> dict:
    """every tensor of a case, as torch tensors on the GPU"""
    g, kind = _Gen(seed), case["kind"]
    c = case
    if kind == "linear_fp8":
        return dict(x=g.normal(c["rows"], c["k"]), w=g.fp8(c["n"], c["k"]))
    if kind == "mlp_nvf4":
        return dict(x=g.normal(c["rows"], c["hidden"], std=0.5), gu=g.nvf4(c["hidden"], 2 * c["inter"]), down=g.nvf4(c["inter"], c["hidden"]))
    if kind == "mlp_fp8":
        return dict(x=g.normal(c["rows"], c["hidden"]), gate=g.fp8(c["inter"], c["hidden"]), up=g.fp8(c["inter"], c["hidden"]),
                    down=g.fp8(c["hidden"], c["inter"]))
    if kind == "attn_decode":
        H, G, S = c["heads"], c["kv_heads"], c["seqs"]
        return dict(x=g.normal(S, c["hidden"]), qkv=g.fp8((H + 2 * G) * 128, c["hidden"]), o=g.fp8(c["hidden"], H * 128),
                    qn=g.around(1.0, 128, dtype=torch.bfloat16), kn=g.around(1.0, 128, dtype=torch.bfloat16),
                    k=g.normal(S * G, c["ctx"], 128), v=g.normal(S * G, c["ctx"], 128))
    if kind == "moe_nvf4":
        E, H, I = c["experts"], c["hidden"], c["inter"]
        return dict(x=g.normal(c["tokens"], H), router=g.mat(E, H), gate=g.nvf4(E * H, I), up=g.nvf4(E * H, I), down=g.nvf4(E * I, H))
    if kind == "prompt_fp8":
        H, G, W, I = c["heads"], c["kv_heads"], c["hidden"], c["inter"]
        return dict(embed=g.normal(VOCAB, W), head=g.mat(VOCAB, W), n1=g.around(1.0, W, dtype=torch.bfloat16), n2=g.around(1.0, W, dtype=torch.bfloat16),
                    nf=g.around(1.0, W, dtype=torch.bfloat16), qkv=g.fp8((H + 2 * G) * 128, W), o=g.fp8(W, H * 128), gate=g.fp8(I, W),
                    up=g.fp8(I, W), down=g.fp8(W, I), tokens=g.tokens(c["tokens"]))
    if kind == "rows":
        dt = torch.bfloat16 if c["dtype"] == "bfloat16" else torch.float32
        return dict(x=g.normal(c["rows"], c["k"], dtype=torch.float32), w=g.mat(c["n"], c["k"], dtype=dt))
    if kind == "attn_prompt":
        W, H, G, D = c["width"], c["heads"], c["kv_heads"], c["dim"]
        return dict(embed=g.normal(VOCAB, W), head=g.mat(VOCAB, W), qkvg=g.mat(2 * H * D + 2 * G * D, W), o=g.mat(W, H * D),
                    qn=g.around(1.0, D), kn=g.around(1.0, D), n1=g.around(1.0, W), b1=g.around(0.0, W), nf=g.around(1.0, W), bf=g.around(0.0, W),
                    tokens=g.tokens(c["tokens"]))
    if kind == "latent_prompt":
        return dict(tokens=g.tokens(c["tokens"]), **_latent_tensors(g, c), embed=g.normal(VOCAB, c["width"]), head=g.mat(VOCAB, c["width"]),
                    en=g.around(0.0, c["width"]), n1=g.around(0.0, c["width"]), nf=g.around(0.0, c["width"]), s1=g.around(0.8, c["width"]))
    if kind == "linear_prompt":
        W, H, D, Dv = c["width"], c["heads"], c["dim"], c["vdim"]
        return dict(tokens=g.tokens(c["tokens"]), embed=g.normal(VOCAB, W), head=g.mat(VOCAB, W), n1=g.around(1.0, W), nf=g.around(1.0, W),
                    conv=g.normal(W, c["taps"], std=0.2, dtype=torch.float32), proj=g.mat(2 * H * D + 2 * H * Dv, W), o=g.mat(W, H * Dv),
                    on=g.around(1.0, H * Dv))
    if kind == "experts":
        W, E, F, S = c["width"], c["experts"], c["ff"], c["shared_ff"]
        t = dict(x=g.normal(c["tokens"], W, dtype=torch.float32), router=g.mat(E + c["identity"] + (1 if S else 0), W, dtype=torch.float32),
                 corr=g.around(0.0, E + c["identity"], spread=0.02), gu=g.mat(E, 2 * F, W), down=g.mat(E, W, F))
        if S:
            t.update(sgu=g.mat(2 * S, W), sdn=g.mat(W, S))
        return t
    W, H, G, D, F, sd = c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"], c["side"]
    pages = -(-(c["ctx"] + 1) // 64) * c["requests"]
    t = dict(embed=g.normal(VOCAB, W), head=g.mat(VOCAB, W), en=g.around(0.0, W), nf=g.around(0.0, W), side=g.normal(VOCAB, 2 * sd),
             tokens=g.tokens(c["requests"]), latent=_latent_tensors(g, c),
             win=dict(proj=g.mat(H * D + G * D + H, W), o=g.mat(W, H * D), qb=g.around(0.0, H * D), kb=g.around(0.0, G * D),
                      qn=g.around(1.0, H * D), kn=g.around(1.0, G * D)))
    for i in range(2):
        t[f"l{i}"] = dict(n1=g.around(0.0, W), s1=g.around(0.5, W), s2=g.around(0.5, W), gu=g.mat(2 * F, W), down=g.mat(W, F), sg=g.mat(sd, W),
                          sp=g.mat(W, sd), sn=g.around(0.5, W))
    t["pages"] = [dict(lat=g.normal(pages, 64, c["kv_rank"] + c["rot"]), k=g.normal(pages, G, 64, D), v=g.normal(pages, G, 64, D))
                  for _ in range(c["times"])]
    return t


def _latent_tensors(g: _Gen, c: dict) -> dict:
    W, H, D, R, kr, qr = c["width"], c["heads"], c["dim"], c["rot"], c["kv_rank"], c["q_rank"]
    return dict(lproj=g.mat(qr + kr + R + H, W), quq=g.mat(H * (D + R), qr), kab=g.normal(H, kr, D, std=kr ** -0.5), vup=g.mat(H, 128, kr),
                lo=g.mat(W, H * 128), lqn=g.around(1.0, qr), lcn=g.around(1.0, kr), sinks=g.around(0.0, H))


# ---------------------------------------------------------------------------------------------------- prepare
def _fp8_layer(p):
    return llm.LinearFP8(_arr(p[0]), _arr(p[1]))


def _mlp_config(hidden, inter, **kw):
    return llm.TransformerConfig(vocab_size=VOCAB, hidden_size=hidden, num_layers=1, num_heads=kw.pop("heads", 32),
                                 num_kv_heads=kw.pop("kv_heads", 8), intermediate_size=inter, _head_dim=128, norm_eps=1e-6,
                                 rope_theta=1e6, tie_word_embeddings=False, **kw)


def _latent_mixer(spec, t, layer):
    return llm.LatentAttentionMixer(spec, layer, llm.LinearRows(_arr(t["lproj"])), llm.LinearRows(_arr(t["quq"])),
                                    llm.LinearRows(_arr(t["kab"])), llm.LinearRows(_arr(t["vup"])), llm.LinearRows(_arr(t["lo"])),
                                    _arr(t["lqn"]), _arr(t["lcn"]), 1e-6, sinks=_arr(t["sinks"]))


def _latent_json(c):
    return {"type": "latent_attention", "mixer": {"heads": c["heads"], "dim": c["dim"], "rot_dim": c["rot"], "vdim": 128,
                                                  "kv_rank": c["kv_rank"], "q_rank": c["q_rank"], "scale": (c["dim"] + c["rot"]) ** -0.5,
                                                  "rot": {"dims": c["rot"], "base": 10000.0}}}


def _rms_1p(w):
    return llm.RowNorm("rmsnorm", _arr(w), None, 1e-6, offset=1.0)


def prepare(case: dict, seed: int) -> dict:
    c, kind, t = case, case["kind"], _make(case, seed)
    s = dict(case=case, t=t)
    if kind == "linear_fp8":
        s["y"] = torch.empty(c["rows"], c["n"], dtype=torch.bfloat16, device=DEV)
        s.update(layer=_fp8_layer(t["w"]), x=_arr(t["x"]), out=_arr(s["y"]))
    elif kind == "mlp_nvf4":
        s["y"] = torch.empty(c["rows"], c["hidden"], dtype=torch.bfloat16, device=DEV)
        gu = llm.LinearNVF4(_arr(t["gu"][0]), _arr(t["gu"][1]), c["hidden"], 2 * c["inter"])
        dn = llm.LinearNVF4(_arr(t["down"][0]), _arr(t["down"][1]), c["inter"], c["hidden"])
        s.update(layer=llm.MLP(_mlp_config(c["hidden"], c["inter"]), down_proj=dn, gate_up_proj=gu), x=_arr(t["x"]), out=_arr(s["y"]),
                 act=GPUArray((c["rows"], c["inter"]), bfloat16))
    elif kind == "mlp_fp8":
        s["y"] = torch.empty(c["rows"], c["hidden"], dtype=torch.bfloat16, device=DEV)
        s.update(layer=llm.MLP(_mlp_config(c["hidden"], c["inter"]), gate_proj=_fp8_layer(t["gate"]), up_proj=_fp8_layer(t["up"]),
                               down_proj=_fp8_layer(t["down"])), x=_arr(t["x"]), out=_arr(s["y"]), act=GPUArray((c["rows"], c["inter"]), bfloat16))
    elif kind == "attn_decode":
        H, G, S = c["heads"], c["kv_heads"], c["seqs"]
        cfg = _mlp_config(c["hidden"], 4 * c["hidden"], heads=H, kv_heads=G, max_position_embeddings=c["ctx"])
        norm = [llm.Norm(_arr(t[n]), None, "rmsnorm", 1e-6) if c["qk_norm"] else None for n in ("qn", "kn")]
        a = llm.Attention(None, None, None, _fp8_layer(t["o"]), cfg, q_norm=norm[0], k_norm=norm[1], qkv_proj=_fp8_layer(t["qkv"]))
        a.init_fixed_cache(c["ctx"], num_sequences=S)
        _view(a._k_cache).copy_(t["k"])
        _view(a._v_cache).copy_(t["v"])
        s["y"] = torch.empty(S, c["hidden"], dtype=torch.bfloat16, device=DEV)
        s["pos"] = torch.full((S,), c["ctx"] - 1, dtype=torch.int32, device=DEV)
        s["len"] = torch.full((S,), c["ctx"], dtype=torch.int32, device=DEV)
        from pygpukit_b200.core.dtypes import int32
        s.update(layer=a, x=_arr(t["x"]), out=_arr(s["y"]), kc=_view(a._k_cache), vc=_view(a._v_cache),
                 pos_arr=GPUArray((S,), int32, ptr=s["pos"].data_ptr(), source=s["pos"]),
                 len_arr=GPUArray((S,), int32, ptr=s["len"].data_ptr(), source=s["len"]),
                 qkv=GPUArray((S, (H + 2 * G) * 128), bfloat16), flat=GPUArray((S, H * 128), bfloat16))
    elif kind == "moe_nvf4":
        E, H, I = c["experts"], c["hidden"], c["inter"]
        cfg = _mlp_config(H, I, num_experts=E, num_experts_per_tok=c["top"], moe_intermediate_size=I)
        st = {"format": "nvf4"}
        for n, (k, w) in (("gate", (H, I)), ("up", (H, I)), ("down", (I, H))):
            st[n] = (_arr(t[n][0].view(E, k // 2, w)), _arr(t[n][1].view(E, k // 32, w)))
        s["y"] = torch.empty(c["tokens"], H, dtype=torch.bfloat16, device=DEV)
        s.update(layer=llm.MoELayer(cfg, _arr(t["router"]), stacked=st), x=_arr(t["x"]), out=_arr(s["y"]))
    elif kind == "prompt_fp8":
        W, T = c["hidden"], c["tokens"]
        cfg = _mlp_config(W, c["inter"], heads=c["heads"], kv_heads=c["kv_heads"], max_position_embeddings=T)
        rms = {n: llm.Norm(_arr(t[n]), None, "rmsnorm", 1e-6) for n in ("n1", "n2", "nf")}
        a = llm.Attention(None, None, None, _fp8_layer(t["o"]), cfg, qkv_proj=_fp8_layer(t["qkv"]))
        m = llm.MLP(cfg, gate_proj=_fp8_layer(t["gate"]), up_proj=_fp8_layer(t["up"]), down_proj=_fp8_layer(t["down"]))
        model = llm.CausalTransformerModel(cfg, _arr(t["embed"]), [llm.TransformerBlock(rms["n1"], a, rms["n2"], m)], rms["nf"],
                                           lm_head=_arr(t["head"]), spec=llm.LLAMA_SPEC)
        model.init_decode(T, max_batch_size=min(64, T))
        s.update(model=model, kc=_view(a._k_cache), vc=_view(a._v_cache))
    elif kind == "rows":
        epi = c["epilogue"]
        s["layer"] = llm.LinearRows(_arr(t["w"]), epilogue=epi)
        s["y"] = torch.empty(c["rows"], s["layer"].out_cols, dtype=torch.float32, device=DEV)
    elif kind == "attn_prompt":
        W, H, G, D = c["width"], c["heads"], c["kv_heads"], c["dim"]
        cfg = llm.layered_config_from_json(
            {"architecture": "Dolurax", "width": W, "vocab": VOCAB, "logit_scale": 1.0, "logit_softcap": 30.0, "norm": {"eps": 1e-5},
             "layers": [{"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5,
                                                        "softcap": c["softcap"], "mask": {"size": c["chunk"]}}}]})
        mixer = llm.PagedAttentionMixer(cfg.layers[0].mixer, 0, llm.LinearRows(_arr(t["qkvg"])), llm.LinearRows(_arr(t["o"])), _arr(t["qn"]),
                                        _arr(t["kn"]), 1e-5)
        block = llm.PostNormBlock(mixer, (_arr(t["n1"]), _arr(t["b1"])), None, None, 1e-5)
        model = llm.LayeredCausalModel(cfg, _arr(t["embed"]), [block], (_arr(t["nf"]), _arr(t["bf"])),
                                       llm.LinearRows(_arr(t["head"]), epilogue=2, scale=1.0, cap=30.0))
        s.update(_prompt_state(model, cfg, _requests(t["tokens"], c["requests"])))
    elif kind == "latent_prompt":
        cfg = llm.layered_config_from_json({"architecture": "Turutar", "width": c["width"], "vocab": VOCAB, "norm": {"eps": 1e-6},
                                            "layers": [_latent_json(c)]})
        block = llm.ParallelBlock(_rms_1p(t["n1"]), _latent_mixer(cfg.layers[0].mixer, t, 0), _arr(t["s1"]), None, None)
        model = llm.LayeredCausalModel(cfg, _arr(t["embed"]), [block], _rms_1p(t["nf"]), llm.LinearRows(_arr(t["head"])),
                                       embed_norm=_rms_1p(t["en"]))
        s.update(_prompt_state(model, cfg, _requests(t["tokens"], c["requests"])))
    elif kind == "linear_prompt":
        H = c["heads"]
        cfg = llm.layered_config_from_json(
            {"architecture": "Rezulorn", "width": c["width"], "vocab": VOCAB, "norm": {"eps": 1e-6}, "residual_mult": 0.5,
             "canon": {"taps": c["taps"]},
             "layers": [{"type": "lightning", "mixer": {"heads": H, "dim": c["dim"], "vdim": c["vdim"], "decay": _decays(H)}}]})
        mixer = llm.LinearAttentionMixer(cfg.layers[0].mixer, 0, llm.LinearRows(_arr(t["proj"])), llm.LinearRows(_arr(t["o"])), _arr(t["on"]), 1e-6)
        block = llm.PreNormBlock(llm.RowNorm("layernorm_nobias", _arr(t["n1"]), None, 1e-6), llm.CausalConvRows(_arr(t["conv"])), mixer, None, None,
                                 None, _arr(torch.full((c["width"],), 0.5, device=DEV)))
        model = llm.LayeredCausalModel(cfg, _arr(t["embed"]), [block], llm.RowNorm("layernorm_nobias", _arr(t["nf"]), None, 1e-6),
                                       llm.LinearRows(_arr(t["head"]), epilogue=2, scale=1.0, cap=0.0))
        s.update(_prompt_state(model, cfg, _requests(t["tokens"], c["requests"])))
        s["slots"] = [model.cache.pool.slots, len(s["entries"])]
    elif kind == "experts":
        W, E, F, S, T = c["width"], c["experts"], c["ff"], c["shared_ff"], c["tokens"]
        spec = llm.MoESpec(experts=E, top=c["top"], ff=F, shared_ff=S, router="biased", identity=c["identity"], renorm=False, shared_gate=S > 0)
        moe = llm.BiasedRouterMoE(spec, _arr(t["router"]), _arr(t["corr"]), llm.LinearRows(_arr(t["gu"]), epilogue=1), llm.LinearRows(_arr(t["down"])),
                                  llm.LinearRows(_arr(t["sgu"]), epilogue=1) if S else None, llm.LinearRows(_arr(t["sdn"])) if S else None)
        mx = llm.AttentionMixerSpec(heads=1, kv_heads=1, dim=16, vdim=16, scale=0.25, out_gate=False, distance_bias=False)
        cfg = llm.LayeredConfig("Sumitar", VOCAB, W, [llm.LayerSpec(mx, spec)], block="sandwich", norm="dyt")
        small = torch.zeros(48, W, dtype=torch.bfloat16, device=DEV)
        unit = torch.ones(W, device=DEV)
        mixer = llm.PagedAttentionMixer(mx, 0, llm.LinearRows(_arr(small)), llm.LinearRows(_arr(torch.zeros(W, 16, dtype=torch.bfloat16, device=DEV))),
                                        _arr(unit[:16]), _arr(unit[:16]), 1e-6)
        norms = [llm.RowNorm("dyt", _arr(unit), None, 1e-6) for _ in range(4)]
        model = llm.LayeredCausalModel(cfg, _arr(small), [llm.SandwichBlock(norms[0], mixer, norms[1], norms[2], moe, norms[3])], norms[0],
                                       llm.LinearRows(_arr(small)))
        model.init_cache(max_tokens=T + 64)
        ctx = StepContext(model, [(0, [0] * T, [])], model._tile_sizes, model._tops)
        s["y"] = torch.empty(T, W, dtype=torch.float32, device=DEV)
        s.update(layer=moe, ctx=ctx, model=model, x=_arr(t["x"]), out=_arr(s["y"]))
    else:
        W, F, sd, n = c["width"], c["ff"], c["side"], c["times"]
        mlp = {"kind": "dense", "ff": F, "limit": 7.0}
        win = {"type": "attention", "mlp": mlp, "mixer": {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": c["dim"], "vdim": c["dim"],
                                                          "scale": c["dim"] ** -0.5, "mask": {"size": c["window"]}}}
        cfg = llm.layered_config_from_json({"architecture": "Turutar", "width": W, "vocab": VOCAB, "norm": {"eps": 1e-6}, "token_side": {"dim": sd},
                                            "loop": {"start": 0, "stop": 2, "times": n}, "layers": [dict(_latent_json(c), mlp=mlp), win]})
        blocks, table = [], _arr(t["side"])
        for i in range(2):
            p, m = t[f"l{i}"], cfg.layers[i].mixer
            if i == 0:
                mixer = _latent_mixer(m, t["latent"], 0)
            else:
                w = t["win"]
                mixer = llm.PagedAttentionMixer(m, 1, llm.LinearRows(_arr(w["proj"])), llm.LinearRows(_arr(w["o"])), _arr(w["qn"]), _arr(w["kn"]), 1e-6,
                                                q_bias=_arr(w["qb"]), k_bias=_arr(w["kb"]))
            ff = llm.GatedDenseRows(cfg.layers[i].mlp, llm.LinearRows(_arr(p["gu"])), llm.LinearRows(_arr(p["down"])))
            side = llm.TokenSideInput(table, i, sd, llm.LinearRows(_arr(p["sg"])), llm.LinearRows(_arr(p["sp"])),
                                      llm.RowNorm("rmsnorm", _arr(p["sn"]), None, 1e-6))
            blocks.append(llm.ParallelBlock(_rms_1p(p["n1"]), mixer, _arr(p["s1"]), ff, _arr(p["s2"]), side))
        model = llm.LayeredCausalModel(cfg, _arr(t["embed"]), blocks, _rms_1p(t["nf"]), llm.LinearRows(_arr(t["head"])), embed_norm=_rms_1p(t["en"]))
        R, L = c["requests"], c["ctx"]
        cache = model.init_cache(max_tokens=R * (L + 65), slots=R)
        for r in range(R):                   # contexts that earlier steps left: pages are handed out lowest first
            cache.extend(r, L)
        per = -(-(L + 1) // 64)
        have = -(-L // 64)
        for run in range(2 * n):
            p = t["pages"][run // 2]
            for src, dst in ([("lat", cache.k[run])] if run % 2 == 0 else [("k", cache.k[run]), ("v", cache.v[run])]):
                d, u = _view(dst), p[src]
                d = d.view(d.shape[0], *u.shape[1:])
                for r in range(R):
                    d[r * have:(r + 1) * have] = u[r * per:r * per + have]
        s.update(model=model, entries=[(r, [tok], [0]) for r, tok in enumerate(t["tokens"])], lengths=[(r, L) for r in range(R)])
    return s


def _decays(heads: int) -> list[float]:
    return [1.0 - 2.0 ** (-5.0 - 5.0 * h / max(1, heads - 1)) for h in range(heads)]


# ---------------------------------------------------------------------------------------------------- one pass
def run(s: dict):
    c = s["case"]
    kind = c["kind"]
    if kind == "linear_fp8":
        s["layer"](s["x"], out=s["out"])
        return s["y"]
    if kind in ("mlp_nvf4", "mlp_fp8"):
        s["layer"].forward(s["x"], out=s["out"], act_buf=s["act"])
        return s["y"]
    if kind == "attn_decode":
        a, L = s["layer"], c["ctx"]
        if c["seqs"] == 1:
            a.forward_fixed_cache(s["x"], L - 1, L, out=s["out"], qkv_buf=s["qkv"], attn_buf=s["flat"])
        else:
            h = a.attend_multi(s["x"], s["pos_arr"], s["len_arr"], qkv_buf=s["qkv"], attn_buf=s["flat"])
            a.o_proj.forward(h, out=s["out"])
        return {"y": s["y"], "k": s["kc"][:, L - 1], "v": s["vc"][:, L - 1]}          # the cache rows that the token wrote
    if kind == "moe_nvf4":
        s["layer"].forward(s["x"], out=s["out"])
        return s["y"]
    if kind == "prompt_fp8":
        hidden, _ = s["model"](s["t"]["tokens"], use_cache=True)
        logits = s["model"].get_logits(hidden.row(hidden.shape[0] - 1).view((1, c["hidden"])))
        s["kept"] = logits
        return {"hidden": _view(hidden), "logits": _view(logits), "k": s["kc"], "v": s["vc"]}
    if kind == "rows":
        t = s["t"]
        s["layer"].forward(t["x"].data_ptr(), c["k"], c["rows"], s["y"].data_ptr(), s["y"].shape[1])
        return s["y"]
    if kind in ("attn_prompt", "latent_prompt"):
        return _run_prompt(s)
    if kind == "linear_prompt":
        out = _run_prompt(s)
        st = s["model"].cache.state[0][-1]                       # the state that every sequence leaves behind
        out["state"] = _view(st)[:s["slots"][1]]
        return out
    if kind == "experts":
        s["layer"].forward_rows(s["ctx"], s["x"], s["out"])
        return s["y"]
    out, n = s["model"].step_device(s["entries"])
    for r, L in s["lengths"]:                                    # the tokens of this pass are taken back
        s["model"].cache.truncate(r, L)
    return {"logits": _view(out)[:n], "rows": _view(s["model"]._buf.x)[:n]}


# ---------------------------------------------------------------------------------------------------- in 64 bits
def _d(t):
    return t.to(F64)


def _softmax_heads(q, k, v, scale, mask, cap=0.0, slopes=None, dist=None, sinks=None):
    """q [t, H, D], k [s, G, D], v [s, G, Dv], mask [t, s] -> [t, H, Dv]"""
    H, G = q.shape[1], k.shape[1]
    out = torch.empty(q.shape[0], H, v.shape[2], dtype=F64, device=DEV)
    for h in range(H):
        g = h // (H // G)
        z = (q[:, h] @ k[:, g].T) * scale
        if cap:
            z = cap * torch.tanh(z / cap)
        if slopes is not None:
            z = z - slopes[h] * dist
        z = z.masked_fill(~mask, -math.inf)
        m = z.amax(-1, keepdim=True)
        if sinks is not None:
            m = torch.maximum(m, sinks[h])
        e = torch.exp(z - m)
        den = e.sum(-1, keepdim=True) + (torch.exp(sinks[h] - m) if sinks is not None else 0.0)
        out[:, h] = (e / den) @ v[:, g]
    return out


def _latent_exact(h, t, c, pos, past=None):
    """h [T, W] normed rows of one sequence at positions `pos`, `past` the cached rows before them -> the mixer's result"""
    H, D, R, kr, qr = c["heads"], c["dim"], c["rot"], c["kv_rank"], c["q_rank"]
    T = h.shape[0]
    z = h @ _d(t["lproj"]).T
    q = (_rms(z[:, :qr], _d(t["lqn"]), 1e-6) @ _d(t["quq"]).T).view(T, H, D + R)
    rows = torch.cat([_rms(z[:, qr:qr + kr], _d(t["lcn"]), 1e-6), _rope_pairs(z[:, qr + kr:qr + kr + R], pos, 10000.0)], 1)
    if past is not None:
        rows = torch.cat([past, rows])
    qa = torch.cat([torch.einsum("thd,hkd->thk", q[..., :D], _d(t["kab"])), _rope_pairs(q[..., D:], pos, 10000.0)], -1)
    mask = torch.arange(rows.shape[0], device=DEV)[None, :] <= pos[:, None]
    o = _softmax_heads(qa, rows[:, None], rows[:, None, :kr], (D + R) ** -0.5, mask, sinks=_d(t["sinks"]))
    o = torch.einsum("thk,hvk->thv", o, _d(t["vup"])) * torch.sigmoid(z[:, qr + kr + R:])[:, :, None]
    return o.reshape(T, -1) @ _d(t["lo"]).T


def exact(case: dict, seed: int):
    c, kind, t = case, case["kind"], _make(case, seed)
    if kind == "linear_fp8":
        return _d(t["x"]) @ _fp8_f64(*t["w"]).T
    if kind == "mlp_nvf4":
        z = _nvf4_times(_d(t["x"]), *t["gu"]).view(c["rows"], -1, 2, 8)          # eight gate columns, eight up columns, ...
        return _nvf4_times((_silu(z[:, :, 0]) * z[:, :, 1]).reshape(c["rows"], -1), *t["down"])
    if kind == "mlp_fp8":
        x = _d(t["x"])
        return (_silu(x @ _fp8_f64(*t["gate"]).T) * (x @ _fp8_f64(*t["up"]).T)) @ _fp8_f64(*t["down"]).T
    if kind == "attn_decode":
        H, G, S, L = c["heads"], c["kv_heads"], c["seqs"], c["ctx"]
        z = (_d(t["x"]) @ _fp8_f64(*t["qkv"]).T).view(S, H + 2 * G, 128)
        q, k, v = z[:, :H], z[:, H:H + G], z[:, H + G:]
        if c["qk_norm"]:
            q, k = _rms(q, _d(t["qn"]), 1e-6), _rms(k, _d(t["kn"]), 1e-6)
        pos = torch.full((S,), L - 1, device=DEV)
        q, k = _rope_half(q, pos, 1e6), _rope_half(k, pos, 1e6)
        y = torch.empty(S, H * 128, dtype=F64, device=DEV)
        one = torch.ones(1, L, dtype=torch.bool, device=DEV)
        for s in range(S):
            kk, vv = _d(t["k"][s * G:(s + 1) * G]).transpose(0, 1).clone(), _d(t["v"][s * G:(s + 1) * G]).transpose(0, 1).clone()
            kk[L - 1], vv[L - 1] = k[s], v[s]
            y[s] = _softmax_heads(q[s:s + 1], kk, vv, 128 ** -0.5, one).reshape(-1)
        return {"y": y @ _fp8_f64(*t["o"]).T, "k": k.reshape(S * G, 128), "v": v.reshape(S * G, 128)}
    if kind == "moe_nvf4":
        E, H, I, x = c["experts"], c["hidden"], c["inter"], _d(t["x"])
        z = (x @ _d(t["router"]).T).to(torch.bfloat16)           # the routing reads the logits in bfloat16, ties to the lower expert
        zs, idx = torch.sort(z.float(), dim=1, descending=True, stable=True)
        w = torch.softmax(zs[:, :c["top"]].to(F64), 1)
        y = torch.zeros(c["tokens"], H, dtype=F64, device=DEV)
        for e in range(E):
            r, j = torch.nonzero(idx[:, :c["top"]] == e, as_tuple=True)
            if r.numel():
                p = [(t[n][0].view(E, -1, t[n][0].shape[1])[e], t[n][1].view(E, -1, t[n][1].shape[1])[e]) for n in ("gate", "up", "down")]
                h = _silu(_nvf4_times(x[r], *p[0])) * _nvf4_times(x[r], *p[1])
                y[r] += w[r, j, None] * _nvf4_times(h, *p[2])
        return y
    if kind == "prompt_fp8":
        H, G, T, W = c["heads"], c["kv_heads"], c["tokens"], c["hidden"]
        x = _d(t["embed"])[t["tokens"]]
        z = (_rms(x, _d(t["n1"]), 1e-6) @ _fp8_f64(*t["qkv"]).T).view(T, H + 2 * G, 128)
        pos = torch.arange(T, device=DEV)
        q, k, v = _rope_half(z[:, :H], pos, 1e6), _rope_half(z[:, H:H + G], pos, 1e6), z[:, H + G:]
        o = _softmax_heads(q, k, v, 128 ** -0.5, pos[None, :] <= pos[:, None]).reshape(T, -1)
        x = x + o @ _fp8_f64(*t["o"]).T
        h = _rms(x, _d(t["n2"]), 1e-6)
        x = x + (_silu(h @ _fp8_f64(*t["gate"]).T) * (h @ _fp8_f64(*t["up"]).T)) @ _fp8_f64(*t["down"]).T
        x = _rms(x, _d(t["nf"]), 1e-6)
        slab = min(64, T)
        last = T - (T - 1) // slab * slab                        # the call returns the rows of its last slab
        return {"hidden": x[-last:], "logits": x[-1:] @ _d(t["head"]).T, "k": k.transpose(0, 1).contiguous(), "v": v.transpose(0, 1).contiguous()}
    if kind == "rows":
        y, e = _d(t["x"]) @ _d(t["w"]).T, c["epilogue"]
        if e == 1:
            return _silu(y[:, 0::2]) * y[:, 1::2]
        if e == 7:
            return torch.nn.functional.gelu(y[:, 0::2], approximate="tanh") * y[:, 1::2]
        if e == 6:
            return torch.relu(y) ** 2
        return torch.nn.functional.gelu(y, approximate="tanh") if e == 9 else y
    if kind == "attn_prompt":
        H, G, D, C = c["heads"], c["kv_heads"], c["dim"], c["chunk"]
        slopes = [2.0 ** (-8.0 * (h + 1) / H) for h in range(H)]
        rows, logits = [], []
        for toks in _requests(t["tokens"], c["requests"]):
            T = len(toks)
            x = _d(t["embed"])[toks]
            z = x @ _d(t["qkvg"]).T
            q = _rms(z[:, :H * D].view(T, H, D), _d(t["qn"]), 1e-5)
            k = _rms(z[:, H * D:(H + G) * D].view(T, G, D), _d(t["kn"]), 1e-5)
            v = z[:, (H + G) * D:(H + 2 * G) * D].view(T, G, D)
            i = torch.arange(T, device=DEV)
            mask = i[None, :] <= i[:, None]
            if C:
                mask &= i[None, :] // C == i[:, None] // C
            o = _softmax_heads(q, k, v, D ** -0.5, mask, c["softcap"], slopes, (i[:, None] - i[None, :]).to(F64)).reshape(T, -1)
            x = x + _layer_norm((o * torch.sigmoid(z[:, (H + 2 * G) * D:])) @ _d(t["o"]).T, _d(t["n1"]), 1e-5) + _d(t["b1"])
            rows.append(x)
            f = _layer_norm(x[-1:], _d(t["nf"]), 1e-5) + _d(t["bf"])
            logits.append(30.0 * torch.tanh(f @ _d(t["head"]).T / 30.0))
        return {"logits": torch.cat(logits), "rows": torch.cat(rows)}
    if kind == "latent_prompt":
        rows, logits = [], []
        for toks in _requests(t["tokens"], c["requests"]):
            x = _rms(_d(t["embed"])[toks], _d(t["en"]), 1e-6, 1.0)
            x = x + _d(t["s1"]) * _latent_exact(_rms(x, _d(t["n1"]), 1e-6, 1.0), t, c, torch.arange(len(toks), device=DEV))
            rows.append(x)
            logits.append(_rms(x[-1:], _d(t["nf"]), 1e-6, 1.0) @ _d(t["head"]).T)
        return {"logits": torch.cat(logits), "rows": torch.cat(rows)}
    if kind == "linear_prompt":
        H, D, Dv, dec = c["heads"], c["dim"], c["vdim"], _decays(c["heads"])
        rows, logits, states = [], [], []
        for toks in _requests(t["tokens"], c["requests"]):
            T = len(toks)
            x = _d(t["embed"])[toks]
            h = _layer_norm(x, _d(t["n1"]), 1e-6)
            u, w = h.clone(), _d(t["conv"])
            for j in range(c["taps"]):
                back = c["taps"] - 1 - j
                if back < T:
                    u[back:] += w[:, j] * h[:T - back]
            z = u @ _d(t["proj"]).T
            q, k, v = (_silu(p).view(T, H, -1) for p in (z[:, :H * D], z[:, H * D:2 * H * D], z[:, 2 * H * D:2 * H * D + H * Dv]))
            i = torch.arange(T, device=DEV, dtype=F64)
            o, st = torch.empty(T, H, Dv, dtype=F64, device=DEV), []
            for n in range(H):
                a = float(np.float32(dec[n]))
                gap = i[:, None] - i[None, :]
                wgt = torch.where(gap >= 0, a ** gap.clamp(min=0), torch.zeros((), dtype=F64, device=DEV))
                o[:, n] = ((q[:, n] @ k[:, n].T) * wgt) @ v[:, n]
                st.append((k[:, n] * (a ** (T - 1 - i))[:, None]).T @ v[:, n])
            o = _rms(o.view(T, -1), _d(t["on"]), 1e-6) * torch.sigmoid(z[:, 2 * H * D + H * Dv:])
            x = x + 0.5 * (o @ _d(t["o"]).T)
            rows.append(x)
            states.append(torch.stack(st).reshape(-1))
            logits.append(_layer_norm(x[-1:], _d(t["nf"]), 1e-6) @ _d(t["head"]).T)
        return {"logits": torch.cat(logits), "rows": torch.cat(rows), "state": torch.stack(states)}
    if kind == "experts":
        E, S, x = c["experts"], c["shared_ff"], _d(t["x"])
        z = x @ _d(t["router"]).T
        sc = torch.softmax(z[:, :E + c["identity"]], 1)
        idx = torch.sort(sc + _d(t["corr"]), dim=1, descending=True, stable=True)[1][:, :c["top"]]
        w = torch.gather(sc, 1, idx)
        y = torch.zeros_like(x)
        for e in range(E + c["identity"]):
            r, j = torch.nonzero(idx == e, as_tuple=True)
            if not r.numel():
                continue
            h = x[r]
            if e < E:
                p = h @ _d(t["gu"][e]).T
                h = (_silu(p[:, 0::2]) * p[:, 1::2]) @ _d(t["down"][e]).T
            y[r] += w[r, j, None] * h
        if S:
            p = x @ _d(t["sgu"]).T
            y += torch.sigmoid(z[:, -1:]) * ((_silu(p[:, 0::2]) * p[:, 1::2]) @ _d(t["sdn"]).T)
        return y
    # decode_step: one token of every request over the pages that `prepare` fills
    H, G, D, L, R, W, sd = c["heads"], c["kv_heads"], c["dim"], c["ctx"], c["requests"], c["width"], c["side"]
    per = -(-(L + 1) // 64)
    x = _rms(_d(t["embed"])[t["tokens"]], _d(t["en"]), 1e-6, 1.0)
    x0, pos = x.clone(), torch.full((1,), L, device=DEV)
    for r in range(2 * c["times"]):
        i, pg, p = r % 2, t["pages"][r // 2], t[f"l{r % 2}"]
        if r and i == 0:
            x = x + x0
        h = _rms(x, _d(p["n1"]), 1e-6, 1.0)
        mix = torch.empty_like(x)
        for q in range(R):
            if i == 0:
                past = _d(pg["lat"][q * per:(q + 1) * per].reshape(per * 64, -1)[:L])
                mix[q:q + 1] = _latent_exact(h[q:q + 1], t["latent"], c, pos, past)
                continue
            w = t["win"]
            z = h[q:q + 1] @ _d(w["proj"]).T
            qq, kk = z[:, :H * D] + _d(w["qb"]), z[:, H * D:(H + G) * D] + _d(w["kb"])
            past = [_d(pg[n][q * per:(q + 1) * per]).transpose(1, 2).reshape(per * 64, G, D)[:L] for n in ("k", "v")]
            keys = torch.cat([past[0], _rms(kk, _d(w["kn"]), 1e-6).view(1, G, D)])
            vals = torch.cat([past[1], kk.view(1, G, D)])
            j = torch.arange(L + 1, device=DEV)
            o = _softmax_heads(_rms(qq, _d(w["qn"]), 1e-6).view(1, H, D), keys, vals, D ** -0.5, (L - j < c["window"])[None],
                               sinks=torch.zeros(H, dtype=F64, device=DEV))
            mix[q:q + 1] = (o * torch.sigmoid(z[:, (H + G) * D:])[:, :, None]).reshape(1, -1) @ _d(w["o"]).T
        gu = h @ _d(p["gu"]).T
        ga, up = gu[:, 0::2].clamp(max=7.0), gu[:, 1::2].clamp(-7.0, 7.0)
        x = x + _d(p["s1"]) * mix + _d(p["s2"]) * ((ga * torch.sigmoid(1.702 * ga) * (up + 1.0)) @ _d(p["down"]).T)
        e = _d(t["side"])[t["tokens"]][:, i * sd:(i + 1) * sd]
        y = (torch.nn.functional.gelu(x @ _d(p["sg"]).T, approximate="tanh") * e) @ _d(p["sp"]).T
        x = x + _rms(y, _d(p["sn"]), 1e-6)
    return {"logits": _rms(x, _d(t["nf"]), 1e-6, 1.0) @ _d(t["head"]).T, "rows": x}


# ---------------------------------------------------------------------------------------------------- work and tolerance
def work(case: dict) -> dict:
    """bytes: matrices, inputs, cached rows and outputs once; flops: the products (attention over the visible keys)"""
    c, kind = case, case["kind"]
    if kind == "linear_fp8":
        w = c["k"] * c["n"]
        return dict(bytes=w + w / 8192 + 2 * c["rows"] * (c["k"] + c["n"]), flops=2 * c["rows"] * w)
    if kind in ("mlp_nvf4", "mlp_fp8"):
        w = 3 * c["hidden"] * c["inter"]
        return dict(bytes=w * (17 / 32 if kind == "mlp_nvf4" else 1 + 1 / 8192) + 4 * c["rows"] * c["hidden"], flops=2 * c["rows"] * w)
    if kind == "attn_decode":
        w = c["hidden"] * 128 * (2 * c["heads"] + 2 * c["kv_heads"])
        kv = c["seqs"] * c["ctx"] * c["kv_heads"] * 128
        return dict(bytes=w + 4 * kv + 4 * c["seqs"] * c["hidden"], flops=2 * c["seqs"] * w + 4 * c["seqs"] * c["ctx"] * c["heads"] * 128)
    if kind == "moe_nvf4":
        w = 3 * c["hidden"] * c["inter"]
        used = c["experts"] * (1 - (1 - min(1.0, c["top"] / c["experts"])) ** c["tokens"])
        return dict(bytes=used * w * 17 / 32 + 2 * c["experts"] * c["hidden"] + 4 * c["tokens"] * c["hidden"], flops=2 * c["tokens"] * min(c["top"], c["experts"]) * w)
    if kind == "prompt_fp8":
        W, T = c["hidden"], c["tokens"]
        w = W * (128 * (2 * c["heads"] + 2 * c["kv_heads"]) + 3 * c["inter"])
        return dict(bytes=w + 2 * VOCAB * W + 2 * T * W + 4 * T * c["kv_heads"] * 128,
                    flops=2 * T * w + 2 * T * T * c["heads"] * 128 + 2 * VOCAB * W)
    if kind == "rows":
        out = c["n"] // 2 if c["epilogue"] in (1, 7) else c["n"]
        return dict(bytes=c["n"] * c["k"] * (2 if c["dtype"] == "bfloat16" else 4) + 4 * c["rows"] * (c["k"] + out), flops=2 * c["rows"] * c["n"] * c["k"])
    if kind == "attn_prompt":
        W, H, G, D = c["width"], c["heads"], c["kv_heads"], c["dim"]
        w = W * (3 * H * D + 2 * G * D)
        pairs = sum(_pairs(n, c["chunk"]) for n in _split(c["tokens"], c["requests"]))
        return dict(bytes=2 * w + c["tokens"] * (4 * W + 4 * G * D + 2 * W) + c["requests"] * VOCAB * 4 + 2 * VOCAB * W,
                    flops=2 * c["tokens"] * w + 4 * pairs * H * D + 2 * c["requests"] * VOCAB * W)
    if kind == "latent_prompt":
        W, H, D, R, kr, qr, T = c["width"], c["heads"], c["dim"], c["rot"], c["kv_rank"], c["q_rank"], c["tokens"]
        w = W * (qr + kr + R + H) + qr * H * (D + R) + 2 * H * kr * 128 + W * H * 128
        pairs = sum(_pairs(n, 0) for n in _split(T, c["requests"]))
        return dict(bytes=2 * w + T * (4 * W + 2 * (kr + R) + 2 * W) + c["requests"] * VOCAB * 4 + 2 * VOCAB * W,
                    flops=2 * T * w + 2 * pairs * H * (D + R + 128) + 2 * c["requests"] * VOCAB * W)
    if kind == "linear_prompt":
        W, H, D, Dv, T = c["width"], c["heads"], c["dim"], c["vdim"], c["tokens"]
        w = W * (2 * H * D + 3 * H * Dv)
        return dict(bytes=2 * w + T * 6 * W + c["requests"] * (4 * H * D * Dv + VOCAB * 4) + 2 * VOCAB * W,
                    flops=2 * T * w + 4 * T * H * D * Dv + 2 * c["requests"] * VOCAB * W)
    if kind == "experts":
        W, T = c["width"], c["tokens"]
        return dict(bytes=2 * W * 3 * (c["experts"] * c["ff"] + c["shared_ff"]) + 8 * T * W,
                    flops=2 * T * 3 * W * (c["top"] * c["ff"] * c["experts"] / (c["experts"] + c["identity"]) + c["shared_ff"]))
    W, H, G, D, R, L, kr, qr = c["width"], c["heads"], c["kv_heads"], c["dim"], c["requests"], c["ctx"], c["kv_rank"], c["q_rank"]
    lat = W * (qr + kr + c["rot"] + H) + qr * H * (D + c["rot"]) + 2 * H * kr * 128 + W * H * 128
    win = W * (H * D + G * D + H) + W * H * D
    per = lat + win + 2 * (3 * c["ff"] * W + 2 * c["side"] * W)
    seen = min(L + 1, c["window"])
    return dict(bytes=2 * per + 2 * VOCAB * W + c["times"] * R * (2 * L * (kr + c["rot"]) + 4 * seen * G * D) + 4 * R * VOCAB,
                flops=2 * R * (c["times"] * per + VOCAB * W) + c["times"] * R * (2 * L * H * (2 * kr + c["rot"]) + 4 * seen * H * D))


def _pairs(n: int, chunk: int) -> float:
    """(query, key) pairs of one causal prompt under a chunk size"""
    if not chunk or chunk >= n:
        return n * (n + 1) / 2
    full, rest = divmod(n, chunk)
    return full * chunk * (chunk + 1) / 2 + rest * (rest + 1) / 2


def tolerance(case: dict) -> dict:
    """bfloat16 outputs or bfloat16 operands: an eighth bit that falls the other way somewhere in the chain; float32: the order
    of a sum"""
    kind = case["kind"]
    if kind == "rows" and case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if kind in ("moe_nvf4", "prompt_fp8", "decode_step", "attn_decode"):
        return {"rel": 1.5e-2, "max": 0.5}          # several roundings to bfloat16 one behind the other
    return {"rel": 1e-2, "max": 0.25}
