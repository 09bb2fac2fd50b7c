"""Which prompts run in portions of 512 rows, and what a feed-forward calls: the Python side of the FP8 path, without a GPU."""
import os
import subprocess
import sys

import pytest

from pygpukit_b200.core.array import GPUArray
from pygpukit_b200.core.dtypes import bfloat16, uint8
from pygpukit_b200.llm.config import TransformerConfig
from pygpukit_b200.llm.layers import mlp as mlp_module
from pygpukit_b200.llm.layers.attention import Attention
from pygpukit_b200.llm.layers.block import TransformerBlock
from pygpukit_b200.llm.layers.linear import LinearFP8
from pygpukit_b200.llm.layers.mlp import MLP
from pygpukit_b200.llm.models.causal import CausalTransformerModel


def array(*shape, dtype=bfloat16):
    return GPUArray(shape, dtype, ptr=256)               # never read


def fp8(n, k):
    return LinearFP8(array(n, k, dtype=uint8), array(-(-n // 128), -(-k // 128)))


def model(heads, kv_heads, dim):
    c = TransformerConfig(vocab_size=256, hidden_size=256, num_layers=1, num_heads=heads, num_kv_heads=kv_heads, intermediate_size=512, _head_dim=dim,
                          norm_eps=1e-6, rope_theta=1e4, max_position_embeddings=64, tie_word_embeddings=False)
    attn = Attention(None, None, None, fp8(256, heads * dim), c, qkv_proj=fp8((heads + 2 * kv_heads) * dim, 256))
    mlp = MLP(c, gate_proj=fp8(512, 256), up_proj=fp8(512, 256), down_proj=fp8(256, 512))
    m = object.__new__(CausalTransformerModel)
    m.comm, m.blocks = None, [TransformerBlock(None, attn, None, mlp)]
    return m


@pytest.mark.parametrize("heads,kv_heads,dim,portions", [(4, 2, 128, True), (128, 1, 128, True), (256, 2, 128, True), (129, 1, 128, False), (4, 2, 64, False),
                                                         (8, 4, 32, False), (2, 1, 256, False)])
def test_long_portions_need_attention_for_many_rows(heads, kv_heads, dim, portions):
    """Other heads keep their slabs: their kernel reads the context for every four rows and refuses more than 16384 groups of four."""
    assert model(heads, kv_heads, dim)._long_portions() is portions


class Calls(list):
    def __getattr__(self, name):
        return lambda *a: self.append(name)


@pytest.mark.parametrize("impl,rows,products,fused", [(None, 16, 0, 1), ("1", 64, 0, 1), ("2", 16, 2, 0), ("2", 64, 2, 0), (None, 200, 0, 1), ("2", 200, 0, 1)])
def test_the_other_product_serves_gate_and_up_too(monkeypatch, impl, rows, products, fused):
    """PGK_TC_IMPL=2 selects the product of the codes themselves (up to 64 rows), which has no form for gate and up together; prompts keep
    their slabs then."""
    from pygpukit_b200.llm.layers import linear as linear_module
    asked = "import os, sys; sys.path.insert(0, os.getcwd()); from pygpukit_b200.llm.layers.linear import raw_codes_asked; print(raw_codes_asked())"
    env = {k: v for k, v in os.environ.items() if k != "PGK_TC_IMPL"} | ({} if impl is None else {"PGK_TC_IMPL": impl})
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    assert subprocess.run([sys.executable, "-c", asked], env=env, cwd=root, capture_output=True, text=True).stdout.strip() == str(impl == "2")
    monkeypatch.setattr(linear_module, "_RAW_CODES", impl == "2")
    m = model(4, 2, 128)
    calls = Calls()
    monkeypatch.setattr(mlp_module, "api", calls)
    monkeypatch.setattr(linear_module, "api", calls)
    monkeypatch.setattr(mlp_module, "silu", lambda x, out: out)
    monkeypatch.setattr(mlp_module, "mul", lambda x, y, out: out)
    mlp = m.blocks[0].mlp
    mlp._scratch[rows] = (array(rows, 512), array(rows, 512))
    mlp.gate_up_act(array(rows, 256), out=array(rows, 512))
    assert (calls.count("gemv_fp8_bf16_ex"), calls.count("gemv_fp8_swiglu_bf16")) == (products, fused)
    assert m._long_portions() is (impl != "2")


def test_arrays_of_a_portion(monkeypatch):
    """No room is no error, anything else is; the arrays stay for the next prompt, and go when idle memory is asked for or an allocation
    would fail without them."""
    from types import SimpleNamespace
    from pygpukit_b200.core import array as array_module, idle
    from pygpukit_b200.llm.models import causal
    m, room, freed = model(4, 2, 128), [1 << 20], []

    def malloc(out, n):
        if n > room[0]:
            raise RuntimeError("cudaMalloc(ptr, bytes) failed: out of memory (runtime.cu:303)")
        room[0] -= n
        out._obj.value = 4096
        out._obj.size = n

    def free(ptr):
        freed.append(ptr)
        room[0] = 1 << 20

    api = SimpleNamespace(malloc=malloc, free=free)
    monkeypatch.setattr(array_module, "api", api)
    m.config = m.blocks[0].attn.config
    m._buffers, m._max_seq, m._prompt_bufs = SimpleNamespace(max_batch_size=16), 4096, None
    m._embed = lambda part, n, start, b: array(n, 256)
    m._layers = lambda *a: None
    m._final = lambda tail, b: tail
    ids = list(range(40))
    assert m._prompt(ids, 0).shape == (8, 256)
    kept = m._prompt_bufs
    assert kept is not None and m._prompt(ids, 0).shape == (8, 256) and m._prompt_bufs is kept and not freed
    kept = None
    x = GPUArray(((1 << 20) - 256,), uint8)                  # fits once the arrays are given back
    assert freed == [4096] and m._prompt_bufs is None
    assert m._prompt(ids, 0) is None                         # no room: slabs
    del x
    assert m._prompt(ids, 0) is not None and idle.give_back() and m._prompt_bufs is None and not idle.give_back()

    def fault(out, n):
        raise RuntimeError("cudaMalloc(ptr, bytes) failed: an illegal memory access was encountered (runtime.cu:303)")

    api.malloc = fault
    with pytest.raises(RuntimeError, match="illegal"):
        m._prompt(ids, 0)
