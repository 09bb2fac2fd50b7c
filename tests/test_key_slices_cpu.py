"""Which form of attention decoding takes and into how many key slices it is cut: the host's rule, on a stand-in for a step."""
from types import SimpleNamespace

import pytest

from pygpukit_b200.llm.layers.paged_attention import TENSOR, key_slices


def step(requests, keys, dtype_code=2, page_size=64, max_pages=64):
    return SimpleNamespace(decode_only=True, tiles=lambda q: (None, requests), max_keys=lambda *a: keys,
                           cache=SimpleNamespace(dtype_code=dtype_code, page_size=page_size, pool=SimpleNamespace(max_pages=max_pages)))


def slices(ctx, heads, kv_heads, dims):
    rep = heads // kv_heads
    return key_slices(ctx, heads, kv_heads, 0, 0, 32 // min(rep, 32), min(rep, 32), 8, tensor_dims=dims)


@pytest.mark.parametrize("dims,kw", [((100, 128, 100, 128), {}), ((128, 100, 128, 100), {}), ((128, 128, 132, 128), {}), ((128, 128, 128, 130), {}),
                                     ((128, 128, 128, 128), dict(dtype_code=0)), ((128, 128, 128, 128), dict(page_size=1 << 12, max_pages=(1 << 12) + 1)),
                                     ((712, 512, 712, 712), {})])
@pytest.mark.parametrize("requests,keys", [(1, 60), (8, 1024), (24, 4096)])
def test_what_the_tensor_form_refuses_is_cut_for_the_float32_form(requests, keys, dims, kw):
    """rows off 16 bytes, float32 caches, positions beyond float32's whole numbers, key rows too long for shared memory"""
    assert slices(step(requests, keys, **kw), 16, 4, dims) == slices(step(requests, keys, **kw), 16, 4, None) < TENSOR


@pytest.mark.parametrize("dims", [(128, 128, 128, 128), (64, 80, 64, 80), (96, 24, 104, 24)])
def test_what_it_serves_takes_it(dims):
    assert slices(step(8, 1024), 16, 4, dims) >= TENSOR
    assert slices(step(8, 1024, page_size=1 << 12, max_pages=1 << 12), 16, 4, dims) >= TENSOR


@pytest.mark.parametrize("heads,dims", [(16, (576, 512, 576, 576)), (32, (320, 256, 320, 320)), (8, (256, 256, 256, 256))])
@pytest.mark.parametrize("requests", [1, 2, 7, 10, 24, 73, 75, 148, 200])
def test_long_value_rows_take_an_sm_each(requests, heads, dims):
    """blocks that fill an SM's tensor memory never outnumber the SMs because of the slices, and slices are a power of two"""
    for keys in (300, 1024, 4096, 1 << 15):
        s = slices(step(requests, keys, max_pages=1 << 10), heads, 1 if dims[0] > 256 else 2, dims)
        if s >= TENSOR:
            s -= TENSOR
            blocks = requests * (1 if dims[0] > 256 else 2)
            assert s & (s - 1) == 0 and 1 <= s <= 64 and (s == 1 or blocks * s <= 148)


def test_few_requests_of_many_latent_heads_stay_in_float32():
    dims = (576, 512, 576, 576)
    assert slices(step(1, 2000), 32, 1, dims) < TENSOR <= slices(step(1, 4096), 32, 1, dims)
    assert slices(step(1, 2000), 16, 1, dims) < TENSOR <= slices(step(2, 2000), 16, 1, dims)
