"""Decoding on the kernel of few queries (a cluster of blocks per request) against float64 and the float32 kernel: head layouts that leave rows, warps
and blocks idle, value rows that are a prefix of the key rows, pages of any multiple of eight, runs of keys that begin and end anywhere in a
tile, blocks without a tile, operands that are not finite.  Queries and weights hold all 24 bits and sums are float32: the bounds of the
tensor-core form."""
import numpy as np
import pytest

from pygpukit_b200._lib import api
from tests.test_gpu_seq_attention_tc import Case, bf16

pytestmark = pytest.mark.gpu

FORMS = [
    dict(H=16, G=4, D=128, Dv=136, window=90, gate=1),
    dict(H=16, G=1, D=576, Dv=512, alias=True, sinks=True),
    dict(H=8, G=8, D=64, Dv=208, slopes=1, cap=20.0, PS=8),
    dict(H=40, G=1, D=40, Dv=256, chunk=100, gate=2, PS=16, slopes=2),
    dict(H=12, G=1, D=576, Dv=320, alias=True, sinks=True, gate=2, PS=128, window=333),
    dict(H=5, G=1, D=16, Dv=144, PS=24),
    dict(H=16, G=1, D=176, Dv=144, alias=True, PS=32, cap=7.0),
    dict(H=6, G=2, D=100, Dv=136),                               # not served: the float32 kernel
]


@pytest.mark.parametrize("blocks", [1, 2, 4, 16])
@pytest.mark.parametrize("form", range(len(FORMS)))
def test_decoding(form, blocks):
    c = Case([(p, 1) for p in (0, 1, 62, 63, 64, 127, 300, 1030)], splits=blocks, single=3, **FORMS[form])
    served = api.seq_attention_few_plan(c.D, c.Dv, c.D, c.D if c.alias else c.Dv, 1 if c.alias else 0, c.H, c.G, 2, c.PS, c.T, 1031)
    assert (served > 0) == (c.D != 100)
    ref = c.exact()
    new = c.run(False)
    c.single, c.splits = 1, 1
    old = c.run(True)
    top = np.abs(ref).max()
    assert np.abs(new - ref).max() <= 2 * np.abs(old - ref).max() + 2 * 2.0 ** -23 * top
    rms_old, rms_new = (np.sqrt(np.mean((x - ref) ** 2)) for x in (old, new))
    print(f"form {form} blocks {blocks}: rms {rms_old:.2e} -> {rms_new:.2e}")
    assert rms_new <= 1.5 * rms_old + 2.0 ** -24 * top


@pytest.mark.parametrize("form", [0, 1, 5])
def test_queries_at_odd_columns(form):
    """rows of an odd stride (a layer's gate per head of an odd number of heads): the bits of rows on even ones"""
    c = Case([(p, 1) for p in (0, 127, 300)], splits=2, single=3, **FORMS[form])
    want = c.run(False)
    c.q, c.ld = np.ascontiguousarray(np.pad(c.q, ((0, 0), (0, 1)))), c.ld + 1
    assert c.ld % 2 and np.array_equal(c.run(False), want)


def test_stale_rows_stay_outside():
    c = Case([(100, 1), (530, 1)], 8, 2, 128, 192, window=64, seed=4, single=3, splits=2)
    clean = c.run(False)
    used = np.zeros((c.k.shape[0], c.PS), bool)
    for s, (p, n) in enumerate(c.portions):
        j = np.arange(max(0, p - 63), p + n)
        used[c.table[s][j // c.PS], j % c.PS] = True
    for arr in (c.k, c.v):
        arr.transpose(0, 2, 1, 3)[~used] = np.nan
    assert (c.run(False) == clean).all()


@pytest.mark.parametrize("where", ["query", "key", "value"])
@pytest.mark.parametrize("alias", [False, True])
def test_infinities_follow_float32(where, alias):
    kw = dict(H=16, G=1, D=192, Dv=144, alias=True) if alias else dict(H=16, G=2, D=128, Dv=200)
    c = Case([(59, 1), (127, 1), (300, 1)], seed=8, single=3, splits=2, **kw)
    if where == "query":
        c.k[..., 5] = bf16(np.abs(c.k[..., 5]) + 0.01)
        q = c.q[:, 4:].reshape(c.T, c.H, c.D)
        q[::3, ::2, 5], q[1::3, 1::2, 5] = np.inf, -np.inf
        c.q[:, 4:] = q.reshape(c.T, -1)
        c.q[:, 4:][:, ::7] = bf16(c.q[:, 4:][:, ::7])    # elements whose smaller terms are 0
    for n, (s, j) in enumerate([(0, 2), (0, 31), (1, 57)]):
        pg, r = c.table[s][j // c.PS], j % c.PS
        if where == "key":
            c.k[pg, n % c.G, r, 3 if not alias else 150] = np.inf if n % 2 else -np.inf
        if where == "value":
            c.v[pg, :, r, 5 * n:5 * n + 9] = np.inf if n % 2 else -np.inf
    new, c.single, c.splits = c.run(False), 0, 1
    old = c.run(True)
    assert (np.isnan(old) == np.isnan(new)).all()
    assert not np.isfinite(old).all() or where == "query"
    inf = np.isinf(old)
    assert (inf == np.isinf(new)).all() and (np.sign(old[inf]) == np.sign(new[inf])).all()
    fin = np.isfinite(old)
    assert fin.any() and np.abs(old[fin] - new[fin]).max() <= 2.0 ** -18 * (1 + np.abs(old[fin]).max())
