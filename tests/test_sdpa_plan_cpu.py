"""How attention of many query rows cuts its keys and queries, from the library's own rule: no GPU."""
import ctypes as C

import numpy as np
import pytest

from pygpukit_b200._lib import api

RECORD = 132 * 4                                         # m, l and 128 sums


def plan(hq, n_kv, q_len, ctx, sms=148):
    out = (C.c_int32 * 3)()
    api.sdpa_prompt_plan(hq, n_kv, q_len, ctx, sms, out)
    return tuple(out)


def test_ranges_and_records_are_bounded():
    """Sums stay within 64 tiles of 128 keys, whatever the number of queries and heads, and records within 64 MB or one block of queries."""
    rng = np.random.default_rng(0)
    for _ in range(4000):
        n_kv = int(2 ** rng.integers(0, 6))
        hq = n_kv * int(rng.integers(1, 33))
        ctx = int(2 ** rng.uniform(5, 20))
        q_len = max(1, min(ctx, int(2 ** rng.uniform(4, 16))))
        rows_of_block, splits, rows = plan(hq, n_kv, q_len, ctx, int(rng.choice([1, 132, 148])))
        tiles = -(-ctx // 128)
        assert splits >= 1 and -(-tiles // splits) <= 64
        assert 1 <= rows <= q_len and (rows == q_len or rows % rows_of_block == 0)
        if splits > 1:
            assert rows * hq * splits * RECORD <= 64 << 20 or rows <= rows_of_block


@pytest.mark.parametrize("args,splits,rows", [((32, 8, 512, 512), 1, 512), ((32, 8, 64, 8192), 9, 64), ((64, 8, 512, 131072), 16, 112), ((4, 1, 20, 9000), 17, 20)])
def test_plans_of_usual_shapes(args, splits, rows):
    assert plan(*args)[1:] == (splits, rows)
