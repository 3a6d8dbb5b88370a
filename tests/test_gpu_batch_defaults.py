"""Batched group-by with the default tuning where a query sits at the edge of the shared
table or of the arena, against the oracle's per-query group-by (integers, exact)."""

import numpy as np
import pytest

from numfast_b200 import batch as B
from oracle import nf_oracle as O
from tests.gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3_000, 32_768, 32_769])
@pytest.mark.parametrize("extra", [8191, 8192, 8193, 16_384])
def test_spans_around_the_shared_table(cuda, rows, extra):
    """One query per span just below, at and above the table's slots; none is deferred."""
    rs = np.random.default_rng(rows + extra)
    spans = [extra, extra + 1, min(4 * rows + extra, rows + 40_000)]
    keys, vals = [], []
    for s in spans:
        k = rs.integers(0, s, rows)
        k[0], k[-1] = 0, s - 1
        keys.append(k.astype(np.int32) - 5)
        vals.append(rs.integers(-1000, 1001, rows).astype(np.int32))
    off = np.arange(len(spans) + 1, dtype=np.int64) * rows
    k, v = np.concatenate(keys), np.concatenate(vals)
    b = B.BatchGroupby(off)
    for _ in range(2):  # the second run finds the arena as the first one left it
        r = b.run(to_dev(k), to_dev(v))
        if rows <= 32_768:
            assert r.deferred == 0
        for q, (uk, su, ct) in enumerate(O.batch_sum_count(k, v, off)):
            gk, gs, gc = r.query(q)
            np.testing.assert_array_equal(gk, uk)
            np.testing.assert_array_equal(gs, su)
            np.testing.assert_array_equal(gc, ct)
    b.close()


@pytest.mark.parametrize("slots,ctas", [(16_384, 1), (8_192, 2), (1_024, 1)])
@pytest.mark.parametrize("rows", [2_500, 30_000])
def test_small_arena(cuda, rows, slots, ctas):
    """A small explicit arena: queries of up to 16,384 keys never needed it; wider ones are deferred
    and still right."""
    rs = np.random.default_rng(rows)
    spans = [100, 8_192, 8_193, 12_000, 16_383, 16_384] * 60 + [17_000]
    keys = [np.concatenate([[0, s - 1], rs.integers(0, s, rows - 2)]).astype(np.int32) - 9 for s in spans]
    vals = [rs.integers(-1000, 1001, rows).astype(np.int32) for _ in spans]
    off = np.arange(len(spans) + 1, dtype=np.int64) * rows
    k, v = np.concatenate(keys), np.concatenate(vals)
    t = B.default_tuning()
    t.arena_bytes, t.smem_slots, t.ctas_per_sm = 64 * 1024, slots, ctas
    b = B.BatchGroupby(off, tuning=t)
    assert b.info()["arena_bytes"] == 64 * 1024
    for graph in (False, True, True):
        r = b.run(to_dev(k), to_dev(v), graph=graph)
        assert r.deferred == 1
        for q, (uk, su, ct) in enumerate(O.batch_sum_count(k, v, off)):
            gk, gs, gc = r.query(q)
            np.testing.assert_array_equal(gk, uk)
            np.testing.assert_array_equal(gs, su)
            np.testing.assert_array_equal(gc, ct)
    b.close()
