"""SORTED strategy (csrc/sorted.cu) over run lengths around its rows per thread, warp and
tile, against the oracle: many short runs (staged output), long ones (whole warps and tiles
without a head), NULL rows at the edges, columns of every count and type."""

import numpy as np
import pytest

from oracle import nf_oracle as O
from tests.gpu_util import assert_carry_equal, device_groupby

pytestmark = pytest.mark.gpu

KINDS = {"": [], "i": ["i"], "f": ["f"], "if": ["i", "f"], "lf": ["l", "f"], "ilff": ["i", "l", "f", "f"]}


def _check(k, kinds, ops_of, val, rs):
    n = k.size
    cols = {}
    for j, t in enumerate(KINDS[kinds]):
        v = rs.lognormal(3.0, 1.0, n) if t == "f" else rs.integers(-2 ** 31, 2 ** 31, n)
        if t == "f":
            v[rs.random(n) < 0.001] = np.nan
        cols["%s%d" % (t, j)] = v if t == "f" else v.astype(np.int32 if t == "i" else np.int64)
    ops = {c: ops_of for c in cols}
    got = device_groupby(k, cols, val, "auto", ops=ops)
    assert got["strategy"] == "sorted"
    assert_carry_equal(got, O.groupby_multi(k, cols, ops, val), float_cols=[c for c in cols if c[0] == "f"])


@pytest.mark.parametrize("run", [1, 2, 3, 4, 7, 8, 9, 16, 17, 255, 256, 257, 2047, 2048, 4096, 4097, 30_000])
@pytest.mark.parametrize("kinds", list(KINDS))
def test_even_runs(cuda, run, kinds):
    n = 70_003
    rs = np.random.default_rng(run)
    k = (np.arange(n, dtype=np.int64) // run * 3 - 20_000).astype(np.int32)
    ops = ("sum", "count") if run % 2 else ("sum", "count", "min", "max")
    _check(k, kinds, ops, {}, rs)
    _check(k, kinds, ops, {"__key__": rs.random(n) > 0.3}, rs)


@pytest.mark.parametrize("gap", [40, 2100, 5000, 17_000, 40_000])
@pytest.mark.parametrize("kinds", ["i", "if", "lf"])
def test_stretches_of_null_rows(cuda, gap, kinds):
    """Stretches without a valid row, up to more than a probe block, inside and between runs."""
    n = 120_000
    rs = np.random.default_rng(gap)
    k = np.sort(rs.integers(0, 3000, n)).astype(np.int32)
    valid = np.ones(n, bool)
    for at in (0, 30_001, 70_016):
        valid[at:at + gap] = False
    _check(k, kinds, ("sum", "count", "min", "max"), {"__key__": valid}, rs)


@pytest.mark.parametrize("kinds", ["i", "if", "ilff"])
def test_mixed_run_lengths(cuda, kinds):
    rs = np.random.default_rng(4)
    lens = np.concatenate([rs.integers(1, 4, 30_000), [9000], rs.integers(1, 60, 3000), [1, 50_000, 1],
                           rs.integers(1, 3, 9000)])
    k = np.repeat(np.arange(lens.size), lens).astype(np.int32)
    _check(k, kinds, ("sum", "min"), {"__key__": rs.random(k.size) > 0.1}, rs)
