"""Few keys and skewed keys: copies of the shared-memory state, slices, hot keys and the
skewed ranking of the partition path, against the oracle."""

import numpy as np
import pytest

from numfast_b200 import device as dev
from oracle import nf_oracle as O
from tests.gpu_util import assert_carry_equal, device_groupby

pytestmark = pytest.mark.gpu


def _cols(kinds, n, rs):
    cols = {}
    for i, k in enumerate(kinds):
        name = "%s%d" % (k, i)
        if k == "f":
            cols[name] = rs.lognormal(3.0, 1.0, n)
        elif k == "l":
            cols[name] = rs.integers(-2 ** 40, 2 ** 40, n).astype(np.int64)
        else:
            cols[name] = rs.integers(-2 ** 31, 2 ** 31, n).astype(np.int32)
    return cols


def _check(k, cols, val, strategy):
    ops = {c: ("sum", "count", "min", "max") for c in cols}
    got = device_groupby(k, cols, val, strategy, ops=ops)
    assert_carry_equal(got, O.groupby_multi(k, cols, ops, val), float_cols=[c for c in cols if c[0] == "f"])


@pytest.mark.parametrize("card", [1, 2, 3, 31, 32, 33, 71, 145, 364, 2300])
@pytest.mark.parametrize("kinds", ["if", "i", "fli"])
@pytest.mark.parametrize("n", [20_001, 700_003])
def test_few_keys(cuda, card, kinds, n):
    """From 32 copies of the state down to one; CTAs of one step and of several."""
    rs = np.random.default_rng(card * 7 + n)
    k = (rs.integers(0, card, n) - 3).astype(np.int32)
    _check(k, _cols(kinds, n, rs), {"__key__": rs.random(n) > 0.1}, "dense_smem")


@pytest.mark.parametrize("share", [0.0, 0.03, 0.1, 0.6, 1.0])
@pytest.mark.parametrize("kinds", ["if", "fl", "i", "iff", "ilff"])
def test_hot_keys(cuda, share, kinds):
    """One key with the given share of the rows, a second with half of it: below and above
    the hot-key and skew limits, several slices per bucket, and buckets of one slice."""
    n, span = 1_300_001, 300_000
    rs = np.random.default_rng(int(share * 100) + len(kinds))
    k = rs.integers(0, span, n)
    u = rs.random(n)
    k[u < share] = 4097
    k[(u >= share) & (u < 1.5 * share)] = 4100
    val = {"__key__": rs.random(n) > 0.05}
    _check(k.astype(np.int32) - span // 2, _cols(kinds, n, rs), val, "partition")


def test_hot_key_in_every_bucket_and_nan(cuda):
    n = 900_000
    rs = np.random.default_rng(5)
    b = rs.integers(0, 20, n)
    k = (b * 2048 + np.where(rs.random(n) < 0.5, 7, rs.integers(0, 2048, n))).astype(np.int32)
    f = rs.standard_normal(n)
    f[rs.random(n) < 0.001] = np.nan
    f[rs.random(n) < 0.001] = np.inf
    v = np.where(rs.random(n) < 0.5, 32767, -32768).astype(np.int32)
    _check(k, {"i0": v, "f1": f}, {}, "partition")


def test_skewed_keys_leave_the_global_atomics(cuda):
    """2M rows over an L2-resident span: even keys stay with DENSE_GLOBAL, hot ones partition."""
    n = 2_000_000
    rs = np.random.default_rng(8)
    even = rs.integers(0, 100_000, n).astype(np.int32)
    hot = even.copy()
    hot[rs.random(n) < 0.2] = 77
    v = rs.integers(-1000, 1001, n).astype(np.int32)
    from tests.gpu_util import to_dev
    for k, name in ((even, "dense_global"), (hot, "partition")):
        r = dev.groupby(to_dev(k), [dev.DeviceColumn("v", to_dev(v), ("sum",))])
        assert r.strategy == name
        ref = O.groupby_multi(k, {"v": v}, {"v": ("sum", "count")}, {})
        np.testing.assert_array_equal(r.ukeys.cpu().numpy(), ref["ukeys"])
        np.testing.assert_array_equal(r.counts.cpu().numpy(), ref["counts"])
        np.testing.assert_array_equal(r.sums["v"].cpu().numpy(), ref["sums"]["v"])
