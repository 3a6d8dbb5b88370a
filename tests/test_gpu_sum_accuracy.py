"""Accuracy of float64 group sums against exact sums.

The values are m * 2^-52 with integers m of 53 significant bits, so a group's exact sum is
an integer sum.  A correctly rounded sum is off by at most 2^-53 of itself; sums that are
added up with few or compensated roundings stay below that on average, a chain of partial
sums folded one after the other does not (its error grows with the root of its length)."""

import numpy as np
import pytest
import torch

from numfast_b200 import device as D

pytestmark = pytest.mark.gpu

MEAN_BOUND = 2.0 ** -53


def _values(rng, n):
    m = (rng.integers(0, 1 << 52, n, dtype=np.int64) + (1 << 52)) << rng.integers(0, 7, n)
    return m, m.astype(np.float64) * 2.0 ** -52  # exact: 53 significant bits


def _exact(keys, m, card):
    """Sums of m * 2^-52 per key as long doubles (the integer halves are exact)."""
    order = np.argsort(keys, kind="stable")
    starts = np.searchsorted(keys[order], np.arange(card))
    hi = np.add.reduceat(m[order] >> 30, starts).astype(np.longdouble)
    lo = np.add.reduceat(m[order] & ((1 << 30) - 1), starts).astype(np.longdouble)
    return (hi * np.longdouble(2.0 ** 30) + lo) * np.longdouble(2.0 ** -52)


def _mean_error(keys, card, strategy, two_columns, expect=None):
    rng = np.random.default_rng(keys.size + card)
    keys[:card] = np.arange(card, dtype=np.int32)  # every key occurs
    if expect == "sorted":
        keys.sort()
    m, v = _values(rng, keys.size)
    dev = torch.device("cuda")
    cols = [D.DeviceColumn("f", torch.from_numpy(v).to(dev), ("sum", "min", "max") if two_columns else ("sum",))]
    if two_columns:
        cols.insert(0, D.DeviceColumn("i", torch.from_numpy(keys).to(dev), ("sum", "min", "max")))
    r = D.groupby(torch.from_numpy(keys).to(dev), cols, strategy=strategy)
    if expect is not None:
        assert r.strategy == expect
    exact = _exact(keys, m, card)
    assert r.ngroups == card
    err = np.abs(r.sums["f"].cpu().numpy().astype(np.longdouble) - exact) / exact
    return float(err.mean())


@pytest.mark.parametrize("two_columns", [False, True])
@pytest.mark.parametrize("n,card", [(1_000_000, 1500), (2_000_000, 20_000), (3_000_001, 15_000), (2_000_000, 400_000)])
def test_sorted_sums(cuda, n, card, two_columns):
    keys = np.random.default_rng(card).integers(0, card, n, dtype=np.int32)
    assert _mean_error(keys, card, "auto", two_columns, "sorted") <= MEAN_BOUND


def test_sorted_sums_of_infinities_and_nan(cuda):
    """Infinities and NaN pass through the sums as by plain addition."""
    n = 40_000
    keys = np.repeat(np.arange(n // 20, dtype=np.int32), 20)
    v = np.ones(n)
    v[5::400] = np.inf
    v[25::400] = -np.inf
    v[45::400], v[48::400] = np.inf, -np.inf
    v[65::400] = np.nan
    v[80::400], v[81::400] = 1.7e308, 1.7e308
    dev = torch.device("cuda")
    r = D.groupby(torch.from_numpy(keys).to(dev), [D.DeviceColumn("f", torch.from_numpy(v).to(dev), ("sum",))],
                  strategy="sorted")
    assert r.strategy == "sorted"
    with np.errstate(over="ignore", invalid="ignore"):
        want = v.reshape(-1, 20).sum(axis=1)
    np.testing.assert_array_equal(r.sums["f"].cpu().numpy(), want)


@pytest.mark.parametrize("two_columns", [False, True])
@pytest.mark.parametrize("order", ["sorted", None])
@pytest.mark.parametrize("n,card", [(10_007, 10), (16_384, 40), (9_000, 250), (16_000, 1500)])
def test_small_sums(cuda, n, card, order, two_columns):
    keys = np.random.default_rng(card).integers(0, card, n, dtype=np.int32)
    assert _mean_error(keys, card, "auto", two_columns, order) <= MEAN_BOUND


def test_small_sums_of_infinities_and_nan(cuda):
    k = np.arange(6000, dtype=np.int32) % 300
    v = np.ones(6000)
    v[5], v[905] = np.inf, np.inf
    v[6], v[906] = np.inf, -np.inf
    v[7] = np.nan
    v[8], v[308] = 1.7e308, 1.7e308
    v[9] = -np.inf
    dev = torch.device("cuda")
    r = D.groupby(torch.from_numpy(k).to(dev), [D.DeviceColumn("f", torch.from_numpy(v).to(dev), ("sum",))])
    with np.errstate(over="ignore", invalid="ignore"):
        want = v.reshape(-1, 300).sum(axis=0)
    np.testing.assert_array_equal(r.sums["f"].cpu().numpy(), want)


@pytest.mark.parametrize("two_columns", [False, True])
@pytest.mark.parametrize("n,card,strategy", [(1_000_000, 100, "dense_smem"), (1_000_000, 1500, "dense_smem"),
                                             (4_000_000, 365, "dense_smem"), (1_000_000, 1500, "partition"),
                                             (2_000_000, 20_000, "partition"), (4_000_000, 365, "partition")])
def test_sums_of_many_ctas(cuda, n, card, strategy, two_columns):
    """Keys whose rows are spread over many CTAs or slices."""
    keys = np.random.default_rng(card).integers(0, card, n, dtype=np.int32)
    assert _mean_error(keys, card, strategy, two_columns, strategy) <= MEAN_BOUND
