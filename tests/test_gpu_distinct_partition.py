"""Unique keys and COUNT DISTINCT by partition (csrc/distinct_part.cu) against torch's sorts:
spans at and beside whole buckets and bitmap words, sparse and dense spans, the full int32
range, rows that do not spread (left to the sort), both sides of the row limit, keys off the
16-byte grid, NULL keys and values, and an output too small for the groups.  All results are
whole numbers and must be equal."""

import numpy as np
import pytest
import torch

from numfast_b200 import _lib
from numfast_b200 import device as D

pytestmark = pytest.mark.gpu

LIMIT = 1 << 21


def _rand(lo, hi, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _check_unique(keys, inverse):
    r = D.unique(keys, with_inverse=inverse)
    uk, inv, cnt = torch.unique(keys, return_inverse=True, return_counts=True)
    first = torch.full((uk.numel(),), keys.numel(), dtype=torch.int64, device="cuda")
    first.scatter_reduce_(0, inv, torch.arange(keys.numel(), device="cuda"), "amin")
    assert r["ng"] == uk.numel()
    assert torch.equal(r["uniq"], uk) and torch.equal(r["counts"], cnt)
    assert torch.equal(r["first"].long(), first)
    if inverse:
        assert torch.equal(r["inverse"].long(), inv)


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("span", [127 * 700, 128 * 700, 128 * 700 + 1, 12_800, 1 << 20, 3_000_001, 40_000_000])
def test_unique_spans(span, inverse):
    keys = _rand(-5, span - 5, 3 * LIMIT + 4097, span)
    keys[7], keys[-1] = -5, span - 6
    _check_unique(keys, inverse)


@pytest.mark.parametrize("n", [LIMIT - 1, LIMIT, LIMIT + 1])
def test_unique_row_limit(n):
    _check_unique(_rand(0, 300_000, n, n), True)


def test_unique_full_range():
    keys = _rand(-2 ** 31, 2 ** 31, 35_000_003, 1)
    keys[0], keys[1] = 2 ** 31 - 1, -2 ** 31
    _check_unique(keys, True)


@pytest.mark.parametrize("kind", ["zipf", "hot", "cluster", "stride", "unaligned", "sorted"])
def test_unique_forms(kind):
    n = 2 * LIMIT + 33
    keys = _rand(0, 500_000, n + 1, 2)
    if kind == "zipf":
        keys = (1e6 ** torch.rand(n, device="cuda", dtype=torch.float64)).to(torch.int32)
    elif kind == "hot":  # too rare for the sample, too many for a bucket
        keys[torch.randperm(n, device="cuda")[:30_000]] = 77
    elif kind == "cluster":
        keys[: n // 2] = keys[: n // 2] % 1000
    elif kind == "stride":
        keys = keys * 4096
    elif kind == "sorted":
        keys = keys.sort().values
    _check_unique(keys[1:] if kind == "unaligned" else keys[:n].contiguous(), True)


def _bits(mask):
    return torch.from_numpy(np.packbits(mask.cpu().numpy(), bitorder="little")).cuda()


def _pairs(keys, values, keep):
    p = torch.unique(((keys.long() << 32) + (values.long() + 2 ** 31))[keep])
    return torch.unique_consecutive(p >> 32, return_counts=True)


@pytest.mark.parametrize("nulls", ["", "k", "v", "kv"])
@pytest.mark.parametrize("span,vspan", [(1000, 50), (65_536, 3), (65_537, 2 ** 32), (700_001, 100), (2_000_000_000, 2)])
def test_count_distinct(span, vspan, nulls):
    n = 2 * LIMIT + 4097
    keys, values = _rand(-9, span - 9, n, 3), _rand(-(vspan // 2), vspan - vspan // 2, n, 4)
    values[:3] = -1
    keep, km, vm = torch.ones(n, dtype=torch.bool, device="cuda"), None, None
    if "k" in nulls:
        m = torch.rand(n, device="cuda") < 0.9
        keys[~m], keep, km = 123, keep & m, _bits(m)  # what a NULL slot holds must not look like a hot key
    if "v" in nulls:
        m = torch.rand(n, device="cuda") < 0.5
        keep, vm = keep & m, _bits(m)
    uk, nu = D.group_count_distinct(keys, values, km, vm)
    wk, wn = _pairs(keys, values, keep)
    assert torch.equal(uk, wk) and torch.equal(nu, wn)


@pytest.mark.parametrize("kind", ["zipf", "hot", "unaligned", "one_value"])
def test_count_distinct_forms(kind):
    n = 2 * LIMIT + 33
    keys, values = _rand(0, 100_000, n, 5), _rand(0, 1000, n, 6)
    if kind == "zipf":
        keys = (1e6 ** torch.rand(n, device="cuda", dtype=torch.float64)).to(torch.int32)
    elif kind == "hot":
        keys[torch.randperm(n, device="cuda")[:14_000]] = 77
    elif kind == "unaligned":
        keys, values = keys[1:], values[1:]
    else:
        values.fill_(-1)
    uk, nu = D.group_count_distinct(keys, values)
    wk, wn = _pairs(keys, values, torch.ones(keys.numel(), dtype=torch.bool, device="cuda"))
    assert torch.equal(uk, wk) and torch.equal(nu, wn)


def test_count_distinct_small_output():
    n, groups = 2 * LIMIT, 50_000
    keys = torch.arange(n, device="cuda", dtype=torch.int32) % groups
    values = torch.zeros_like(keys)
    out = torch.full((2, groups), -7, dtype=torch.int64, device="cuda")
    call = lambda cap: _lib.load().nfc_group_count_distinct(  # noqa: E731
        keys.data_ptr(), None, values.data_ptr(), None, n, cap, out[0].data_ptr(), out[1].data_ptr(), None)
    torch.cuda.synchronize()
    assert call(groups - 1) < 0
    assert bool((out == -7).all())
    assert call(groups) == groups
    assert torch.equal(out[0], torch.arange(groups, device="cuda")) and bool((out[1] == 1).all())
