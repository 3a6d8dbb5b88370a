"""Radix sort (csrc/radix_sort.cu) at the edges of its tiles, groups and digit windows.

The permutation is unique (stable order), so every comparison is exact."""

import numpy as np
import pytest
import torch

from numfast_b200 import device as dev

pytestmark = pytest.mark.gpu

TILE = 4096
SMALL = 2048


def _check(keys, desc=False):
    got = dev.sort_perm(keys, descending=desc)
    want = torch.sort(keys, stable=True, descending=desc).indices.to(torch.int32)
    assert torch.equal(got, want)


@pytest.mark.parametrize("n", [1, SMALL, SMALL + 1, TILE - 1, TILE, TILE + 1, 32 * TILE, 32 * TILE + 1, 33 * TILE - 5])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_sizes(n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    k = torch.randint(-(1 << 30), 1 << 30, (n,), generator=g, dtype=dtype, device="cuda")
    _check(k if dtype == torch.int32 else k * 7_919_123_457)
    _check(k % 5, desc=True)


def test_grouped_tiles():
    """More than 16 tiles per SM: tiles counted in groups of 16, the last group partial."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 16 * sms * TILE + 3 * TILE + 77
    g = torch.Generator(device="cuda").manual_seed(3)
    k = torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, dtype=torch.int64, device="cuda")
    _check(k.to(torch.int32))
    _check((k % 1000).to(torch.int32))
    _check(k << 20)


@pytest.mark.parametrize("mask", [0x1, 0x80, 0x3FC, 0xF0F0F, 0x7F000000, 0x40000001])
@pytest.mark.parametrize("wide", [False, True])
def test_digit_windows(mask, wide):
    """Passes cover only the bits in which keys differ, from any bit on."""
    n = 5 * TILE + 11
    r = torch.randint(0, 1 << 31, (n,), generator=torch.Generator().manual_seed(mask), dtype=torch.int64) & mask
    r |= 0x2 if not mask & 2 else 0  # a constant bit is not sorted on
    k = ((r << 32) | (r >> 3) if wide else r.to(torch.int32)).cuda()
    _check(k)
    _check(k, desc=True)


def test_all_equal_and_unaligned():
    n = 3 * TILE + 5
    _check(torch.full((n,), -7, dtype=torch.int32, device="cuda"))
    g = torch.Generator(device="cuda").manual_seed(9)
    base = torch.randint(-(1 << 30), 1 << 30, (n + 1,), generator=g, dtype=torch.int32, device="cuda")
    r = dev.unique(base[1:])  # the first pass reads the caller's column, 4-byte aligned here
    uk, counts = torch.unique(base[1:], return_counts=True)
    assert torch.equal(r["uniq"], uk) and torch.equal(r["counts"], counts)
    first = np.unique(base[1:].cpu().numpy(), return_index=True)[1]
    assert np.array_equal(r["first"].cpu().numpy(), first)
