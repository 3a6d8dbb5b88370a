"""Which COUNT DISTINCT and unique calls the partition answers, and what a call that it does not
answer has spent before the sort."""

import pytest
import torch

from numfast_b200 import _lib
from numfast_b200 import device as D

pytestmark = pytest.mark.gpu

LIMIT = 1 << 21  # rows from which the partition is tried
NFC_ERR_TIMEOUT = -7


def _count_distinct(keys, values, cap, out):
    return _lib.load().nfc_group_count_distinct(keys.data_ptr(), None, values.data_ptr(), None, keys.numel(), cap,
                                                out[0].data_ptr(), out[1].data_ptr(), None)


def test_output_for_the_groups_only(cuda):
    """An output that holds the groups but not min(span, rows) is answered by the partition (a wait
    that fails there is reported) and left alone when it is too small."""
    n, groups = LIMIT + 5, 40_000
    keys = (torch.arange(n, device="cuda", dtype=torch.int32) % groups) * 37 - 1000
    values = torch.arange(n, device="cuda", dtype=torch.int32) % 3
    out = torch.full((2, groups), -7, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert _count_distinct(keys, values, groups - 1, out) == _lib.ERR_RANGE
    assert bool((out == -7).all())
    _lib.load().nfc_debug_fail_wait(0)
    try:
        assert _count_distinct(keys, values, groups, out) == NFC_ERR_TIMEOUT
    finally:
        _lib.load().nfc_debug_fail_wait(-1)
    assert bool((out == -7).all())
    assert _count_distinct(keys, values, groups, out) == groups
    pairs = torch.unique((keys.long() + 1000) // 37 * 4 + values)
    _, want = torch.unique(pairs // 4, return_counts=True)
    assert torch.equal(out[0], torch.arange(groups, device="cuda") * 37 - 1000)
    assert torch.equal(out[1], want)


def _allocations(call):
    """Scratch allocations of a call: the first one whose failure the call does not see."""
    lib = _lib.load()
    for k in range(64):
        lib.nfc_debug_fail_alloc(k)
        try:
            call()
            return k
        except _lib.NativeError as e:
            assert e.code == _lib.ERR_NOMEM
        finally:
            lib.nfc_debug_fail_alloc(-1)
    raise AssertionError("no end of allocations")


@pytest.mark.parametrize("kind", ["unique", "count distinct"])
def test_unaligned_columns_go_straight_to_the_sort(cuda, kind):
    """The scatter passes need 16-byte aligned columns: an unaligned call allocates what a call
    below the row limit does."""
    def call(n, shift):
        g = torch.Generator(device="cuda").manual_seed(n)
        k = torch.randint(0, 50_000_000, (n + shift,), generator=g, device="cuda", dtype=torch.int32)[shift:]
        if kind == "unique":
            return lambda: D.unique(k)
        return lambda: D.group_count_distinct(k, k)
    assert _allocations(call(LIMIT + 40_000, 1)) == _allocations(call(LIMIT - 40_000, 0))
