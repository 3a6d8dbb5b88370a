"""nfc_plan_strategy on a probe that its caller has filled in: the padding does not count."""

import ctypes

import pytest

from numfast_b200 import _lib
from tests.test_strategy_rule_cpu import DENSE_GLOBAL, I32, SUM_MIN_MAX


@pytest.mark.parametrize("pad", [0, 16, 1024, 2 ** 31 - 1, -1])
def test_padding_is_ignored(pad):
    dummy = ctypes.c_void_p(0x1000)  # never dereferenced
    cols = (_lib.ValueCol * 1)()
    cols[0].dtype, cols[0].aggs = I32, SUM_MIN_MAX
    cols[0].data = cols[0].sum_out = cols[0].min_out = cols[0].max_out = dummy
    a = _lib.GroupbyArgs()
    a.n, a.keys, a.ncols, a.cols = 2_000_000, dummy, 1, cols
    a.ukeys_out = a.counts_out = dummy
    p = _lib.Probe(2_000_000, 0, 99_999, 0, pad)
    assert _lib.load().nfc_plan_strategy(ctypes.byref(a), ctypes.byref(p)) == DENSE_GLOBAL
