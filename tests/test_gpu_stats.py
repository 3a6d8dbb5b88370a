"""nfc_groupby_stats: a struct that is used again holds nothing of the call before."""

import ctypes

import pytest
import torch

from numfast_b200 import _lib

pytestmark = pytest.mark.gpu


def groupby(n, strategy, stats, span=50):
    k = (torch.arange(n, device="cuda", dtype=torch.int32) * 7919) % span
    out = torch.empty((2, max(n, 1)), dtype=torch.int64, device="cuda")
    a = _lib.GroupbyArgs()
    a.n, a.keys, a.ncols, a.out_cap = n, k.data_ptr(), 0, n
    a.ukeys_out, a.counts_out = out[0].data_ptr(), out[1].data_ptr()
    ng = _lib.load().nfc_groupby(ctypes.byref(a), strategy, None, ctypes.byref(stats))
    torch.cuda.synchronize()
    return int(ng)


@pytest.mark.parametrize("n", [100, 16_384, 16_385, 300_000])
def test_reused_stats(cuda, n):
    s = _lib.GroupbyStats()
    s.overflowed, s.buckets, s.status, s.ng, s.nstages = 2, 77, -7, 99, 5
    assert groupby(n, _lib.STRAT_AUTO, s) == 50
    assert (s.overflowed, s.buckets, s.status, s.ng, s.nstages) == (0, 0, 0, 50, 0)


@pytest.mark.parametrize("strategy", [_lib.STRAT_AUTO, _lib.STRAT_PARTITION])
def test_hot_key_sample(cuda, strategy):
    """The library's own rule samples for hot keys on large inputs; a named strategy does not."""
    s = _lib.GroupbyStats()
    assert groupby(1_200_000, strategy, s, span=3) == 3
    assert (s.probe.pad >= 200) == (strategy == _lib.STRAT_AUTO)
    assert groupby(100_000, strategy, s, span=3) == 3
    assert s.probe.pad == 0
