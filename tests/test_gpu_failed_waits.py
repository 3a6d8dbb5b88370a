"""A wait that runs out in a scatter pass: the kernels after it leave the incomplete records alone,
the call reports NFC_ERR_TIMEOUT and writes no output, and the next call is right.  The status
is set from the host (nfc_debug_fail_wait), before, between and after the passes."""

import numpy as np
import pytest
import torch

from numfast_b200 import _lib
from numfast_b200 import device as D

pytestmark = pytest.mark.gpu

NFC_ERR_TIMEOUT = -7


def _keys(n, span):
    g = torch.Generator(device="cuda").manual_seed(span)
    return torch.randint(0, span, (n,), generator=g, device="cuda", dtype=torch.int32)


def _groupby(n, span, shift):
    k = _keys(n + shift, span)[shift:]
    v = torch.ones(n, dtype=torch.float64, device="cuda")
    cols = [D.DeviceColumn("v", v, ("sum", "min"))]
    buf = D.GroupbyBuffers(min(n, span), cols, k.device)
    outs = [buf.ukeys, buf.counts, buf.sum["v"], buf.min["v"]]

    def call():
        r = D.groupby(k, cols, strategy="partition", buffers=buf)
        uk, c = torch.unique(k, return_counts=True)
        assert torch.equal(r.ukeys, uk.long()) and torch.equal(r.counts, c) and torch.equal(r.sums["v"], c.double())
    return call, outs


def _unique(n):
    k = _keys(n, 1 << 27)  # 1,024 buckets

    def call():
        r = D.unique(k, with_inverse=True)
        uk, c = torch.unique(k, return_counts=True)
        assert torch.equal(r["uniq"], uk) and torch.equal(r["counts"], c)
        assert torch.equal(r["uniq"][r["inverse"].long()], k)
    return call, []


def _count_distinct(n):
    k, v = _keys(n, 60_000), _keys(n, 50)

    def call():
        uk, nu = D.group_count_distinct(k, v)
        pairs = torch.unique(k.long() * 64 + v)
        wk, wn = torch.unique(pairs // 64, return_counts=True)
        assert torch.equal(uk, wk) and torch.equal(nu, wn)
    return call, []


# Calls and the points they pass: one scatter pass 2, two passes 3.
CALLS = {"two passes": (lambda: _groupby(300_000, 2_000_000, 0), 3),
         "one pass": (lambda: _groupby(300_000, 9_000, 0), 2),
         "slices": (lambda: _groupby(3_000_000, 9_000, 0), 2),
         "unaligned": (lambda: _groupby(300_000, 2_000_000, 1), 2),
         "unique": (lambda: _unique(2_200_000), 3),
         "count distinct": (lambda: _count_distinct(2_200_000), 3)}


@pytest.mark.parametrize("name,point", [(c, p) for c in CALLS for p in range(CALLS[c][1])])
def test_later_kernels_stop(cuda, name, point):
    call, outs = CALLS[name][0]()
    for t in outs:
        t.fill_(-12345)
    _lib.load().nfc_debug_fail_wait(point)
    try:
        with pytest.raises(_lib.NativeError) as e:
            call()
        assert e.value.code == NFC_ERR_TIMEOUT
    finally:
        _lib.load().nfc_debug_fail_wait(-1)
    for t in outs:
        assert bool((t == -12345).all())
    call()
