"""Small inputs (csrc/small.cu: one launch for probe and group-by) at the edges of its rows,
of the shared-memory state and of alignment, against the oracle and the general path."""

import numpy as np
import pytest
import torch

from numfast_b200 import device as dev
from oracle import nf_oracle as O
from tests.gpu_util import assert_carry_equal, bitmap, to_dev

pytestmark = pytest.mark.gpu

DTYPES = {"a": np.int32, "b": np.float64, "c": np.int64, "d": np.float64}


def _inputs(n, span, ncols, nulls, rs):
    k = (rs.integers(0, span, n) - span // 3).astype(np.int32)
    cols = {}
    for name in list(DTYPES)[:ncols]:
        if DTYPES[name] == np.float64:
            cols[name] = rs.lognormal(3.0, 1.0, n)
        else:
            cols[name] = rs.integers(-2 ** 31, 2 ** 31, n).astype(DTYPES[name])
    val = {}
    if nulls:
        val = {x: rs.random(n) > 0.2 for x in ["__key__"] + list(cols)}
    return k, cols, val


def _run(k, cols, val, strategy="auto", shift=0, row_filter=None):
    """shift: place every column `shift` elements past an aligned start."""
    def put(a):
        t = torch.empty(a.size + shift, dtype=torch.from_numpy(a[:0].copy()).dtype, device="cuda")
        t[shift:] = to_dev(a)
        return t[shift:]
    dc = [dev.DeviceColumn(c, put(v), ("sum", "min", "max"), bitmap(val.get(c))) for c, v in cols.items()]
    return dev.groupby(put(k), dc, bitmap(val.get("__key__")), strategy=strategy,
                       row_filter=None if row_filter is None else bitmap(row_filter))


def _host(r):
    return {"ukeys": r.ukeys.cpu().numpy(), "counts": r.counts.cpu().numpy(),
            "sums": {c: t.cpu().numpy() for c, t in r.sums.items()},
            "mins": {c: t.cpu().numpy() for c, t in r.mins.items()},
            "maxs": {c: t.cpu().numpy() for c, t in r.maxs.items()}}


@pytest.mark.parametrize("n", [1, 3, 4, 127, 4095, 4097, 16_383, 16_384, 16_385])
@pytest.mark.parametrize("ncols", [0, 1, 2, 4])
@pytest.mark.parametrize("nulls", [False, True])
def test_rows_and_columns(cuda, n, ncols, nulls):
    rs = np.random.default_rng(n * 10 + ncols)
    k, cols, val = _inputs(n, 300, ncols, nulls, rs)
    ops = {c: ("sum", "count", "min", "max") for c in cols}
    for shift in (0, 1):
        r = _run(k, cols, val, shift=shift)
        ref = O.groupby_multi(k, cols, ops, val)
        assert_carry_equal(_host(r), ref, float_cols=("b", "d"))
        g = _run(k, cols, val, strategy="dense_global")
        assert {x: r.probe[x] for x in ("n_valid", "kmin", "kmax", "sorted")} == \
               {x: g.probe[x] for x in ("n_valid", "kmin", "kmax", "sorted")}


@pytest.mark.parametrize("span", [1, 2, 2730, 2731, 8191, 8192, 100_000, 2 ** 31])
def test_spans(cuda, span):
    """Around the 96 KB state (36 B per key here) and far beyond it."""
    rs = np.random.default_rng(span % 1000)
    n = 9_001
    k = np.sort(rs.integers(0, span, n)) if span == 8191 else rs.integers(0, span, n)
    k = (k - 2 ** 30).astype(np.int32)
    k[0], k[-1] = -2 ** 30, span - 1 - 2 ** 30
    cols = {"a": rs.integers(-1000, 1001, n).astype(np.int32), "c": rs.integers(-99, 99, n).astype(np.int64)}
    ops = {c: ("sum", "count", "min", "max") for c in cols}
    flt = rs.random(n) < 0.5
    val = {"a": rs.random(n) > 0.1}
    r = _run(k, cols, val, row_filter=flt)
    ref = O.groupby_multi(k[flt], {c: v[flt] for c, v in cols.items()}, ops, {"a": val["a"][flt]})
    assert_carry_equal(_host(r), ref)


def test_sorted_flag_and_capacity(cuda):
    """Sortedness across lanes, warps and steps; all rows NULL; output too small."""
    n = 16_384
    base = np.arange(n, dtype=np.int32) // 7
    for at in (None, 2, 128, 4096, 12_288, n - 1):
        k = base.copy()
        if at is not None:
            k[at] = k[at - 1] - 1
        r = dev.groupby(to_dev(k), [])
        assert r.probe["sorted"] == (at is None)
        uk, c = np.unique(k, return_counts=True)
        np.testing.assert_array_equal(r.ukeys.cpu().numpy(), uk)
        np.testing.assert_array_equal(r.counts.cpu().numpy(), c)
    r = dev.groupby(to_dev(base), [], bitmap(np.zeros(n, bool)))
    assert r.ngroups == 0
    from numfast_b200 import _lib
    with pytest.raises(_lib.NativeError):
        dev.groupby(to_dev(base), [], buffers=dev.GroupbyBuffers(10, [], torch.device("cuda")))
