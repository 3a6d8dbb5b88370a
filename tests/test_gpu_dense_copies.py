"""DENSE_SMEM's copies of the state (csrc/agg_smem.cuh: fold_copies) around the numbers of keys at
which the copies and the lanes per slot change, against the oracle."""

import numpy as np
import pytest

from oracle import nf_oracle as O
from tests.gpu_util import assert_carry_equal, device_groupby

pytestmark = pytest.mark.gpu

COLUMNS = {"": [], "i": ["i"], "f": ["f"], "if": ["i", "f"], "ilff": ["i", "l", "f", "f"]}


@pytest.mark.parametrize("card", [1, 2, 15, 16, 17, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1000, 1600])
@pytest.mark.parametrize("kinds", list(COLUMNS))
def test_dense_smem(cuda, card, kinds):
    n = 90_001
    rs = np.random.default_rng(card)
    k = (rs.integers(0, card, n) - card // 2).astype(np.int32)
    k[:2] = -(card // 2), card - 1 - card // 2
    cols = {}
    for j, t in enumerate(COLUMNS[kinds]):
        v = rs.lognormal(3.0, 1.0, n) if t == "f" else rs.integers(-2 ** 31, 2 ** 31, n)
        if t == "f":
            v[rs.random(n) < 0.0002] = np.nan
        cols["%s%d" % (t, j)] = v if t == "f" else v.astype(np.int32 if t == "i" else np.int64)
    ops = {c: ("sum", "count", "min", "max") for c in cols}
    val = {x: rs.random(n) > 0.1 for x in ["__key__"] + list(cols)[:1]}
    for validity in ({}, val):
        got = device_groupby(k, cols, validity, "dense_smem", ops=ops)
        assert got["strategy"] == "dense_smem"
        ref = O.groupby_multi(k, cols, ops, validity)
        assert_carry_equal(got, ref, float_cols=[c for c in cols if c[0] == "f"])
