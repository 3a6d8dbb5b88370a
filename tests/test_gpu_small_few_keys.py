"""Small group-bys over few keys (csrc/small.cu: copies of the state, warps of one key, runs of
sorted keys) against the oracle: int32, int64 and float64 columns, NULL rows, NaN."""

import numpy as np
import pytest

from oracle import nf_oracle as O
from tests.gpu_util import assert_carry_equal, device_groupby

pytestmark = pytest.mark.gpu

COLUMNS = {"f": ["f"], "l": ["l"], "if": ["i", "f"], "ilff": ["i", "l", "f", "f"]}


@pytest.mark.parametrize("n", [6, 500, 9_001, 16_384])
@pytest.mark.parametrize("card", [1, 2, 3, 31, 64, 300])
@pytest.mark.parametrize("kinds", list(COLUMNS))
def test_few_keys(cuda, n, card, kinds):
    rs = np.random.default_rng(n + card)
    for order in ("any", "sorted", "runs of 128"):
        k = rs.integers(0, card, n) - card // 2
        if order == "sorted":
            k.sort()
        elif order == "runs of 128":
            k = k[np.arange(n) // 128]
        k = k.astype(np.int32)
        cols = {}
        for j, t in enumerate(COLUMNS[kinds]):
            v = rs.lognormal(3.0, 1.0, n) if t == "f" else rs.integers(-2 ** 31, 2 ** 31, n)
            if t == "f":
                v[rs.random(n) < 0.0005] = np.nan
            cols["%s%d" % (t, j)] = v if t == "f" else v.astype(np.int32 if t == "i" else np.int64)
        ops = {c: ("sum", "count", "min", "max") for c in cols}
        for val in ({}, {x: rs.random(n) > 0.2 for x in ["__key__"] + list(cols)}):
            got = device_groupby(k, cols, val, "auto", ops=ops)
            ref = O.groupby_multi(k, cols, ops, val)
            assert_carry_equal(got, ref, float_cols=[c for c in cols if c[0] == "f"])
