"""Top-k with a sampled threshold (csrc/topk.cu): columns that a sample represents badly or
barely -- sorted, clustered, tied, narrow ranges, few valid rows -- where the call has to
notice and take the exact passes.  The order is unique, so the comparison with the full
argsort (pinned to the oracle elsewhere) is exact."""

import pytest
import torch

from numfast_b200 import device as dev

pytestmark = pytest.mark.gpu


def _column(kind, n, g):
    def i64(lo, hi, m=n):
        return torch.randint(lo, hi, (m,), generator=g, dtype=torch.int64, device="cuda")
    if kind == "i32":
        return i64(-(1 << 31), 1 << 31).to(torch.int32)
    if kind == "i32_sorted":
        return torch.sort(i64(-(1 << 31), 1 << 31).to(torch.int32)).values
    if kind == "i32_narrow":
        return i64(0, 1 << 20).to(torch.int32)
    if kind == "i32_ties":
        return i64(0, 50).to(torch.int32)
    if kind == "i64_narrow":
        return i64(-(1 << 40), 1 << 40)
    if kind == "i64_clustered":  # the smallest and largest rows sit in two short stretches
        k = i64(-1000, 1000)
        k[n // 3:n // 3 + 5000] = i64(-(1 << 50), 0, 5000)
        k[n // 2:n // 2 + 5000] = i64(0, 1 << 50, 5000)
        return k
    f = torch.randn(n, generator=g, dtype=torch.float64, device="cuda")
    if kind == "f64_nan":
        f[::40_009] = float("nan")
        f[::977] = float("inf")
        f[::1009] = -0.0
    if kind == "f64_all_nan":
        f[:] = float("nan")
    return f


KINDS = ["i32", "i32_sorted", "i32_narrow", "i32_ties", "i64_narrow", "i64_clustered", "f64", "f64_nan",
         "f64_all_nan"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("desc", [False, True])
@pytest.mark.parametrize("n", [65_536, 3_000_001, 20_000_003])
def test_against_full_argsort(kind, desc, n):
    g = torch.Generator(device="cuda").manual_seed(n + KINDS.index(kind))
    k = _column(kind, n, g)
    valid = dev.pack_validity_dev(torch.rand(n, generator=g, device="cuda") > 0.05)
    for bits in (None, valid):
        full = dev.sort_perm(k, desc, bits)
        for kk in (1, 37, 1000, 2500, 4999):
            assert torch.equal(dev.sort_topk(k, kk, desc, bits), full[:kk]), (bits is None, kk)


def test_few_valid_rows():
    n = 5_000_000
    k = torch.arange(n, dtype=torch.int32, device="cuda").flip(0)
    m = torch.zeros(n, dtype=torch.bool, device="cuda")
    m[::100_000] = True
    bits = dev.pack_validity_dev(m)
    full = dev.sort_perm(k, False, bits)
    for kk in (1, 49, 50, 51, 1000):
        assert torch.equal(dev.sort_topk(k, kk, False, bits), full[:kk])


def test_unaligned_column():
    base = torch.randn(2_000_001, generator=torch.Generator(device="cuda").manual_seed(1), dtype=torch.float64,
                       device="cuda")
    k = base[1:]
    assert torch.equal(dev.sort_topk(k, 100, True), dev.sort_perm(k, True)[:100])
