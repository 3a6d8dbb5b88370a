"""Top-k where many rows tie at the k-th key (csrc/topk.cu: the exact selection starts from the
sampled prefix): the sample names the right key, or a neighbour of it, with and without bits left
below the sampled ones.  Against the full argsort, which is pinned to the oracle elsewhere."""

import pytest
import torch

from numfast_b200 import device as dev

pytestmark = pytest.mark.gpu


def _column(kind, n, g):
    if kind == "i32 few values":
        return torch.randint(0, 40, (n,), generator=g, device="cuda", dtype=torch.int32)
    if kind == "i64 low bits":  # all ties as far as the sampled bits go
        return torch.randint(0, 1 << 19, (n,), generator=g, device="cuda", dtype=torch.int64)
    if kind == "i64 few values":
        return torch.randint(-3, 4, (n,), generator=g, device="cuda", dtype=torch.int64) << 50
    if kind == "f64 rounded":
        return torch.randint(-50, 50, (n,), generator=g, device="cuda").double()
    if kind == "f64 nan and ties":
        f = torch.randint(0, 3, (n,), generator=g, device="cuda").double()
        f[::7] = float("nan")
        return f
    k = torch.full((n,), 1000, dtype=torch.int32, device="cuda")  # a few rare keys on both sides
    at = torch.randperm(n, generator=g, device="cuda")[:600]
    k[at[:300]] = torch.arange(300, dtype=torch.int32, device="cuda")
    k[at[300:]] = torch.arange(2000, 2300, dtype=torch.int32, device="cuda")
    return k


KINDS = ["i32 few values", "i64 low bits", "i64 few values", "f64 rounded", "f64 nan and ties", "one value"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [70_001, 1_500_000, 9_000_001])
def test_ties(cuda, kind, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    k = _column(kind, n, g)
    few = torch.zeros(n, dtype=torch.bool, device="cuda")
    few[::37] = True
    for mask in (None, torch.rand(n, generator=g, device="cuda") > 0.1, few):
        bits = None if mask is None else dev.pack_validity_dev(mask)
        for desc in (False, True):
            full = dev.sort_perm(k, desc, bits)
            for kk in (1, 7, 299, 300, 301, 1500, 4000):
                assert torch.equal(dev.sort_topk(k, kk, desc, bits), full[:kk]), (desc, kk)
