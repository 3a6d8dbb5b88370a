"""Concurrent calls: threads with their own streams whose kernels need very different amounts of
dynamic shared memory (the limit is per function, not per launch), and live batch plans of
different table sizes."""

import threading

import numpy as np
import pytest
import torch

from numfast_b200 import batch as B
from numfast_b200 import device as D

pytestmark = pytest.mark.gpu


def _keys(n, span, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, span, (n,), generator=g, device="cuda", dtype=torch.int32)


def _unique(n, span):
    k = _keys(n, span, span)

    def call():
        r = D.unique(k)
        return int(r["uniq"].numel()), int(r["counts"].sum())
    return call


def _count_distinct(n, card, values):
    k, v = _keys(n, card, card), _keys(n, values, values)

    def call():
        uk, nu = D.group_count_distinct(k, v)
        return int(uk.numel()), int(nu.sum())
    return call


def _partition(n, span, cols):
    k = _keys(n, span, span)
    v = _keys(n, 1000, 7)

    def call():
        r = D.groupby(k, [D.DeviceColumn("c%d" % i, v, ("sum", "min", "max")) for i in range(cols)],
                      strategy="partition")
        return r.ngroups, int(r.sums["c0"].sum())
    return call


def _dense(n, span):
    k = _keys(n, span, span)

    def call():
        r = D.groupby(k, [D.DeviceColumn("v", k, ("sum",))], strategy="dense_smem")
        return r.ngroups, int(r.sums["v"].sum())
    return call


PAIRS = {"unique": lambda: (_unique(2_200_000, 600_000_000), _unique(2_300_000, 1_200_000)),
         "count distinct": lambda: (_count_distinct(2_200_000, 2_000, 90_000), _count_distinct(2_200_000, 2_000_000, 50)),
         "partition": lambda: (_partition(60_000, 25_000_000, 1), _partition(60_000, 9_000, 4)),
         "dense": lambda: (_dense(60_000, 8_000), _dense(60_000, 3))}


@pytest.mark.parametrize("kind", list(PAIRS))
def test_calls_of_two_sizes_at_once(cuda, kind):
    calls = PAIRS[kind]()
    want = [c() for c in calls]
    torch.cuda.synchronize()
    failed = []
    rounds = 400 if kind in ("partition", "dense") else 250

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(rounds):
                try:
                    got = calls[i]()
                    if got != want[i]:
                        failed.append((i, got, want[i]))
                except Exception as e:  # a refused launch
                    failed.append((i, repr(e)))
                if failed:
                    return
    threads = [threading.Thread(target=work, args=(i,)) for i in (0, 1, 0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[:2]


def test_batch_plan_outlives_a_smaller_one(cuda):
    """A plan with a large shared table still runs after a default one is made."""
    rows = np.array([0, 5_000, 45_000, 300_000], dtype=np.int64)
    k, v = _keys(300_000, 9_000, 3), _keys(300_000, 100, 4)
    t = B.default_tuning()
    t.smem_slots, t.ctas_per_sm = 24 * 1024, 1
    big = B.BatchGroupby(rows, tuning=t)
    small = B.BatchGroupby(rows)
    for _ in range(2):
        for plan in (big, small):
            r = plan.run(k, v, graph=False)
            for q in range(3):
                a, b = int(rows[q]), int(rows[q + 1])
                uk, su, co = r.query(q)
                wk, inv, wc = np.unique(k[a:b].cpu().numpy(), return_inverse=True, return_counts=True)
                np.testing.assert_array_equal(uk, wk)
                np.testing.assert_array_equal(co, wc)
                np.testing.assert_array_equal(su, np.bincount(inv, weights=v[a:b].cpu().numpy()).astype(np.int64))
