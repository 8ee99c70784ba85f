"""How a streaming batch's entries are cut into items: the pruned search finds
the cut that scheduling every one of the 46 item sizes finds (restated here),
and costs little beside the rest of the plan's creation."""
import heapq
import math
import time

import numpy as np
import pytest

from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

pytestmark = pytest.mark.gpu
SYSTEM_US, BUILD_US = [0.13, 0.20, 0.40, 1.25, 2.40], [7, 7, 8, 10, 13]


def _full_search(specs, refine, sms):
    """(items, systems of the largest item) of the first cut of least greedy end."""
    def shape(m):
        return next(k for k, rows in enumerate((128, 256, 512, 1024, 2048)) if m <= rows)

    us = [(1.0 if refine else 0.55) * SYSTEM_US[shape(m)] for m, _ in specs]
    total = 0.0
    for (_, n), u in zip(specs, us):
        total += n * u
    best, share = None, 0.5
    while share <= 8.0:
        quantum = max(total / sms / share, 0.5)
        costs, items, most = [], 0, 0
        for (m, n), u in zip(specs, us):
            groups = 16 // (1, 1, 1, 2, 4)[shape(m)]
            rounds = -(-n // groups)
            parts = max(1, min(rounds, math.ceil(n * u / quantum)))
            per = max(1, -(-rounds // parts))
            most = max(most, per * groups)
            full, rest = divmod(rounds, per)
            costs += [BUILD_US[shape(m)] + float(per) * groups * u] * full
            if rest:
                costs.append(BUILD_US[shape(m)] + float(rest) * groups * u)
            items += full + (rest > 0)
        busy, end = [], 0.0
        for c in sorted(costs, reverse=True):
            at = heapq.heappop(busy) if len(busy) >= sms else 0.0
            heapq.heappush(busy, at + c)
            end = max(end, at + c)
        if best is None or end < best[0]:
            best = (end, items, most)
        share *= 1.0625
    return best[1:]


def _batch(specs, refine, **kw):
    import torch

    from pfsolve_b200.api import Batch
    t = torch.zeros(1 << 16, dtype=torch.float64, device="cuda")  # plans only: nothing is launched
    return Batch([dict(M=m, nsys=n, bands=t, input=t, output=t, inputStride=m, outputStride=m) for m, n in specs],
                 upperBanded=2, jw_type=13, mixedPrecisionRefinement=refine, **kw)


@pytest.mark.parametrize("seed", range(12))
def test_cut_matches_full_search(seed):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(seed)
    count = int(np.exp(rng.uniform(0, np.log(200))))
    specs = [(int(m), int(n)) for m, n in zip(np.exp(rng.uniform(0, np.log(2048), count)).astype(int) + (rng.random() < 0.5),
                                              np.exp(rng.uniform(np.log(64), np.log(20000), count)).astype(int))]
    specs = [(min(m, 2048), n) for m, n in specs]
    for refine in (0, 2):
        b = _batch(specs, refine)
        assert b.kernel() == capi.PFSOLVE_BATCH_STREAMING
        s = b.shape()
        assert (s["items"], s["systemsPerItem"]) == _full_search(specs, refine, sms)
        b.close()


@pytest.mark.parametrize("count", [32, 1000])
def test_creation_cost(count):
    """At most twice the creation of the same batch on the group kernel, which
    searches nothing (before the pruning: 1.7 and 3.5 times)."""
    specs = [(r.M, r.nrhs) for r in WL.config5_requests(count, seed=4)]
    for refine in (0, 2):
        best = []
        for kw in (dict(), dict(rowsPerThread=8)):
            ts = []
            for _ in range(9):
                t0 = time.perf_counter()
                b = _batch(specs, refine, **kw)
                ts.append(time.perf_counter() - t0)
                b.close()
            best.append(min(ts))
        assert best[0] <= 2 * best[1] + 1e-4, (count, refine, best)
