"""The rule between the streaming solve and the group kernel for uneven batches
of real systems: many entries of few systems, whose table builds would follow
one another on each SM, run on the group kernel; batches with work behind each
table on the streaming solve.  Results of both against the __float128 oracle
(relative L2 per system 1e-13 FP64, 1e-12 for two FP64 refinement sweeps)."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
TOL = {0: 1e-13, 2: 1e-12}
GROUP, STREAMING = capi.PFSOLVE_BATCH_GROUP, capi.PFSOLVE_BATCH_STREAMING


def _batch(M, E, n, ub, refine):
    import torch

    from pfsolve_b200.api import Batch
    rng = np.random.default_rng(M + E + n + ub)
    bands = WL.permute_bands(J.random_bands(rng, M, ub), M)
    rhs = rng.uniform(-1, 1, E * n * M)
    tb, ti = torch.from_numpy(bands).cuda(), torch.from_numpy(rhs).cuda()
    to = torch.zeros_like(ti)
    step = 8 * n * M
    b = Batch([dict(M=M, nsys=n, bands=tb, input=ti.data_ptr() + step * e, output=to.data_ptr() + step * e,
                    inputStride=M, outputStride=M) for e in range(E)], upperBanded=ub, jw_type=13,
              mixedPrecisionRefinement=refine)
    return b, (tb, ti), bands, rhs, to


@pytest.mark.parametrize("refine", [0, 2])
@pytest.mark.parametrize("ub", [2, 0])
@pytest.mark.parametrize("M,E,n,kernel", [(200, 1500, 1, GROUP), (500, 1500, 1, GROUP), (500, 400, 1, GROUP),
                                          (40, 64, 300, STREAMING), (200, 148, 64, STREAMING),
                                          (1000, 8, 300, STREAMING), (200, 1500, 64, STREAMING)])
def test_rule(M, E, n, kernel, ub, refine):
    import torch
    b, keep, bands, rhs, to = _batch(M, E, n, ub, refine)
    assert b.kernel() == kernel
    b.append()
    torch.cuda.synchronize()
    got = to.cpu().numpy().reshape(E * n, M)
    ys = np.unique(np.linspace(0, E * n - 1, 60).astype(int))
    case = O.Case(M=M, batch=len(ys), upperBanded=ub, jw_type=13, cfg_scaleC=1.0)
    ref = O.jw_step(case, bands, rhs.reshape(E * n, M)[ys].ravel(), "q", nthreads=16).reshape(len(ys), M)
    assert (np.linalg.norm(got[ys] - ref, axis=1) <= TOL[refine] * np.linalg.norm(ref, axis=1)).all()
    b.close()


def test_autotune_may_take_either():
    """The autotuner times both, whatever the rule says."""
    import torch
    for M, E, n in ((200, 1500, 1), (200, 148, 64)):
        b, keep, _, _, to = _batch(M, E, n, 2, 0)
        b.append()
        torch.cuda.synchronize()
        want = to.clone()
        b.autotune(iterations=2)
        b.append()
        torch.cuda.synchronize()
        assert ((to - want).norm() / want.norm()).item() <= 1e-13
        assert b.kernel() in (GROUP, STREAMING) and b.shape()["tunedMs"] > 0
        b.close()
