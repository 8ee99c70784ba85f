"""Uneven batches of a fused 3-band matvec and upper-bidiagonal step on real
systems, at the edges of the streaming solve's shapes: every length in FP64,
up to 1 024 rows in the mixed mode (beyond, its table leaves the staging buffers
no room and the batch runs on the group kernel).

Relative L2 per system against the __float128 oracle: 1e-13 FP64, 1e-12 for two
FP64 refinement sweeps."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
TOL = {0: 1e-13, 2: 1e-12}


@pytest.mark.parametrize("refine", [0, 2])
@pytest.mark.parametrize("rows", [[1], [2, 33, 100], [127, 128], [129, 256, 20], [257, 512, 3], [513, 1001, 1024, 5],
                                  [1025, 64], [2048, 1500, 700]])
def test_three_bands(rows, refine):
    import torch

    from pfsolve_b200.api import Batch
    rng = np.random.default_rng(sum(rows) + refine)
    entries, data = [], []
    for M in rows:
        B, stride = 150, M + (M % 3)
        bands = WL.permute_bands(J.random_bands(rng, M, 0), M)
        mat, rhs = rng.uniform(-1, 1, 3 * M), rng.uniform(-1, 1, B * stride)
        t = [torch.from_numpy(a).cuda() for a in (bands, mat, rhs)]
        out = torch.full_like(t[2], 7.0)
        data.append((M, B, stride, bands, mat, rhs, t, out))
        entries.append(dict(M=M, nsys=B, bands=t[0], dgbmvBands=t[1], input=t[2], output=out, inputStride=stride,
                            outputStride=stride, scaleC=0.75))
    b = Batch(entries, upperBanded=0, jw_type=13, LDA=3, KU=1, KL=1, mixedPrecisionRefinement=refine)
    streams = not refine or max(rows) <= 1024
    assert b.kernel() == (capi.PFSOLVE_BATCH_STREAMING if streams else capi.PFSOLVE_BATCH_GROUP)
    b.append()
    torch.cuda.synchronize()
    b.close()
    for M, B, stride, bands, mat, rhs, _, out in data:
        y = O.dgbmv(O.Case(M=M, batch=B, LDA=3, KU=1, KL=1, jw_type=0, cfg_outputBufferStride=stride), mat, rhs,
                    nthreads=16)
        case = O.Case(M=M, batch=B, upperBanded=0, jw_type=13, cfg_scaleC=0.75, cfg_outputBufferStride=stride)
        ref = O.jw_step(case, bands, y, "q", nthreads=16).reshape(B, stride)[:, :M]
        got = out.cpu().numpy().reshape(B, stride)
        d, n = np.linalg.norm(got[:, :M] - ref, axis=1), np.linalg.norm(ref, axis=1)
        assert (d <= TOL[refine] * n).all(), (M, refine, (d / np.maximum(n, 1e-300)).max())
        assert (got[:, M:] == 7.0).all()
