"""Which kernel a launch takes: pairs of systems exactly where that form is
compiled and the batch is large enough, element copies for rows no tensor map
describes, and the streaming batch kernel for every operator kind it holds.
(The results of these routes are checked in the tests of each.)"""
import numpy as np
import pytest

from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
# shapes (rows per thread, warps) whose pair form is compiled
PAIRS = {"f64": {(8, 1), (16, 1), (16, 2), (16, 4)}, "mixed": {(16, 1), (16, 2), (16, 4)},
         "f32": {(8, 1), (16, 2), (16, 4)}, "f32mem": {(8, 1), (16, 1)}}


def _launch(M, B, prec, ub=2, jwt=13):
    import torch

    from pfsolve_b200.api import App, last_launch, last_launch_form
    dt = np.float32 if prec in ("f32", "f32mem") else np.float64
    bands = WL.permute_bands(J.random_bands(np.random.default_rng(M), M, ub), M).astype(dt)
    tb = torch.from_numpy(bands).cuda()
    x = torch.zeros(M * B, dtype=tb.dtype, device="cuda")
    app = App(buffer=tb, outputBuffer=x, M_size=M, size=(M, B), upperBanded=ub, jw_type=jwt, scaleC=1.0,
              doublePrecision=int(dt == np.float64), doublePrecisionFloatMemory=int(prec == "f32mem"),
              mixedPrecisionRefinement=2 if prec == "mixed" else 0)
    app.append()
    torch.cuda.synchronize()
    app.close()
    return last_launch(), last_launch_form()


@pytest.mark.parametrize("prec", list(PAIRS))
@pytest.mark.parametrize("M,R,W", [(200, 8, 1), (512, 16, 1), (1008, 16, 2), (2048, 16, 4), (127, 4, 1), (201, 8, 1),
                                   (511, 16, 1), (1001, 16, 2), (1999, 16, 4)])
def test_pairs_where_compiled(M, R, W, prec):
    elem = M % 8 != 0
    for ub, jwt in [(2, 13), (1, 13), (0, 13), (1, 10), (0, 10)]:
        info, form = _launch(M, 80000 if M <= 512 else 24000, prec, ub, jwt)
        assert (info["kernel"], info["rowsPerThread"], info["warpsPerSystem"]) == (capi.PFSOLVE_KERNEL_STREAMING, R, W)
        assert form == dict(systemsPerGroup=2 if (R, W) in PAIRS[prec] else 1, elementCopies=int(elem)), (M, prec, ub)
    if not elem:
        assert _launch(M, 100, prec)[1] == dict(systemsPerGroup=1, elementCopies=0)
    else:  # few odd rows: the group kernel
        info, form = _launch(M, 64, prec)
        assert info["kernel"] == capi.PFSOLVE_KERNEL_GROUP and form == dict(systemsPerGroup=1, elementCopies=0)


BATCH_KINDS = [(2, 13, 0, 0), (0, 13, 0, 0), (0, 13, 3, 0), (0, 13, 3, 2), (2, 13, 0, 2), (0, 13, 0, 2), (1, 13, 0, 2), (1, 10, 0, 2),
               (0, 10, 0, 2)]


@pytest.mark.parametrize("ub,jwt,lda,refine", BATCH_KINDS)
def test_batch_kernel(ub, jwt, lda, refine):
    import torch

    from pfsolve_b200.api import Batch
    rng = np.random.default_rng(ub + jwt + lda)
    for Ms in ([100], [33, 500], [64, 1000], [2048, 300]):
        ents = []
        for M in Ms:
            tb = torch.from_numpy(WL.permute_bands(J.random_bands(rng, M, ub), M)).cuda()
            ti = torch.zeros(M * 400, dtype=torch.float64, device="cuda")
            ents.append(dict(M=M, nsys=400, bands=tb, input=ti, output=torch.zeros_like(ti), inputStride=M,
                             outputStride=M, dgbmvBands=torch.zeros(3 * M, dtype=torch.float64, device="cuda")))
        kw = dict(upperBanded=ub, jw_type=jwt, mixedPrecisionRefinement=refine)
        if lda:
            kw.update(LDA=lda, KU=1, KL=1)
        # (the mixed mode's 3-band kind beyond 1 024 rows: the group kernel)
        chosen = capi.PFSOLVE_BATCH_GROUP if lda and refine and max(Ms) > 1024 else capi.PFSOLVE_BATCH_STREAMING
        for extra, kernel in ((dict(), chosen), (dict(rowsPerThread=8), capi.PFSOLVE_BATCH_GROUP)):
            b = Batch(ents, **kw, **extra)
            assert b.kernel() == kernel, (Ms, extra)
            b.append()
            torch.cuda.synchronize()
            b.close()
