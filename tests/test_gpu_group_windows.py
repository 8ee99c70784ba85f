"""Keep-windows of the group kernel at the limits of their range: inside the
rows, reaching far beyond them (past 2^32), and wholly outside (nothing read or
nothing written), for every precision and for ALT row sets.

Relative L2 per system against the __float128 oracle, the precisions' own
bounds: 1e-13 FP64, 1e-12 for two FP64 refinement sweeps, 3e-7 and 2e-5 for
FP32 storage and arithmetic; rows outside the output window keep their values."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-13, "mixed": 1e-12, "f32": 2e-5, "f32mem": 3e-7}
FAR = 1 << 40


def _windows(M):
    return [((0, FAR), (2, M - 3)), ((3, M - 5), (0, FAR)), (((1 << 32) + 2, FAR), (0, M)), ((0, M), ((1 << 32) + 1, FAR)),
            ((M, FAR), (1, FAR)), ((0, 0), (0, M - 1))]


@pytest.mark.parametrize("prec", list(TOL))
@pytest.mark.parametrize("M", [33, 512, 1001, 2048])
def test_windows(M, prec):
    import torch

    from pfsolve_b200.api import App, last_launch
    B, dt = 37, np.float32 if prec in ("f32", "f32mem") else np.float64
    for ub, jwt in [(2, 13), (1, 10), (0, 10), (2, 113), (1, 110)]:
        alt = jwt > 100
        if alt and prec in ("f32", "f32mem"):
            continue
        rng = np.random.default_rng(M + ub + jwt)
        bands = WL.alt_bands(rng, M, ub) if alt else WL.permute_bands(J.random_bands(rng, M, ub), M)
        bands = bands.astype(dt)
        for wi, wo in _windows(M):
            case = O.Case(M=M, batch=B, upperBanded=ub, jw_type=jwt, run_inputZeropad=wi, run_outputZeropad=wo,
                          bitmask=capi.RUNTIME_INPUTZEROPAD | capi.RUNTIME_OUTPUTZEROPAD)
            rhs = rng.uniform(-1, 1, B * M).astype(dt)
            tb, to = torch.from_numpy(bands).cuda(), torch.from_numpy(rhs.copy()).cuda()
            app = App(buffer=tb, outputBuffer=to, kernelPath=1, **J.case_fields(
                case, doublePrecision=int(dt == np.float64), doublePrecisionFloatMemory=int(prec == "f32mem"),
                mixedPrecisionRefinement=2 if prec == "mixed" else 0))
            app.append(**J.launch_fields(case))
            torch.cuda.synchronize()
            assert last_launch()["kernel"] == capi.PFSOLVE_KERNEL_GROUP
            x = to.cpu().numpy().astype(np.float64).reshape(B, M)
            app.close()
            step = O.jw_step_alt if alt else (lambda *a: O.jw_step(*a, "q"))
            ref = step(case, bands.astype(np.float64), rhs.astype(np.float64)).reshape(B, M)
            inside = (np.arange(M) >= wo[0]) & (np.arange(M) < wo[1])
            np.testing.assert_array_equal(x[:, ~inside], rhs.reshape(B, M)[:, ~inside])
            d, n = (np.linalg.norm(v[:, inside], axis=1) for v in (x - ref, ref))
            assert (d <= TOL[prec] * n).all(), (M, prec, ub, jwt, wi, wo, d.max())
