"""Real systems solved two at a time on the streaming kernel: batches large
enough for its rule (two rounds of pairs for every resident group), odd and even
counts, by tensor copies and by element copies, padded strides, an input window.

A sample of systems (first, last, random) against the __float128 oracle with
the single-system kernel's bounds: relative L2 per system <= 1e-13 FP64, 1e-12
for two FP64 refinement sweeps, 3e-7 for one rounding to FP32 storage and 2e-5
for FP32 arithmetic."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-13, "mixed": 1e-12, "f32": 2e-5, "f32mem": 3e-7}


def _run(M, B, ub, jwt, prec, stride, window):
    import torch

    from pfsolve_b200.api import App, last_launch
    rng = np.random.default_rng(M + B + ub + jwt)
    dt = np.float32 if prec in ("f32", "f32mem") else np.float64
    bands = WL.permute_bands(J.random_bands(rng, M, ub), M).astype(dt)
    kw = dict(bitmask=capi.RUNTIME_OUTPUTBUFFERSTRIDE | capi.RUNTIME_INPUTZEROPAD, run_outputBufferStride=stride,
              run_inputZeropad=window)
    case = O.Case(M=M, batch=B, upperBanded=ub, jw_type=jwt, **kw)
    rhs = rng.uniform(-1, 1, B * stride).astype(dt)
    tb, to = torch.from_numpy(bands).cuda(), torch.from_numpy(rhs.copy()).cuda()
    app = App(buffer=tb, outputBuffer=to, **J.case_fields(
        case, doublePrecision=int(dt == np.float64), doublePrecisionFloatMemory=int(prec == "f32mem"),
        mixedPrecisionRefinement=2 if prec == "mixed" else 0))
    app.append(**J.launch_fields(case))
    torch.cuda.synchronize()
    assert last_launch()["kernel"] == capi.PFSOLVE_KERNEL_STREAMING
    got = to.cpu().numpy().reshape(B, stride)
    app.close()
    ys = np.unique(np.concatenate([np.arange(20), np.arange(B - 20, B), rng.integers(0, B, 60)]))
    rows = rhs.reshape(B, stride)
    sub = O.Case(M=M, batch=len(ys), upperBanded=ub, jw_type=jwt, **kw)
    ref = O.jw_step(sub, bands.astype(np.float64), rows[ys].astype(np.float64).ravel(), "q", nthreads=16)
    ref = ref.reshape(len(ys), stride)[:, :M]
    e = (np.linalg.norm(got[ys, :M] - ref, axis=1) / np.linalg.norm(ref, axis=1)).max()
    assert e <= TOL[prec], (M, B, ub, jwt, prec, stride, e)
    np.testing.assert_array_equal(got[:, M:], rows[:, M:])


@pytest.mark.parametrize("prec", list(TOL))
@pytest.mark.parametrize("M", [200, 256, 512, 1008, 2048, 201, 511, 1001, 1999])
def test_pairs(M, prec):
    for ub, jwt in [(2, 13), (1, 13), (0, 13), (1, 10), (0, 10)]:
        B = (9500 if prec != "f32" else 38000) * 512 // max(512, M) + (ub + jwt) % 2  # odd and even counts
        _run(M, B, ub, jwt, prec, M, (0, M))
    _run(M, B | 1, 2, 13, prec, M + 7, (3, M - 5))
