"""Mixed-precision steps of 2 049 to 4 096 rows, beyond the group kernel's
compiled rows: whatever the row count, stride and number of systems, by element
copies where no tensor map describes the rows.

Relative L2 per system against the __float128 oracle: 1e-12 after two FP64
refinement sweeps (the mixed mode's bound)."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [2049, 2050, 3001, 3072, 3104, 4095, 4096])
@pytest.mark.parametrize("ub,jwt", [(2, 13), (1, 13), (0, 13), (1, 10), (0, 10)])
def test_row_counts(M, ub, jwt):
    import torch

    from pfsolve_b200.api import App, last_launch, last_launch_form
    rng = np.random.default_rng(M + ub + jwt)
    bands = WL.permute_bands(J.random_bands(rng, M, ub), M)
    tb = torch.from_numpy(bands).cuda()
    for B, stride in [(1, M), (3, M + 1), (1201, M), (601, M + (-M) % 2 + 6)]:
        case = O.Case(M=M, batch=B, upperBanded=ub, jw_type=jwt, cfg_outputBufferStride=stride, cfg_scaleC=0.75)
        rhs = rng.uniform(-1, 1, B * stride)
        to = torch.from_numpy(rhs.copy()).cuda()
        app = App(buffer=tb, outputBuffer=to, mixedPrecisionRefinement=2, **J.case_fields(case))
        assert app.shape()["streaming"] == 1
        app.append()
        torch.cuda.synchronize()
        whole = M % 32 == 0 and M > 3072 and stride % 2 == 0  # four warps of 32 rows per thread
        assert last_launch()["kernel"] == capi.PFSOLVE_KERNEL_STREAMING
        assert last_launch_form() == dict(systemsPerGroup=1, elementCopies=0 if whole else 1)
        got = to.cpu().numpy().reshape(B, stride)
        app.close()
        ys = np.unique(np.concatenate([[0, B - 1], rng.integers(0, B, 24)]))
        sub = O.Case(M=M, batch=len(ys), upperBanded=ub, jw_type=jwt, cfg_outputBufferStride=stride, cfg_scaleC=0.75)
        ref = O.jw_step(sub, bands, rhs.reshape(B, stride)[ys].ravel(), "q", nthreads=16).reshape(len(ys), stride)
        d, n = (np.linalg.norm(v, axis=1) for v in (got[ys, :M] - ref[:, :M], ref[:, :M]))
        assert (d <= 1e-12 * n).all(), (M, B, stride, (d / n).max())
        np.testing.assert_array_equal(got[:, M:], rhs.reshape(B, stride)[:, M:])


def test_refused_launches():
    """What only the group kernel takes (a partial output window) is refused
    here, at the launch, with the buffers untouched."""
    import torch

    from pfsolve_b200.api import App
    M, B = 3001, 5
    t = torch.ones(3 * M, dtype=torch.float64, device="cuda")
    x = torch.full((M * B,), 2.0, dtype=torch.float64, device="cuda")
    app = App(buffer=t, outputBuffer=x, M_size=M, size=(M, B), upperBanded=2, jw_type=13, doublePrecision=1,
              mixedPrecisionRefinement=2, jw_control_bitmask=capi.RUNTIME_OUTPUTZEROPAD)
    with pytest.raises(capi.PfSolveError) as ei:
        app.append(outputZeropad=(0, 100))
    torch.cuda.synchronize()
    assert ei.value.code == capi.PFSOLVE_ERROR_UNSUPPORTED_COMBINATION and (x == 2).all().item()
    app.close()
    with pytest.raises(capi.PfSolveError) as ei:  # the group kernel's own path holds no such rows
        App(buffer=t, outputBuffer=x, M_size=M, size=(M, B), upperBanded=2, jw_type=13, doublePrecision=1,
            mixedPrecisionRefinement=2, kernelPath=1)
    assert ei.value.code == capi.PFSOLVE_ERROR_UNSUPPORTED_COMBINATION
