"""Where launches whose rows no tensor map describes take the streaming kernel
with element copies, and where its compiled shapes pad too much and the group
kernel keeps them: complex chains and ALT row sets.  Both kernels' results agree
(relative norm 1e-13 FP64, 1e-12 after two FP64 refinement sweeps, 2e-5 FP32
arithmetic, 3e-7 one rounding to FP32 storage)."""
import numpy as np
import pytest

from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
GROUP, STREAMING = capi.PFSOLVE_KERNEL_GROUP, capi.PFSOLVE_KERNEL_STREAMING
FIELDS = {"f64": dict(doublePrecision=1), "mixed": dict(doublePrecision=1, mixedPrecisionRefinement=2),
          "f32": dict(doublePrecision=0), "f32mem": dict(doublePrecision=0, doublePrecisionFloatMemory=1)}
TOL = {"f64": 1e-13, "mixed": 1e-12, "f32": 2e-5, "f32mem": 3e-7}


def _agree(a, b, prec):
    return ((a.double() - b.double()).norm() / b.double().norm()).item() <= TOL[prec]


@pytest.mark.parametrize("lda,prec,M,kernel", [
    (5, "f64", 33, GROUP), (5, "f64", 127, GROUP), (5, "f64", 129, STREAMING), (5, "f64", 511, STREAMING),
    (5, "f64", 513, GROUP), (5, "f64", 703, GROUP), (5, "f64", 705, STREAMING), (5, "mixed", 127, GROUP),
    (5, "mixed", 129, STREAMING), (5, "mixed", 513, STREAMING), (5, "f32", 127, GROUP), (5, "f32", 129, STREAMING),
    (5, "f32mem", 513, STREAMING), (3, "f64", 255, GROUP), (3, "f64", 257, STREAMING), (3, "f64", 513, GROUP),
    (3, "f64", 1023, GROUP), (3, "f32mem", 127, GROUP), (3, "f32mem", 129, STREAMING), (3, "f32", 255, GROUP),
    (3, "f32", 257, STREAMING), (3, "f32", 1001, STREAMING)])
def test_complex_chains(lda, prec, M, kernel):
    import torch

    from pfsolve_b200.api import App, append_chain, last_launch
    ub, ku, block = (2, 2, 7) if lda == 5 else (0, 1, 307)
    kw, B = FIELDS[prec], (1 << 22) // M
    plain = {k: v for k, v in kw.items() if k != "mixedPrecisionRefinement"}
    dt = torch.float32 if prec in ("f32", "f32mem") else torch.float64
    rng = np.random.default_rng(M)
    mat = torch.from_numpy(rng.uniform(-1, 1, lda * M)).to(dt).cuda()
    bands = torch.from_numpy(WL.permute_bands(J.random_bands(rng, M, ub), M)).to(dt).cuda()
    x = torch.randn(2 * M * B, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M))
    outs = []
    for path in (0, 1):
        o = torch.zeros_like(x)
        apps = [App(buffer=mat, outputBuffer=x, M_size=M, size=(M, 2 * B), LDA=lda, KU=ku, KL=ku, **plain),
                App(buffer=bands, outputBuffer=x, M_size=M, size=(M, 2 * B), upperBanded=ub, jw_type=13, scaleC=1.0,
                    kernelPath=path, **kw),
                App(buffer=x, outputBuffer=o, M_size=M, size=(M, B), block=block, lshift=2, scaleC=-0.5, **plain)]
        append_chain(apps, [a.launch_params() for a in apps])
        torch.cuda.synchronize()
        assert last_launch()["kernel"] == (GROUP if path else kernel), (M, prec, path)
        outs.append(o)
        for a in apps:
            a.close()
    assert _agree(outs[0], outs[1], prec)


@pytest.mark.parametrize("M,B,kernel", [(1001, 2401, STREAMING), (1025, 4000, GROUP), (1281, 4000, STREAMING),
                                        (2047, 2401, STREAMING), (2049, 4000, GROUP), (3583, 2500, GROUP),
                                        (3585, 2500, STREAMING), (4095, 2401, STREAMING), (4095, 600, GROUP)])
def test_alt_row_sets(M, B, kernel):
    import torch

    from pfsolve_b200.api import App, last_launch
    x0 = torch.randn(M * B, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M))
    for ub, jwt in [(2, 113), (1, 110), (0, 113)]:
        bands = torch.from_numpy(WL.alt_bands(np.random.default_rng(M), M, ub)).cuda()
        outs = []
        for path in (0, 1):
            x = x0.clone()
            app = App(buffer=bands, outputBuffer=x, M_size=M, size=(M, B), upperBanded=ub, jw_type=jwt, scaleC=1.0,
                      doublePrecision=1, kernelPath=path)
            app.append()
            torch.cuda.synchronize()
            assert last_launch()["kernel"] == (GROUP if path else kernel), (M, B, ub, path)
            outs.append(x)
            app.close()
        assert _agree(outs[0], outs[1], "f64")


@pytest.mark.parametrize("M,rows,kernel", [(500, 32, GROUP), (1000, 32, GROUP), (2047, 32, GROUP), (2049, 32, STREAMING),
                                           (501, 16, STREAMING), (255, 8, STREAMING), (257, 8, GROUP),
                                           (127, 4, STREAMING), (129, 4, GROUP)])
def test_rows_per_thread(M, rows, kernel):
    """A caller's rows per thread, where one of the compiled shapes of that many
    fits the system."""
    import torch

    from pfsolve_b200.api import App, last_launch
    B = (1 << 22) // M
    x0 = torch.randn(M * B, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(M))
    bands = torch.from_numpy(WL.permute_bands(J.random_bands(np.random.default_rng(M), M, 2), M)).cuda()
    outs = []
    for r in (rows, 0):
        x = x0.clone()
        app = App(buffer=bands, outputBuffer=x, M_size=M, size=(M, B), upperBanded=2, jw_type=13, scaleC=1.0,
                  doublePrecision=1, rowsPerThread=r)
        app.append()
        torch.cuda.synchronize()
        assert last_launch()["kernel"] == (kernel if r else STREAMING), (M, r)
        outs.append(x)
        app.close()
    assert _agree(outs[0], outs[1], "f64")
