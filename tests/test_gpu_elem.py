"""The streaming kernel with element copies (jw_stream_elem_kernel): launches
whose rows no tensor map describes, at the edges of its shapes (4, 8 and 16
rows per thread of one warp, 16 of two and four, 32 of four) and of its two
copy forms (single values; 16-byte units with a ragged last one).

Tolerances, relative L2 per system against the __float128 oracle, as the other
kernels of the same precisions are held to: 1e-13 FP64, 1e-12 for two FP64
refinement sweeps, 3e-7 for one rounding to FP32 storage and 2e-5 for FP32
arithmetic."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-13, "mixed": 1e-12, "f32": 2e-5, "f32mem": 3e-7}
SHAPE = [(128, 4, 1), (256, 8, 1), (512, 16, 1), (1024, 16, 2), (2048, 16, 4), (4096, 32, 4)]


def _run(M, B, ub, jwt, prec, stride, offset):
    import torch

    from pfsolve_b200.api import App, last_launch
    rng = np.random.default_rng(M + 7 * B + ub + jwt)
    dt = np.float32 if prec in ("f32", "f32mem") else np.float64
    bands = WL.permute_bands(J.random_bands(rng, M, ub), M).astype(dt)
    kw = dict(bitmask=capi.RUNTIME_OFFSETSOLUTION | capi.RUNTIME_OUTPUTBUFFERSTRIDE, run_offsetSolution=offset,
              run_outputBufferStride=stride)
    case = O.Case(M=M, batch=B, upperBanded=ub, jw_type=jwt, **kw)
    rhs = rng.uniform(-1, 1, offset + B * stride + 8).astype(dt)
    tb, to = torch.from_numpy(bands).cuda(), torch.from_numpy(rhs.copy()).cuda()
    extra = dict(doublePrecision=int(dt == np.float64), doublePrecisionFloatMemory=int(prec == "f32mem"),
                 mixedPrecisionRefinement=2 if prec == "mixed" else 0)
    app = App(buffer=tb, outputBuffer=to, **J.case_fields(case, **extra))
    app.append(**J.launch_fields(case))
    torch.cuda.synchronize()
    info = last_launch()
    x = to.cpu().numpy()
    app.close()
    ref = O.jw_step(case, bands.astype(np.float64), rhs.astype(np.float64), "q", nthreads=16)
    got = x[offset:offset + B * stride].reshape(B, stride).astype(np.float64)
    want = ref[offset:offset + B * stride].reshape(B, stride)
    e = (np.linalg.norm(got[:, :M] - want[:, :M], axis=1) / np.linalg.norm(want[:, :M], axis=1)).max()
    np.testing.assert_array_equal(got[:, M:], rhs[offset:offset + B * stride].reshape(B, stride)[:, M:])
    np.testing.assert_array_equal(x[:offset], rhs[:offset])
    np.testing.assert_array_equal(x[offset + B * stride:], rhs[offset + B * stride:])
    return e, info


@pytest.mark.parametrize("M,prec", [(M, p) for p in TOL for M in (33, 127, 129, 257, 511, 513, 1001, 1025, 2047, 2049,
                                                                   4095) if p != "mixed" or M <= 2048])
def test_rows_at_shape_edges(M, prec):
    """(The mixed mode plans odd row counts up to 2 048 rows.)"""
    for ub, jwt in [(2, 13), (1, 10), (0, 13)]:
        for stride, offset in [(M, 0), (M + (-M) % 4 + 4, 8)]:  # odd rows; whole units with a ragged last one
            B = 20001 if M < 64 else (9601 if M < 256 else (4001 if M < 1024 else 1201))  # beyond the group kernel's rule
            e, info = _run(M, B, ub, jwt, prec, stride, offset)
            cap, R, W = next(s for s in SHAPE if s[0] >= M)
            assert (info["kernel"], info["rowsPerThread"], info["warpsPerSystem"]) == (
                capi.PFSOLVE_KERNEL_STREAMING, R, W), (M, prec, info)
            assert e <= TOL[prec], (M, prec, ub, jwt, stride, e)


@pytest.mark.parametrize("M,stride,offset", [(512, 513, 0), (512, 512, 1), (250, 251, 1), (64, 67, 3)])
def test_unaligned_rows_of_whole_chunks(M, stride, offset):
    for ub, jwt in [(2, 13), (1, 11), (0, 12), (0, 11)]:
        e, info = _run(M, 4001 if M > 256 else 20001, ub, jwt, "f64", stride, offset)
        assert info["kernel"] == capi.PFSOLVE_KERNEL_STREAMING
        assert e <= TOL["f64"], (ub, jwt, e)


@pytest.mark.parametrize("M,block,lshift", [(255, 7, 0), (511, 307, 3), (1001, 7, 0), (1023, 307, 3)])
def test_complex_chain_odd_rows(M, block, lshift):
    """dgbmv (5 bands) -> tridiagonal step -> XXII to packed (and a Scale
    operator), odd row counts packed at their own stride."""
    import torch

    from pfsolve_b200.api import App, append_chain, last_launch
    Y = 6001 if M < 512 else 2401  # beyond the group kernel's rule
    wl = WL.config2(M=M, B=Y)
    tA, tb, tr = (torch.from_numpy(a).cuda() for a in (wl.dgbmv, wl.jw_bands, wl.rhs))
    tout = torch.zeros(2 * M * Y + 2, dtype=torch.float64, device="cuda")
    dg = App(buffer=tA, outputBuffer=tr, M_size=M, size=(M, 2 * Y), LDA=5, KU=2, KL=2, doublePrecision=1, scaleC=1.0)
    jw = App(buffer=tb, outputBuffer=tr, M_size=M, size=(M, 2 * Y), upperBanded=2, jw_type=13, doublePrecision=1,
             scaleC=1.0)
    bl = App(buffer=tr, outputBuffer=tout, M_size=M, size=(M, Y), block=block, lshift=lshift,
             jw_control_bitmask=capi.RUNTIME_SCALEC, doublePrecision=1)
    append_chain([dg, jw, bl], [dg.launch_params(), jw.launch_params(), bl.launch_params(scaleC=0.5)])
    torch.cuda.synchronize()
    assert last_launch()["kernel"] == capi.PFSOLVE_KERNEL_STREAMING
    y = O.dgbmv(O.Case(M=M, batch=2 * Y, LDA=5, KU=2, KL=2, jw_type=0), wl.dgbmv, wl.rhs, nthreads=16)
    x = O.jw_step(O.Case(M=M, batch=2 * Y, upperBanded=2, jw_type=13), wl.jw_bands, y, "q", nthreads=16)
    cb = O.Case(M=M, batch=Y, block=block, lshift=lshift, jw_type=0, bitmask=O.RUNTIME_SCALEC, run_scaleC=0.5)
    ref = O.block(cb, x, np.zeros(2 * M * Y)).reshape(Y, 2 * M)
    out = tout.cpu().numpy()
    got = out[:2 * M * Y].reshape(Y, 2 * M)
    assert (np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)).max() <= TOL["f64"]
    assert (out[2 * M * Y:] == 0).all()


@pytest.mark.parametrize("M", [100, 255, 500, 999, 1001, 2047, 4095])
def test_alt_odd_row_sets(M):
    """ALT mode by element copies: row counts the streaming kernel's chunks do
    not divide, odd strides."""
    import torch

    from pfsolve_b200.api import App, last_launch
    B = 9001 if M < 512 else 2401
    for ub, jwt in [(2, 113), (1, 110), (0, 113), (0, 111)]:
        rng = np.random.default_rng(M + ub + jwt)
        bands = WL.alt_bands(rng, M, ub)
        case = O.Case(M=M, batch=B, upperBanded=ub, jw_type=jwt, bitmask=capi.RUNTIME_SCALEC, run_scaleC=0.5)
        rhs = rng.uniform(-1, 1, case.rhs_len())
        tb, to = torch.from_numpy(bands).cuda(), torch.from_numpy(rhs.copy()).cuda()
        app = App(buffer=tb, outputBuffer=to, **J.case_fields(case))
        app.append(**J.launch_fields(case))
        torch.cuda.synchronize()
        info = last_launch()
        assert (info["kernel"], info["alt"]) == (capi.PFSOLVE_KERNEL_STREAMING, 1)
        x = to.cpu().numpy()
        app.close()
        ref = O.jw_step_alt(case, bands, rhs, nthreads=16)
        assert np.abs(x - ref).max() <= 1e-13 * np.abs(ref).max(), (ub, jwt)
