"""Uneven batches of real systems on the streaming solve
(jw_batch_stream_kernel): entries at the edges of its group shapes (4, 8, 16
rows per thread of one warp, 16 of two and four), few and many systems, odd and
whole-unit strides, in place and out of place, one and several items a CTA.

Each entry against the __float128 oracle, relative L2 per system: 1e-13 FP64,
1e-12 for two FP64 refinement sweeps (the bounds of the other kernels)."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
ROWS = [1, 2, 33, 127, 128, 129, 255, 256, 257, 512, 513, 1001, 1024, 1025, 2048]
TOL = {0: 1e-13, 2: 1e-12}


def _check(specs, ub, jwt, refine, inplace=False, reps=1):
    import torch

    from pfsolve_b200.api import Batch
    rng = np.random.default_rng(len(specs) + ub + jwt + refine)
    entries, keep, cases = [], [], []
    for M, B, stride in specs:
        bands = WL.permute_bands(J.random_bands(rng, M, ub), M)
        rhs = rng.uniform(-1, 1, B * stride)
        tb, ti = torch.from_numpy(bands).cuda(), torch.from_numpy(rhs).cuda()
        to = ti if inplace else torch.full_like(ti, 7.0)
        keep.append((tb, ti, to))
        cases.append((M, B, stride, bands, rhs))
        entries.append(dict(M=M, nsys=B, bands=tb, input=ti, output=to, inputStride=stride, outputStride=stride,
                            scaleC=0.75))
    b = Batch(entries, upperBanded=ub, jw_type=jwt, mixedPrecisionRefinement=refine)
    shape = b.shape()
    for _ in range(reps):
        b.append()
    torch.cuda.synchronize()
    for (M, B, stride, bands, rhs), (_, _, to) in zip(cases, keep):
        case = O.Case(M=M, batch=B, upperBanded=ub, jw_type=jwt, cfg_scaleC=0.75, cfg_outputBufferStride=stride)
        ref = O.jw_step(case, bands, rhs, "q", nthreads=16).reshape(B, stride)
        got = to.cpu().numpy().reshape(B, stride)
        d, n = np.linalg.norm(got[:, :M] - ref[:, :M], axis=1), np.linalg.norm(ref[:, :M], axis=1)
        assert (d <= TOL[refine] * n).all(), (M, B, stride, d.max(), shape)  # (one row: zero bands, a zero result)
        pad = rhs.reshape(B, stride)[:, M:] if inplace else np.full((B, stride - M), 7.0)
        np.testing.assert_array_equal(got[:, M:], pad)
    b.close()


@pytest.mark.parametrize("refine", [0, 2])
@pytest.mark.parametrize("ub,jwt", [(2, 13), (0, 13)])
def test_shape_edges(ub, jwt, refine):
    for nsys in (1, 17, 130):
        _check([(M, nsys, M) for M in ROWS], ub, jwt, refine)
    _check([(M, 9, M + (-M) % 2 + 4) for M in ROWS], ub, jwt, refine, inplace=True)


@pytest.mark.parametrize("ub,jwt", [(1, 13), (1, 10), (0, 10)])
def test_mixed_bidiagonal_kinds(ub, jwt):
    """The mixed mode's other operator kinds, matvec halos among them."""
    _check([(M, 40, M + 1) for M in ROWS], ub, jwt, 2)
    _check([(M, 40, M) for M in ROWS], ub, jwt, 2, inplace=True)


def test_more_items_than_ctas_and_uneven_sizes():
    """One dominant entry among small ones, and more entries than SMs; launches
    repeated on the same plan (out of place: same result)."""
    _check([(900, 2500, 900)] + [(40 + k, 1 + k % 5, 40 + k) for k in range(30)], 2, 13, 2, reps=3)
    _check([(20 + (37 * k) % 500, 1 + k % 40, 20 + (37 * k) % 500) for k in range(400)], 2, 13, 0, reps=2)


def test_matches_group_kernel():
    import torch

    from pfsolve_b200.api import Batch
    rng = np.random.default_rng(3)
    specs = [(M, 60) for M in (33, 200, 511, 1024)]
    outs = []
    data = [(torch.from_numpy(WL.permute_bands(J.random_bands(rng, M, 2), M)).cuda(),
             torch.from_numpy(rng.uniform(-1, 1, M * B)).cuda()) for M, B in specs]
    for extra in (dict(), dict(rowsPerThread=8)):
        res = [torch.zeros_like(x) for _, x in data]
        b = Batch([dict(M=M, nsys=B, bands=tb, input=x, output=o, inputStride=M, outputStride=M)
                   for (M, B), (tb, x), o in zip(specs, data, res)], upperBanded=2, jw_type=13, **extra)
        b.append()
        torch.cuda.synchronize()
        b.close()
        outs.append(res)
    for a, c in zip(*outs):
        assert ((a - c).norm() / c.norm()).item() <= 1e-13
