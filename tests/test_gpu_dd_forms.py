"""Double-double launches by number of systems: the register form for few, the
table form with the shortest capacity (4, 8, 16 rows per thread of one warp, 16
of two) for many, at the edges of those capacities.  A sample of systems
against the __float128 oracle: 1e-27 relative L2 per system on double-double
storage, 2e-16 on FP64 storage, as the other double-double tests."""
import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,R,W", [(17, 4, 1), (128, 4, 1), (129, 8, 1), (256, 8, 1), (257, 16, 1), (512, 16, 1),
                                   (513, 16, 2), (1024, 16, 2)])
@pytest.mark.parametrize("storage", ["dd", "f64"])
@pytest.mark.parametrize("few", [True, False])
def test_forms(M, R, W, storage, few):
    import torch

    from pfsolve_b200.api import App, last_launch
    B = 5 if few else 20001
    ys = np.arange(B) if few else np.r_[0:12, 9000:9012, B - 12:B]
    for ub, jwt in [(2, 13), (1, 10), (0, 13)]:
        rng = np.random.default_rng(M + ub + jwt)
        bands = WL.permute_bands(J.random_bands(rng, M, ub), M)
        rows = rng.uniform(-1, 1, (B, M))
        sub = O.Case(M=M, batch=len(ys), upperBanded=ub, jw_type=jwt)
        if storage == "dd":
            low = rng.uniform(-1, 1, bands.shape) * 2.0 ** -60
            bdd = np.stack([bands, bands * low], -1).ravel()
            rdd = np.stack([rows, rows * 2.0 ** -61], -1)
            ref = O.jw_step(sub, bdd, rdd[ys].ravel(), "dd")
            tb, to, mode = bdd, rdd.ravel(), dict(quadDoubleDoublePrecision=1)
        else:
            ref = O.jw_step(sub, bands, rows[ys].ravel(), "q")
            tb, to, mode = bands, rows.ravel(), dict(quadDoubleDoublePrecisionDoubleMemory=1)
        tb, to = torch.from_numpy(tb).cuda(), torch.from_numpy(to.copy()).cuda()
        app = App(buffer=tb, outputBuffer=to, M_size=M, size=(M, B), upperBanded=ub, jw_type=jwt, scaleC=1.0, **mode)
        app.append()
        torch.cuda.synchronize()
        info = last_launch()
        assert (info["rowsPerThread"], info["warpsPerSystem"]) == ((4, -(-M // 128)) if few else (R, W)), info
        got = to.cpu().numpy()
        app.close()
        if storage == "dd":
            e, _ = O.rel_errors_dd(got.reshape(B, 2 * M)[ys].ravel(), ref, M, len(ys), M, 0)
        else:
            e, _ = O.rel_errors(got.reshape(B, M)[ys].ravel(), ref, M, len(ys), M)
        assert e <= (1e-27 if storage == "dd" else 2e-16), (M, storage, few, ub, jwt, e)
