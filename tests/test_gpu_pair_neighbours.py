"""Two real systems that one group solves together share nothing but the
operator: a system full of NaN or infinities leaves every other one's bits as
they are, and values beyond the input window are never data, whatever they are.
By tensor copies and by element copies, odd and even numbers of systems."""
import numpy as np
import pytest

from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
# (rows, form) of each precision whose pair form is compiled
CASES = [(p, M) for p, Ms in {"f64": (200, 512, 511, 1001), "mixed": (512, 511, 1001), "f32": (200, 1008, 1001),
                              "f32mem": (200, 512, 511)}.items() for M in Ms]


@pytest.mark.parametrize("prec,M", CASES)
def test_neighbours(prec, M):
    import torch

    from pfsolve_b200.api import App, last_launch_form
    f32 = prec in ("f32", "f32mem")
    dt, B = (torch.float32 if f32 else torch.float64), 40001 if M <= 512 else 24001
    bands = torch.from_numpy(WL.permute_bands(J.random_bands(np.random.default_rng(M), M, 2), M)).to(dt).cuda()
    gen = torch.Generator(device="cuda").manual_seed(M)
    base = torch.rand((B, M), generator=gen, dtype=dt, device="cuda")

    def run(x, window=None):
        x = x.clone()
        app = App(buffer=bands, outputBuffer=x, M_size=M, size=(M, B), upperBanded=2, jw_type=13, scaleC=1.0,
                  doublePrecision=int(not f32), doublePrecisionFloatMemory=int(prec == "f32mem"),
                  mixedPrecisionRefinement=2 if prec == "mixed" else 0,
                  jw_control_bitmask=capi.RUNTIME_INPUTZEROPAD if window else 0)
        app.append(**(dict(inputZeropad=window) if window else {}))
        torch.cuda.synchronize()
        assert last_launch_form() == dict(systemsPerGroup=2, elementCopies=int(M % 8 != 0))
        app.close()
        return x

    clean = run(base)
    assert torch.isfinite(clean).all()
    hit = [0, 3, 1000, 1001, B // 2, B - 2, B - 1]  # first and second of their pairs, the odd last one
    for bad in (float("nan"), float("inf"), -float("inf")):
        x = base.clone()
        x[hit] = bad
        got = run(x)
        rest = torch.ones(B, dtype=torch.bool)
        rest[hit] = False
        assert torch.equal(got[rest.cuda()], clean[rest.cuda()]), bad
        assert not torch.isfinite(got[hit]).any(dim=1).all()
    lo, hi = 3, M - 5
    zero, poison = base.clone(), base.clone()
    zero[:, :lo] = zero[:, hi:] = 0
    poison[:, :lo] = float("nan")
    poison[:, hi:] = float("inf")
    assert torch.equal(run(poison, (lo, hi)), run(zero))
