"""The forms that a plan chooses at the first launch that asks for them (element
copies, pairs of systems, the double-double forms): first asked for inside a
stream capture, and by several threads at once; and what that leaves of a plan's
creation."""
import os
import subprocess
import sys
import threading
import time

import numpy as np
import pytest

from oracle import oracle as O
from pfsolve_b200 import capi
from pfsolve_b200 import workloads as WL

import jwcases as J

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CAPTURE = r"""
import sys
import numpy as np, torch
from pfsolve_b200 import workloads as WL
from pfsolve_b200.api import App, last_launch, last_launch_form
M, B, kw, want = eval(sys.argv[1])
rng = np.random.default_rng(1)
a, c = rng.uniform(0, 1, M), rng.uniform(0, 1, M)
a[0] = c[-1] = 0
d = a + c + rng.uniform(1, 2, M)
w = 2 if kw.get("quadDoubleDoublePrecision") else 1
bands = WL.permute_bands(np.concatenate([-a / d, 1 / d, -c / d]), M)
pad = lambda v: np.stack([v] + [0 * v] * (w - 1), -1).ravel()
tb = torch.from_numpy(pad(bands)).cuda()
x0 = torch.from_numpy(pad(rng.uniform(-1, 1, M * B))).cuda()
x = x0.clone()
side = torch.cuda.Stream()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.stream(side):
    app = App(buffer=tb, outputBuffer=x, stream=side.cuda_stream, M_size=M, size=(M, B), upperBanded=2, jw_type=13,
              scaleC=1.0, **kw)
    graph.capture_begin()
    app.append()  # the first launch of the process
    graph.capture_end()
info, form = last_launch(), last_launch_form()
graph.replay()
torch.cuda.synchronize()
y = x0.clone()
torch.cuda.synchronize()
app.append(outputBuffer=y)
torch.cuda.synchronize()
assert torch.equal(x, y) and not torch.equal(x, x0)
assert (last_launch(), last_launch_form()) == (info, form)
got = (info["kernel"], info["rowsPerThread"], form["systemsPerGroup"], form["elementCopies"])
assert got == want, got
"""


@pytest.mark.parametrize("case", [
    (1001, 20000, dict(doublePrecision=1), (capi.PFSOLVE_KERNEL_STREAMING, 16, 2, 1)),
    (512, 20001, dict(doublePrecision=1, mixedPrecisionRefinement=2), (capi.PFSOLVE_KERNEL_STREAMING, 16, 2, 0)),
    (127, 20001, dict(doublePrecision=1), (capi.PFSOLVE_KERNEL_STREAMING, 4, 1, 1)),
    (200, 40000, dict(doublePrecision=0, quadDoubleDoublePrecision=1), (capi.PFSOLVE_KERNEL_GROUP, 8, 1, 0)),
    (200, 8, dict(doublePrecision=0, quadDoubleDoublePrecision=1), (capi.PFSOLVE_KERNEL_GROUP, 4, 1, 0))])
def test_first_launch_in_capture(case):
    subprocess.run([sys.executable, "-c", CAPTURE, repr(case)], cwd=ROOT, check=True, timeout=300)


def test_first_launch_from_threads():
    """Eight threads launch one new plan at the same time, each on its own
    right-hand sides: the same bits from every one."""
    import torch

    from pfsolve_b200.api import App, last_launch_form
    M, B = 511, 20000
    bands = torch.from_numpy(WL.permute_bands(J.random_bands(np.random.default_rng(3), M, 2), M)).cuda()
    x0 = torch.rand(M * B, dtype=torch.float64, device="cuda")
    for _ in range(5):
        app = App(buffer=bands, outputBuffer=x0, M_size=M, size=(M, B), upperBanded=2, jw_type=13, doublePrecision=1,
                  scaleC=1.0)
        xs, forms = [x0.clone() for _ in range(8)], [None] * 8
        lps = [app.launch_params(outputBuffer=x) for x in xs]
        torch.cuda.synchronize()
        gate = threading.Barrier(8)

        def launch(k):
            gate.wait()
            app.append(lps[k])
            forms[k] = last_launch_form()

        threads = [threading.Thread(target=launch, args=(k,)) for k in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert forms == [dict(systemsPerGroup=2, elementCopies=1)] * 8
        assert all(torch.equal(x, xs[0]) for x in xs) and not torch.equal(xs[0], x0)
        app.close()


@pytest.mark.parametrize("fields", [dict(M_size=256, size=(256, 8)), dict(M_size=1001, size=(1001, 8)),
                                    dict(M_size=512, size=(512, 8), mixedPrecisionRefinement=2)])
def test_creation_cost(fields):
    """Creating a plan chooses none of the further forms: it takes at most 1.15
    times the creation of a plan that has none (kernelPath 1); choosing them
    there took 1.25 to 1.35 times."""
    import torch

    from pfsolve_b200.api import App
    t = torch.zeros(1 << 16, dtype=torch.float64, device="cuda")

    def cost(path):
        ts = []
        for _ in range(400):
            t0 = time.perf_counter()
            app = App(buffer=t, outputBuffer=t, upperBanded=2, jw_type=13, doublePrecision=1, kernelPath=path, **fields)
            ts.append(time.perf_counter() - t0)
            app.close()
        return sorted(ts)[40]

    cost(0)
    assert min(cost(0) / cost(1) for _ in range(5)) <= 1.15
