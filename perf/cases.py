"""The calls this library is timed on: what a spectral code asks of the
Jones-Worland path, one family per entry of ``FAMILIES``, each over its range
of sizes, options and storage types.

Right-hand sides come from a seeded generator on the GPU; operators are seeded
too.  Steps that solve in place are given operators whose rows conserve a
constant (an implicit diffusion step with zero-flux ends), so that repeated
passes neither grow nor die out.  ``exact`` restates every family in plain
torch in 64 bits from the natural-order bands.
"""
import math

import numpy as np
import torch

from pfsolve_b200 import workloads as WL
from pfsolve_b200.api import App, Batch, append_chain

F64 = torch.float64


def listed():
    return [
        # the smallest call in use: one degree's fused 3-band matvec and bidiagonal step on a few hundred
        # right-hand sides that stay in L2; launch latency counts
        dict(name="chain_small", kind="chain_real", n=256, b=512),
        # the headline call: 5-band matvec, tridiagonal solve and XXII -> packed in one kernel on 65 536
        # complex right-hand sides
        dict(name="chain_complex", kind="chain_complex", n=1024, b=65536),
        # the plain FP64 step on a ragged truncation: an odd row count, rows packed at that odd stride
        dict(name="step_odd", kind="step", n=1001, b=60000, ub=2, prec="f64", weak=False),
        # FP32 solve with two FP64 refinement sweeps on a weakly dominant system
        dict(name="step_mixed", kind="step", n=512, b=131072, ub=2, prec="mixed", weak=True),
        # FP32 storage and arithmetic, the reference's default precision
        dict(name="step_f32", kind="step", n=512, b=131072, ub=2, prec="f32", weak=True),
        # quad emulation: double-double storage and arithmetic
        dict(name="step_dd", kind="step", n=512, b=32768, ub=2, prec="dd", weak=True),
        # a long radial grid, beyond one CTA's rows
        dict(name="step_long", kind="step", n=16384, b=8192, ub=2, prec="f64", weak=True),
        # four consecutive order-changing steps in one launch
        dict(name="steps_k4", kind="ksteps", n=512, b=131072, k=4),
        # ALT stride-2 mode: even and odd rows are two systems of one row set
        dict(name="alt", kind="alt", n=1024, b=131072),
        # radial transform there and back: DCT-II, then DCT-III of its result
        dict(name="dct_round", kind="dct", n=2048, b=32768),
        # one spectral timestep: every harmonic degree its own length, matrix and number of systems
        dict(name="timestep", kind="timestep", lmax=511, nmax=512),
        # a batch of solve requests of mixed sizes, FP32 solve with two FP64 refinement sweeps
        dict(name="requests", kind="requests", n=32, seed=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, lo, hi):
    """A row count spread over its logarithm: half of them multiples of 16."""
    n = _log(rng, lo, hi)
    return max(lo, min(hi, n if rng.random() < 0.5 else (n + 15) // 16 * 16))


def _batch(rng, n, values):
    """Systems of n rows, 2^18 ... `values` values in all, odd counts among them."""
    return max(1, _log(rng, 1 << 18, values) // n)


def draw(rng):
    kind = rng.choice(["chain_real", "chain_complex", "step", "step", "step", "step", "long", "ksteps", "alt", "dct",
                       "timestep", "requests"])
    if kind == "chain_real":
        return dict(kind=kind, n=_rows(rng, 32, 1024), b=_log(rng, 64, 16384))
    if kind == "chain_complex":
        n = _rows(rng, 128, 2048)
        return dict(kind=kind, n=n, b=_batch(rng, n, 1 << 26))
    if kind == "step":
        prec = rng.choice(["f64", "f64", "mixed", "f32", "f32mem", "dd", "ddmem"])
        dd = prec in ("dd", "ddmem")
        n = _rows(rng, 33, 1024 if dd else 4096)
        ub = 2 if prec == "mixed" else rng.choice([0, 1, 2, 2])
        return dict(kind=kind, n=n, b=_batch(rng, n, 1 << (24 if dd else 26)), ub=ub, prec=prec,
                    weak=rng.random() < 0.5)
    if kind == "long":
        n = _rows(rng, 4097, 65536)
        return dict(kind="step", n=n, b=_batch(rng, n, 1 << 27), ub=rng.choice([0, 1, 2, 2]), prec="f64",
                    weak=rng.random() < 0.5)
    if kind == "ksteps":
        n = _rows(rng, 64, 2048)
        return dict(kind=kind, n=n, b=_batch(rng, n, 1 << 26), k=rng.randint(2, 8))
    if kind == "alt":
        n = _rows(rng, 64, 8192)
        return dict(kind=kind, n=n, b=_batch(rng, n, 1 << 27))
    if kind == "dct":
        n = 1 << rng.randint(6, 12)
        return dict(kind=kind, n=n, b=_batch(rng, n, 1 << 26))
    if kind == "timestep":
        lmax = _log(rng, 31, 511)
        return dict(kind=kind, lmax=lmax, nmax=rng.randint(lmax // 2 + 32, 512))
    return dict(kind=kind, n=_log(rng, 4, 64), seed=rng.randrange(1 << 20))


# ---- operators (natural order) and right-hand sides -------------------------

def _diffusion(rng, m, weak=False):
    """Normalised tridiagonal rows (ld, md, ud): couplings -a, -c in U(0, 1),
    diagonal a + c + U(1, 2), or 1.05 (a + c) when weak; the right-hand side's
    factor md makes a constant the step's fixed point."""
    a, c = rng.uniform(0, 1, m), rng.uniform(0, 1, m)
    a[0] = 0
    c[-1] = 0
    e = 0.05 * (a + c) if weak else rng.uniform(1, 2, m)
    d = a + c + e
    d[d == 0] = 1
    return -a / d, e / d, -c / d


def _bidiagonal(rng, m, upper):
    """Unit bidiagonal rows with couplings -h, h in U(0, 1/2), and the factor
    1 - h: (factor, coupling)."""
    h = rng.uniform(0, 0.5, m)
    h[-1 if upper else 0] = 0
    return 1 - h, -h


def _step_bands(case, seed):
    """(factor, lower coupling or None, upper coupling or None) of a step."""
    rng = np.random.default_rng(seed)
    n, ub = case["n"], case["ub"]
    if ub == 2:
        ld, md, ud = _diffusion(rng, n, case["weak"])
        return md, ld, ud
    md, off = _bidiagonal(rng, n, ub == 0)
    return (md, off, None) if ub == 1 else (md, None, off)


def _average(rng, m, kl, ku):
    """dgbmv bands (band-major by column) of rows that are weighted averages."""
    w = rng.uniform(0.1, 1, (kl + ku + 1, m))  # w[k, r] multiplies x[r + ku - k]
    col = np.arange(m)[None, :] + ku - np.arange(kl + ku + 1)[:, None]
    w[(col < 0) | (col >= m)] = 0
    w /= w.sum(0)
    a = np.zeros_like(w)
    for k in range(kl + ku + 1):
        ok = (col[k] >= 0) & (col[k] < m)
        a[k, col[k][ok]] = w[k, ok]
    return w, a.reshape(-1)


def _ksteps_bands(case, seed):
    """Per step (factor, upper coupling, lower coupling) rows of upperBanded 1,
    jw_type 10: the factor acts in the first step only, and is small enough for
    what the steps' couplings add."""
    rng = np.random.default_rng(seed)
    out = []
    for s in range(case["k"]):
        m = case["n"] - s
        lo, up = rng.uniform(-0.25, 0.25, (2, m))
        lo[0] = up[0] = 0
        out.append((rng.uniform(0.3, 0.6, m) * 0.85 ** (case["k"] - 2), up, lo))
    return out


def _gpu(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t if dtype is None else t.to(dtype)


def _uniform(seed, count, dtype=F64):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.rand(count, generator=g, device="cuda", dtype=F64).mul_(2).sub_(1).to(dtype)


def _normal(seed, count):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(count, generator=g, device="cuda", dtype=F64)


def _pairs(t):
    """Double-double values of FP64 ones: a low word 2^-60 of the high one."""
    return torch.stack([t, t * 2.0 ** -60], -1).reshape(-1)


PRECISION = {
    "f64": dict(doublePrecision=1), "mixed": dict(doublePrecision=1, mixedPrecisionRefinement=2),
    "f32": dict(doublePrecision=0), "f32mem": dict(doublePrecision=0, doublePrecisionFloatMemory=1),
    "dd": dict(doublePrecision=0, quadDoubleDoublePrecision=1),
    "ddmem": dict(doublePrecision=0, quadDoubleDoublePrecisionDoubleMemory=1),
}


def _request_specs(case):
    return [(r.M, r.nrhs) for r in WL.config5_requests(case["n"], seed=case["seed"])]


def _timestep_sizes(case):
    return [(l, case["nmax"] - l // 2, 2 * l + 1) for l in range(case["lmax"] + 1)]


def _timestep_bands(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _, n, _ in _timestep_sizes(case):
        d, s = rng.uniform(1, 2, n), rng.uniform(-0.5, 0.5, n)
        s[-1] = 0
        out.append((1 / d, s / d, rng.uniform(-1, 1, (3, n))))  # factor, upper coupling, dgbmv by column
    return out


# ---- one state per family -----------------------------------------------------

def _prepare_chain_real(case, seed):
    n, b = case["n"], case["b"]
    rng = np.random.default_rng(seed)
    md, off = _bidiagonal(rng, n, True)
    _, a = _average(rng, n, 1, 1)
    bands = _gpu(WL.permute_bands(np.concatenate([md, off, np.zeros(n)]), n))
    mat, x = _gpu(a), _uniform(seed, n * b)
    dg = App(buffer=mat, outputBuffer=x, M_size=n, size=(n, b), LDA=3, KU=1, KL=1, doublePrecision=1)
    jw = App(buffer=bands, outputBuffer=x, M_size=n, size=(n, b), upperBanded=0, jw_type=13, doublePrecision=1,
             scaleC=1.0)
    apps = [dg, jw]
    return dict(kind="chain", apps=apps, lps=[p.launch_params() for p in apps], keep=[bands, mat], out=x)


def _prepare_chain_complex(case, seed):
    n, b = case["n"], case["b"]
    rng = np.random.default_rng(seed)
    ld, md, ud = _diffusion(rng, n)
    mat = _gpu(rng.uniform(-1, 1, 5 * n))
    bands = _gpu(WL.permute_bands(np.concatenate([ld, md, ud]), n))
    x = _normal(seed, 2 * n * b)
    out = torch.empty_like(x)
    dg = App(buffer=mat, outputBuffer=x, M_size=n, size=(n, 2 * b), LDA=5, KU=2, KL=2, doublePrecision=1)
    jw = App(buffer=bands, outputBuffer=x, M_size=n, size=(n, 2 * b), upperBanded=2, jw_type=13, doublePrecision=1,
             scaleC=1.0)
    bl = App(buffer=x, outputBuffer=out, M_size=n, size=(n, b), block=7, doublePrecision=1)
    apps = [dg, jw, bl]
    return dict(kind="chain", apps=apps, lps=[p.launch_params() for p in apps], keep=[mat, bands, x], out=out)


def _prepare_step(case, seed):
    n, b, prec = case["n"], case["b"], case["prec"]
    md, lo, up = _step_bands(case, seed)
    if case["ub"] == 2:
        nat = [lo, md, up]
    else:  # jw_type 13 reads the coupling beside the factor
        nat = [lo, md, np.zeros(n)] if case["ub"] == 1 else [md, up, np.zeros(n)]
    bands = WL.permute_bands(np.concatenate(nat), n)
    dtype = torch.float32 if prec in ("f32", "f32mem") else F64
    bands, x = _gpu(bands, dtype), _uniform(seed, n * b, dtype)
    if prec == "dd":
        bands, x = _pairs(bands), _pairs(x)
    app = App(buffer=bands, outputBuffer=x, M_size=n, size=(n, b), upperBanded=case["ub"], jw_type=13, scaleC=1.0,
              **PRECISION[prec])
    out = dict(high=x.view(-1, 2)[:, 0], low=x.view(-1, 2)[:, 1]) if prec == "dd" else x
    return dict(kind="app", apps=[app], lps=[app.launch_params()], keep=[bands], out=out)


def _prepare_ksteps(case, seed):
    n, b, k = case["n"], case["b"], case["k"]
    r = WL.steps_registers(n, 1, k)
    bands = []
    for s, (md, up, lo) in enumerate(_ksteps_bands(case, seed)):
        m = len(md)
        perm = WL.steps_band_order(m, r)
        buf = np.zeros(3 * m)
        for j, band in enumerate((md, up, lo) if s == 0 else (up, lo)):
            buf[j * m + perm] = band
        bands.append(_gpu(buf))
    x = _uniform(seed, n * b)
    app = App(buffer=bands, outputBuffer=x, M_size=n, size=(n, b), upperBanded=1, jw_type=10, doublePrecision=1,
              scaleC=1.0, numConsecutiveJWIterations=k, useMultipleInputBuffers=k)
    return dict(kind="app", apps=[app], lps=[app.launch_params()], keep=bands, out=x)


def _alt_bands(case, seed):
    """(ld, md, ud) over all rows: the even and the odd rows' systems interleaved."""
    rng = np.random.default_rng(seed)
    nat = np.zeros((3, case["n"]))
    for h in (0, 1):
        nat[:, h::2] = _diffusion(rng, len(range(h, case["n"], 2)))
    return nat


def _prepare_alt(case, seed):
    n, b = case["n"], case["b"]
    span, pos = WL.alt_band_span(n), WL.alt_positions(n)
    buf = np.zeros(3 * span)
    for j, band in enumerate(_alt_bands(case, seed)):
        buf[j * span + pos] = band
    bands, x = _gpu(buf), _uniform(seed, n * b)
    app = App(buffer=bands, outputBuffer=x, M_size=n, size=(n, b), upperBanded=2, jw_type=113, doublePrecision=1,
              scaleC=1.0)
    return dict(kind="app", apps=[app], lps=[app.launch_params()], keep=[bands], out=x)


def _prepare_dct(case, seed):
    n, b = case["n"], case["b"]
    x = _normal(seed, n * b)
    y, z = torch.empty_like(x), torch.empty_like(x)
    there = App(buffer=x, outputBuffer=y, size=(n, b), performDCT=2, doublePrecision=1)
    back = App(buffer=y, outputBuffer=z, size=(n, b), performDCT=3, doublePrecision=1)
    apps = [there, back]
    return dict(kind="app", apps=apps, lps=[p.launch_params() for p in apps], keep=[x],
                out=dict(spectral=y, physical=z))


def _prepare_timestep(case, seed):
    sizes = _timestep_sizes(case)
    total = 2 * sum(n * s for _, n, s in sizes)
    inp = _normal(seed, total)
    out = torch.empty_like(inp)
    jw, dg = [], []
    for md, up, a in _timestep_bands(case, seed):
        jw.append(WL.permute_bands(np.concatenate([md, up, np.zeros_like(md)]), len(md)))
        dg.append(a.reshape(-1))
    bands = _gpu(np.concatenate(jw + dg))
    at, mat, off, entries = bands.data_ptr(), bands.data_ptr() + 8 * sum(map(len, jw)), 0, []
    for l, n, s in sizes:
        entries.append(dict(M=n, nsys=s, bands=at, dgbmvBands=mat, input=inp.data_ptr() + 8 * off,
                            output=out.data_ptr() + 8 * off, inputStride=n, outputStride=n, lshift=l, scaleS=-0.5,
                            scaleC=1.0))
        at, mat, off = at + 24 * n, mat + 24 * n, off + 2 * n * s
    batch = Batch(entries, upperBanded=0, jw_type=13, LDA=3, KU=1, KL=1, block=307)
    return dict(kind="batch", batch=batch, keep=[bands, inp], out=out)


def _prepare_requests(case, seed):
    specs = _request_specs(case)
    bands, x, out, entries = [], [], [], []
    for i, (n, b) in enumerate(specs):
        ld, md, ud = _diffusion(np.random.default_rng([seed, i]), n)
        bands.append(_gpu(WL.permute_bands(np.concatenate([ld, md, ud]), n)))
        x.append(_uniform(seed + 1000003 * i, n * b))
        out.append(torch.empty_like(x[-1]))
        entries.append(dict(M=n, nsys=b, bands=bands[-1], input=x[-1], output=out[-1], inputStride=n, outputStride=n,
                            scaleC=1.0))
    batch = Batch(entries, upperBanded=2, jw_type=13, mixedPrecisionRefinement=2)
    return dict(kind="batch", batch=batch, keep=[bands, x], out=out)


FAMILIES = {"chain_real": _prepare_chain_real, "chain_complex": _prepare_chain_complex, "step": _prepare_step,
            "ksteps": _prepare_ksteps, "alt": _prepare_alt, "dct": _prepare_dct, "timestep": _prepare_timestep,
            "requests": _prepare_requests}


def prepare(case, seed):
    return FAMILIES[case["kind"]](case, seed)


def run(state):
    if state["kind"] == "chain":
        append_chain(state["apps"], state["lps"])
    elif state["kind"] == "batch":
        state["batch"].append()
    else:
        for app, lp in zip(state["apps"], state["lps"]):
            app.append(lp)
    return state["out"]


def work(case):
    """Bytes: each right-hand side read once and each result written once, and
    the operators; flops: the matvec and the solve with a factored operator."""
    kind = case["kind"]
    if kind == "timestep":
        rows = sum(n * s for _, n, s in _timestep_sizes(case))
        return dict(bytes=32.0 * rows + 48.0 * sum(n for _, n, _ in _timestep_sizes(case)), flops=2 * 9.0 * rows)
    if kind == "requests":
        specs = _request_specs(case)
        rows = sum(n * b for n, b in specs)
        return dict(bytes=16.0 * rows + 24.0 * sum(n for n, _ in specs), flops=5.0 * rows)
    n, b = case["n"], case["b"]
    rows = float(n * b)
    if kind == "chain_real":
        return dict(bytes=16 * rows + 40.0 * n, flops=8 * rows)
    if kind == "chain_complex":
        return dict(bytes=32 * rows + 64.0 * n, flops=2 * 14 * rows)
    if kind == "dct":
        return dict(bytes=2 * 16 * rows, flops=2 * 2.5 * rows * math.log2(n))
    if kind == "ksteps":
        k = case["k"]
        return dict(bytes=8 * (rows + (n - k + 1.0) * b) + 24.0 * n * k, flops=4 * k * rows)
    if kind == "alt":
        return dict(bytes=16 * rows + 24.0 * n, flops=5 * rows)
    prec = case["prec"]
    word = {"f32": 4, "f32mem": 4, "dd": 16}.get(prec, 8)
    ops = 5 if case["ub"] == 2 else 3
    each = {"dd": 12, "ddmem": 12, "mixed": 4}.get(prec, 1)  # operations per multiply-add; solves and residuals
    return dict(bytes=2 * word * rows + 3.0 * word * n, flops=each * ops * rows)


# ---- the same in 64 bits, plain torch -------------------------------------------

def _solve(y, lo, up):
    """x of (I + lo at row - 1 + up at row + 1) x = y by elimination down the
    rows and back substitution; y: rows x systems, overwritten."""
    n = y.shape[0]
    if lo is not None and up is not None:
        g, inv = np.empty(n), np.empty(n)  # eliminated upper coupling, reciprocal pivot
        prev = 0.0
        for i in range(n):
            inv[i] = 1 / (1 - (lo[i] * prev if i else 0.0))
            prev = g[i] = up[i] * inv[i]
        y[0] *= inv[0]
        for i in range(1, n):
            torch.add(y[i], y[i - 1], alpha=-lo[i], out=y[i]).mul_(inv[i])
        up = g
    elif lo is not None:
        for i in range(1, n):
            y[i].add_(y[i - 1], alpha=-lo[i])
        return y
    for i in range(n - 2, -1, -1):
        y[i].add_(y[i + 1], alpha=-up[i])
    return y


def _rowwise(x, n, b):
    return x.view(b, n).t().contiguous()


def _flat(y):
    return y.t().contiguous().view(-1)


def _col(a):
    return _gpu(a)[:, None]


def _matvec(x, w, ku):
    """Banded rows: y[r] = sum_k w[k, r] x[r + ku - k]."""
    n, y = x.shape[0], torch.zeros_like(x)
    for k in range(len(w)):
        d = ku - k
        r0, r1 = max(0, -d), min(n, n - d)
        if r1 > r0:
            y[r0:r1] += _col(w[k][r0:r1]) * x[r0 + d:r1 + d]
    return y


def _by_row(a, n, kl, ku):
    """Row weights of a dgbmv matrix stored by column."""
    a = np.asarray(a).reshape(kl + ku + 1, n)
    w = np.zeros_like(a)
    for k in range(kl + ku + 1):
        d = ku - k
        r0, r1 = max(0, -d), min(n, n - d)
        w[k, r0:r1] = a[k, r0 + d:r1 + d]
    return w


def _packed(y, b):
    """rows x (re, im of each system) -> packed complex systems."""
    n = y.shape[0]
    return y.view(n, b, 2).permute(1, 0, 2).contiguous().view(-1)


def _sph_lapl_a(n, l, s):
    x = np.arange(n, dtype=np.float64)
    return (4 * (x + l + 2) * (x + l + 3)
            * np.sqrt((x + 1) * (x + 2) / ((x + s + l + 2.5) * (x + s + l + 3.5))))


def exact(case, seed):
    kind = case["kind"]
    if kind == "timestep":
        sizes = _timestep_sizes(case)
        inp = _normal(seed, 2 * sum(n * s for _, n, s in sizes))
        off, out = 0, []
        for (l, n, s), (md, up, a) in zip(sizes, _timestep_bands(case, seed)):
            x = _rowwise(inp[off:off + 2 * n * s], n, 2 * s)
            off += 2 * n * s
            y = _solve(_matvec(x, _by_row(a, n, 1, 1) * md, 1), None, up)
            out.append(_packed(y * _col(_sph_lapl_a(n, l, -0.5)), s))
        return torch.cat(out)
    if kind == "requests":
        out = []
        for i, (n, b) in enumerate(_request_specs(case)):
            ld, md, ud = _diffusion(np.random.default_rng([seed, i]), n)
            out.append(_flat(_solve(_rowwise(_uniform(seed + 1000003 * i, n * b), n, b) * _col(md), ld, ud)))
        return out
    n, b = case["n"], case["b"]
    if kind == "chain_real":
        rng = np.random.default_rng(seed)
        md, off = _bidiagonal(rng, n, True)
        w, _ = _average(rng, n, 1, 1)
        return _flat(_solve(_matvec(_rowwise(_uniform(seed, n * b), n, b), w * md, 1), None, off))
    if kind == "chain_complex":
        rng = np.random.default_rng(seed)
        ld, md, ud = _diffusion(rng, n)
        w = _by_row(rng.uniform(-1, 1, 5 * n), n, 2, 2)
        return _packed(_solve(_matvec(_rowwise(_normal(seed, 2 * n * b), n, 2 * b), w * md, 2), ld, ud), b)
    if kind == "dct":
        x = _normal(seed, n * b).view(b, n)
        i = np.arange(n)
        c = _gpu(2 * np.cos(np.pi * ((2 * i[:, None] + 1) * i[None, :] % (4 * n)) / (2 * n)))  # point x mode
        y = x @ c
        return dict(spectral=y.view(-1), physical=2 * n * x.reshape(-1))
    if kind == "ksteps":
        x0 = _rowwise(_uniform(seed, n * b), n, b)
        x = x0.clone()
        for s, (md, up, lo) in enumerate(_ksteps_bands(case, seed)):
            m = n - s
            y = x[:m] * _col(md) if s == 0 else x[:m].clone()
            inner = m if s else m - 1  # the last row couples to the row that has left the system
            y[:inner] += _col(up[:inner]) * x[1:inner + 1]
            x[:m] = _solve(y, lo, None)
        x[m:] = x0[m:]  # rows that left the system are not written
        return _flat(x)
    if kind == "alt":
        x = _rowwise(_uniform(seed, n * b), n, b)
        nat = _alt_bands(case, seed)
        for h in (0, 1):
            ld, md, ud = nat[:, h::2]
            x[h::2] = _solve(x[h::2] * _col(md), ld, ud)
        return _flat(x)
    md, lo, up = _step_bands(case, seed)
    dtype = torch.float32 if case["prec"] in ("f32", "f32mem") else F64
    if dtype == torch.float32:  # the operator as it is stored
        md, lo, up = (None if v is None else v.astype(np.float32).astype(np.float64) for v in (md, lo, up))
    x = _solve(_rowwise(_uniform(seed, n * b, dtype).to(F64), n, b) * _col(md), lo, up)
    return dict(high=_flat(x), low=None) if case["prec"] == "dd" else _flat(x)
