"""The work a user of this library has it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes a user's inputs and context for it on the GPU, `run` takes
them through the public entry points once, and `exact` gives the same results from plain torch in 64 bits.
Four kinds:

* box       one periodic-box evaluation: PowerSpectrum.paint + power (any precision, host or device arrays);
* gradient  a forward evaluation and PowerSpectrum.backward of a loss on its multipoles;
* batch     many mocks of different boxes and grids in one run_batch call;
* survey    the survey estimator: SurveySpectrum.power on a data and a random catalogue.

Spectra of the FP32-mixed and deterministic modes are returned as float32, the precision those modes hold
them to; FP64 spectra as float64. The multipoles of one spectrum are one [5][NK] array: an error of P_l is
judged against the spectrum's power, as the estimator's noise is.
"""
import math

import numpy as np
import torch

import capow_gb300 as cg

# nfields, exponents of v of the fields A and B, imaginary part, mean-subtracted A, shot-noise moment
FIELDS = {0: (1, 0, 0, 0, 1, 0), 1: (2, 0, 1, 1, 1, 1), 2: (1, 1, 0, 0, 0, 2)}
OMEGA_M, REDSHIFT = 0.3089, 0.1


def _box(name, **kw):
    c = dict(kind="box", nx=128, ny=128, nz=128, lx=1000.0, ly=1000.0, lz=1000.0, order=3, interlace=1, los=3, momentum=0,
             spectra="", odd=0, out2d=0, nmu=1, log=0, nk=41, mink=0.0, maxk=0.41, n=2097152, particles="lattice",
             dtype="f32", weights=False, host=False, precision="fp32")
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a quick look at a small catalogue, every multipole (launches and latency count)
        _box("small_32_tsc", nx=32, ny=32, nz=32, n=20000, particles="uniform", dtype="f64", momentum=1, odd=1, nk=16,
             maxk=0.1),
        # the plain run of the command-line tool: a float64 catalogue of 2M particles, CIC on 128^3
        _box("plain_128_cic", order=2, particles="uniform", dtype="f64"),
        # an odd-shaped box with weights, log k bins and the 2-D (k, mu) histogram
        _box("ragged_100_2d", nx=100, ny=96, nz=75, lx=1000.0, ly=900.0, lz=800.0, order=2, los=2, n=777777,
             particles="random", weights=True, log=1, out2d=1, nmu=5, nk=20, mink=-1.9, maxk=-0.55),
        # a halo-like catalogue (random order) on a grid that is no power of two, the three spectra
        _box("halos_192_tsc", nx=192, ny=192, nz=192, los=1, spectra="dd,dp,pp", nk=60, maxk=0.6, n=3000017,
             particles="random"),
        # a catalogue that lies in host memory, one call after the other (copy included)
        _box("host_256_tsc", nx=256, ny=256, nz=256, momentum=1, los=2, nk=80, maxk=0.8, n=8000000,
             particles="lattice", host=True),
        # the headline evaluation: 16.7M particles on a 512^3 TSC grid, three spectra from one paint
        _box("headline_512_tsc", nx=512, ny=512, nz=512, spectra="dd,dp,pp", nk=161, maxk=1.61, n=16777216),
        # the large single mock: 134M particles, CIC on 1024^3
        _box("large_1024_cic", nx=1024, ny=1024, nz=1024, lx=2000.0, ly=2000.0, lz=2000.0, order=2, spectra="dd,dp,pp",
             nk=160, maxk=1.6, n=134217728),
        # the plain FP64 path, for users who want the reference's arithmetic
        _box("fp64_256_tsc", nx=256, ny=256, nz=256, spectra="dd,dp,pp", nk=81, maxk=0.81, precision="fp64"),
        # the bit-reproducible mode
        _box("det_256_tsc", nx=256, ny=256, nz=256, spectra="dd,dp,pp", nk=81, maxk=0.81, n=4096000, precision="det"),
        # gradients of a loss on P0 and P2 with respect to 16.7M particles (inference, field-level fits)
        _box("gradient_256_tsc", kind="gradient", nx=256, ny=256, nz=256, nk=80, maxk=0.8, n=16777216),
        # a set of mocks of several boxes and grids in one call
        {"name": "batch_16", "kind": "batch", "mocks": 16, "pick": 1000, "nmin": 500000, "nmax": 8000000},
        # a full-sky survey around an observer at the box centre: 3M objects, ten times as many randoms
        {"name": "survey_512_tsc", "kind": "survey", "n": 512, "L": 2000.0, "order": 3, "interlace": 1, "odd": 0, "nk": 100,
         "maxk": 0.5, "ndata": 3181806, "ratio": 10, "precision": "fp32"},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["box"] * 6 + ["fp64", "det", "gradient", "batch", "survey", "survey"])
    if kind == "batch":
        return {"kind": "batch", "mocks": rng.randint(2, 24), "pick": rng.randrange(1 << 20), "nmin": 200000,
                "nmax": logint(1000000, 8000000)}
    if kind == "survey":
        n = rng.choice([64, 128, 256, 256, 512, logint(60, 300) // 2 * 2])
        return {"kind": "survey", "n": n, "L": 2000.0, "order": rng.choice([2, 3, 3]), "interlace": rng.choice([0, 1, 1]),
                "odd": rng.choice([0, 0, 1]), "nk": rng.randint(20, 100), "maxk": math.pi * n / 2000.0 * rng.uniform(0.4, 1.0),
                "ndata": logint(20000, 2000000), "ratio": rng.randint(2, 20), "precision": "fp32"}
    big = {"box": 512, "gradient": 256, "fp64": 192, "det": 256}[kind]
    if rng.random() < 0.65:  # powers of two, not always the same along every axis
        s = 1 << rng.randint(5, int(math.log2(big)))
        axes = [s, s, s] if rng.random() < 0.5 else [max(16, min(big, s * rng.choice([1, 1, 2]) // rng.choice([1, 1, 2]))) for _ in range(3)]
        axes[2] = max(32, axes[2])
    else:
        s = logint(24, min(big, 320))
        axes = [s, s, s] if rng.random() < 0.4 else [max(20, s + rng.randint(-9, 9)) for _ in range(3)]
    side = rng.uniform(300.0, 2000.0)
    L = [round(side * a / s, 3) for a in axes]  # cells near cubic
    knyq = min(math.pi * a / b for a, b in zip(axes, L))
    log = rng.random() < 0.15
    top = knyq * rng.uniform(0.4, 1.05)
    nk = rng.randint(10, 200)
    spectra = rng.choice(["", "", "dd", "dd,dp,pp"])
    lattice = rng.random() < 0.5
    n = logint(10000, 8000000)
    if lattice:
        n = max(16, round(n ** (1.0 / 3.0))) ** 3
    return _box("", kind="gradient" if kind == "gradient" else "box", nx=axes[0], ny=axes[1], nz=axes[2], lx=L[0], ly=L[1], lz=L[2],
                order=rng.choice([1, 2, 2, 3, 3, 3]) if kind != "gradient" else rng.choice([2, 3]), interlace=rng.choice([0, 1, 1]),
                los=rng.choice([0, 1, 2, 3, 3]), momentum=0 if spectra or kind == "gradient" else rng.choice([0, 0, 1, 2]),
                spectra="" if kind == "gradient" else spectra, odd=rng.choice([0, 0, 0, 1]),
                out2d=1 if kind == "box" and rng.random() < 0.1 else 0, nmu=rng.randint(2, 8), log=int(log), nk=nk,
                mink=math.log10(top) - 1.3 if log else 0.0, maxk=math.log10(top) if log else top, n=n,
                particles="lattice" if lattice else rng.choice(["uniform", "random"]), dtype=rng.choice(["f32", "f32", "f64"]),
                weights=rng.random() < 0.2, host=kind == "box" and rng.random() < 0.2,
                precision={"fp64": "fp64", "det": "det"}.get(kind, "fp32"))


# ------------------------------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 7919 + 12345)
    return g


def _displacement(m, L, rms, g):
    """A Gaussian displacement field Psi on an m^3 mesh: P(k) = k^-1.5 exp(-(k/0.5)^2), rms length `rms`."""
    dev = _device()
    wk = torch.fft.rfftn(torch.randn(m, m, m, generator=g, device=dev))
    k1 = torch.fft.fftfreq(m, d=1.0 / m, device=dev) * (2 * math.pi / L)
    kz = torch.fft.rfftfreq(m, d=1.0 / m, device=dev) * (2 * math.pi / L)
    k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    wk *= k2 ** -1.375 * torch.exp(-2.0 * k2)  # sqrt(P) / k^2
    wk[0, 0, 0] = 0.0
    psi = [torch.fft.irfftn(1j * k * wk, s=(m, m, m)) for k in (k1[:, None, None], k1[None, :, None], kz[None, None, :])]
    s = rms / math.sqrt(float(sum((p * p).mean() for p in psi)) + 1e-30)
    return [p.mul_(s) for p in psi]


def _particles(n, L, grid, how, los, dtype, weights, g):
    """x, y, z, v_los (and w) of n particles in the box [0, L): a displaced lattice in lattice order, displaced
    random points in random order (both follow the same kind of field), or uniform points."""
    dev, axis = _device(), 2 if los == 0 else los - 1
    rms = 1.5 * L[0] / grid
    if how == "uniform":
        pos = [torch.rand(n, generator=g, device=dev, dtype=torch.float64) * a for a in L]
        v = 300.0 * torch.randn(n, generator=g, device=dev)
    elif how == "lattice":
        m = round(n ** (1.0 / 3.0))
        psi = _displacement(m, L[0], rms, g)
        pos = []
        for a in range(3):
            q = (torch.arange(m, device=dev, dtype=torch.float64) + 0.5) * (L[a] / m)
            pos.append((q.view([m if b == a else 1 for b in range(3)]) + psi[a]).reshape(-1))
        v = 80.0 * psi[axis].reshape(-1) + 150.0 * torch.randn(n, generator=g, device=dev)
        del psi
    else:
        m = 128
        psi = _displacement(m, L[0], 2.0 * rms, g)
        q = [torch.rand(n, generator=g, device=dev, dtype=torch.float64) for _ in range(3)]
        c = [(t * m).long().clamp_(0, m - 1) for t in q]
        idx = (c[0] * m + c[1]) * m + c[2]
        d = [p.reshape(-1)[idx] for p in psi]
        pos = [t * a + s for t, a, s in zip(q, L, d)]
        v = 80.0 * d[axis] + 150.0 * torch.randn(n, generator=g, device=dev)
    dt = torch.float64 if dtype == "f64" else torch.float32
    out = []
    for p, a in zip(pos, L):
        p = torch.remainder(p, a).to(dt)
        out.append(torch.where((p >= torch.tensor(a, dtype=dt, device=dev)) | (p < 0), torch.zeros_like(p), p).contiguous())
    del pos
    out.append(v.to(dt).contiguous())
    out.append((0.5 + torch.rand(n, generator=g, device=dev)).to(dt) if weights else None)
    return out


def _params(c):
    return cg.Params(NX=c["nx"], NY=c["ny"], NZ=c["nz"], XMIN=0.0, XMAX=c["lx"], YMIN=0.0, YMAX=c["ly"], ZMIN=0.0, ZMAX=c["lz"],
                     InterpOrder=c["order"], DoInterlacing=c["interlace"], NK=c["nk"], NMU=c["nmu"], Output2D=c["out2d"],
                     OutputLog=c["log"], Mink=c["mink"], Maxk=c["maxk"], Omega_m=OMEGA_M, Redshift=REDSHIFT, LOS=c["los"],
                     Momentum=c["momentum"], Odd_Multipoles=c["odd"])


def _box_inputs(c, seed):
    return _particles(c["n"], (c["lx"], c["ly"], c["lz"]), c["nx"], c["particles"], c["los"], c["dtype"], c["weights"], _gen(seed))


def _loss_gradient(c):
    """dL/dP0 and dL/dP2 of a fit's chi^2: weights per bin that change sign and size over the bins."""
    b = np.arange(c["nk"])
    return {"Pk0": 1e-3 * np.cos(0.37 * b + 0.2), "Pk2": 5e-4 * np.sin(0.23 * b + 0.5)}


def _mock_cases(c):
    """The mocks of a batch: boxes, grids and sizes from the case alone."""
    r = np.random.default_rng(c["pick"])
    out = []
    for i in range(c["mocks"]):
        L, ng = float(r.uniform(500.0, 1500.0)), int(r.choice([128, 192, 256]))
        side = max(8, int(round(math.exp(r.uniform(math.log(c["nmin"]), math.log(c["nmax"]))) ** (1.0 / 3.0))))
        nk = int(math.floor(math.pi * ng / L / 0.01))
        out.append(_box("", nx=ng, ny=ng, nz=ng, lx=L, ly=L, lz=L, order=2 + i % 2, nk=nk, maxk=nk * 0.01, n=side ** 3))
    return out


def _survey_inputs(c, seed):
    """Data: displaced random points in a ball around the observer; randoms: uniform in the same ball. Every
    column is float32, as the survey reader keeps them."""
    g, dev, R = _gen(seed), _device(), 0.475 * c["L"]
    nd, nr = c["ndata"], c["ndata"] * c["ratio"]
    m = 128
    psi = _displacement(m, c["L"], 3.0 * c["L"] / c["n"], g)

    def ball(n):
        u = torch.randn(3, n, generator=g, device=dev, dtype=torch.float64)
        r = 0.97 * R * torch.rand(n, generator=g, device=dev, dtype=torch.float64) ** (1.0 / 3.0)
        return u * (r / u.norm(dim=0))

    d = ball(nd)
    q = ((d / c["L"] + 0.5) * m).long().clamp_(0, m - 1)
    idx = (q[0] * m + q[1]) * m + q[2]
    d = torch.stack([d[a] + psi[a].reshape(-1)[idx].double().clamp_(-0.01 * R, 0.01 * R) for a in range(3)])
    cats = []
    for p in (d, ball(nr)):
        rad = p.norm(dim=0)
        nbar = (nd / (4.0 / 3.0 * math.pi * R ** 3)) * (1.5 - rad / R)  # falls with distance, as a flux limit does
        cats.append({"x": p[0].float().contiguous(), "y": p[1].float().contiguous(), "z": p[2].float().contiguous(),
                     "w": torch.ones(p.shape[1], device=dev), "nbar": nbar.float().contiguous()})
    return cats


def _survey_params(c):
    h = c["L"] / 2
    return (cg.Params(NX=c["n"], NY=c["n"], NZ=c["n"], XMIN=-h, XMAX=h, YMIN=-h, YMAX=h, ZMIN=-h, ZMAX=h, InterpOrder=c["order"],
                      DoInterlacing=c["interlace"], NK=c["nk"], NMU=1, Mink=0.0, Maxk=c["maxk"], Omega_m=OMEGA_M, Redshift=REDSHIFT,
                      LOS=0, Momentum=0, Odd_Multipoles=c["odd"]),
            cg.SurveyParams(X_Origin=0.0, Y_Origin=0.0, Z_Origin=0.0, FKP_Column=-1, FKP_Pk=1e4, NBAR_Column=5))


def prepare(case, seed):
    if case["kind"] == "batch":
        mocks = []
        for i, c in enumerate(_mock_cases(case)):
            x, y, z, v, _ = _box_inputs(c, seed * 1000 + i)
            mocks.append((_params(c), (x, y, z, v, None)))
        return {"kind": "batch", "mocks": mocks}
    if case["kind"] == "survey":
        data, rand = _survey_inputs(case, seed)
        p, sv = _survey_params(case)
        return {"kind": "survey", "ctx": cg.SurveySpectrum(p, sv, precision=case["precision"]), "data": data, "rand": rand}
    parts = _box_inputs(case, seed)
    if case["host"]:  # page-locked host arrays
        parts = [None if t is None else t.cpu().pin_memory() for t in parts]
    spectra = [s for s in case["spectra"].split(",") if s] or None
    st = {"kind": case["kind"], "parts": parts, "single": case["precision"] != "fp64",
          "ctx": cg.PowerSpectrum(_params(case), precision=case["precision"], spectra=spectra)}
    if case["kind"] == "gradient":
        st["dL"] = _loss_gradient(case)
        st["grads"] = {k: torch.empty_like(parts[0]) for k in ("dx", "dy", "dz", "dvlos", "dw")}
    return st


# ---------------------------------------------------------------------------------------------- run
def _result(r, single):
    dt = np.float32 if single else np.float64
    out = {"Pk": np.stack([r["Pk%d" % l] for l in range(5)]).astype(dt), "Nmodes": r["Nmodes"],
           "scalars": np.array([r["shot"], r["norm"], r["alpha"]], dtype=dt)}
    if "Pk_2D" in r:
        out["Pk_2D"], out["Nmodes_2D"] = r["Pk_2D"].astype(dt), r["Nmodes_2D"]
    return out


def run(state):
    if state["kind"] == "batch":
        return [_result(res[0], True) for status, res in cg.run_batch(state["mocks"], precision="fp32")]
    if state["kind"] == "survey":
        return _result(state["ctx"].power(state["data"], state["rand"]), True)
    ctx = state["ctx"]
    ctx.paint(*state["parts"])
    out = [_result(r, state["single"]) for r in ctx.power()]
    if state["kind"] == "gradient":
        out.append(dict(ctx.backward(state["dL"], out=state["grads"])))
    return out


# --------------------------------------------------------------------------------------------- work
def _spectra_of(c):
    """Fields' exponents of v, mean subtraction of A, and per spectrum (product, shot moment); products: 0 |A|^2,
    1 Re A*B, 2 Im A*B, 3 |B|^2."""
    names = [s for s in c["spectra"].split(",") if s]
    if not names:
        nf, ea, eb, im, mean, mom = FIELDS[c["momentum"]]
        return ([ea, eb][:nf], mean, [((2 if im else 1) if nf == 2 else 0, mom)])
    need_d, need_p = "dd" in names or "dp" in names, "dp" in names or "pp" in names
    exps = ([0] if need_d else []) + ([1] if need_p else [])
    two = len(exps) == 2
    return exps, int(need_d), [{"dd": (0, 0), "dp": (2, 1), "pp": (3 if two else 0, 2)}[s] for s in names]


def work(case):
    if case["kind"] == "batch":
        w = [work(c) for c in _mock_cases(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if case["kind"] == "survey":
        n, g = case["n"], 1 + case["interlace"]
        cells, modes, objs = n ** 3, n * n * (n // 2 + 1), case["ndata"] * (1 + case["ratio"])
        sets = 25 if case["odd"] else 15
        # catalogues in; painted grids written once; per set the grids read, and their half transform written and read
        return {"bytes": objs * 20 + g * 4 * cells + sets * g * (4 * cells + 16 * modes),
                "flops": 2 * case["order"] ** 3 * g * objs + sets * (g * 2.5 * cells * math.log2(cells) + 30 * modes)}
    exps, _, spec = _spectra_of(case)
    g = len(exps) * (1 + case["interlace"])
    cells, modes = case["nx"] * case["ny"] * case["nz"], case["nx"] * case["ny"] * (case["nz"] // 2 + 1)
    eb, pb = (8 if case["precision"] == "fp64" else 4), (8 if case["dtype"] == "f64" else 4)
    cols = 3 + int(case["los"] != 0 or max(exps) > 0) + int(case["weights"])
    # particles in, each grid written by the paint, read and written by the transform and read by the binning
    b = case["n"] * cols * pb + g * (2 * cells * eb + 4 * modes * eb) + len(spec) * 6 * 8 * case["nk"]
    f = 2 * case["order"] ** 3 * g * case["n"] + g * 2.5 * cells * math.log2(cells) + 40 * modes
    if case["kind"] == "gradient":  # the transposed chain: modes, inverse transform, readout; five columns out
        b += case["n"] * (cols + 5) * pb + g * (2 * cells * eb + 4 * modes * eb)
        f += 8 * case["order"] ** 3 * g * case["n"] + g * 5 * cells * math.log2(cells) + 40 * modes
    return {"bytes": b, "flops": f}


# -------------------------------------------------------------------------------------------- exact
def _axis(order, is_x, n, los, c, mn, mx, length):
    """One axis of the mass assignment in 64 bits: accepted, and per tap (index, weight, d weight / d scale, kept)."""
    d = length / n
    if order == 3 and is_x and los == 0:
        c = torch.where(c - mn < d, c + length, c)
    if order == 3 and is_x:
        acc = (c >= (mn + d if los == 0 else mn)) & (c < mx + d)
    else:
        acc = (c >= mn) & (c < mx)
    s = (c - mn) / d
    if order == 1:
        i = s.long()
        taps = [(i, torch.ones_like(s), torch.zeros_like(s), acc)]
    elif order == 2:
        i = s.long()
        f = s - i
        hi = i + 1
        if not is_x and los == 0:
            hi = torch.where(hi == n, torch.zeros_like(hi), hi)
        one = torch.ones_like(s)
        taps = [(i, 1.0 - f, -one, acc), (hi, f, one, acc)]
    else:
        i = (s + 0.5).long()
        f = s - i
        lo, hi, mid = i - 1, i + 1, i
        if not is_x and los == 0:  # wrapping axis
            lo = torch.where(lo < 0, lo + n, lo)
            over = hi >= n
            hi = torch.where(over, hi - n, hi)
            mid = torch.where(over & (i >= n), torch.zeros_like(i), i)
            hi = torch.where(over & (hi > 1), torch.ones_like(hi), hi)
        taps = [(mid, 0.75 - f * f, -2.0 * f, acc), (lo, 0.5 * (0.5 - f) ** 2, -(0.5 - f), acc & (lo > 0)),
                (hi, 0.5 * (0.5 + f) ** 2, 0.5 + f, acc)]
    out = []
    for idx, w, dw, on in taps:
        if is_x and los == 0:  # the halo slices fold onto the first ones
            idx = torch.where(idx >= n, idx - n, idx)
        on = on & (idx >= 0) & (idx < n)
        out.append((idx.clamp(0, n - 1), w, dw, on))
    return acc, out


def _chunks(n, size=1 << 22):
    return [(a, min(n, a + size)) for a in range(0, n, size)]


class _Exact:
    """The periodic estimator in 64 bits for one case's particles."""

    def __init__(self, c, parts):
        self.c = c
        self.L, self.N = (c["lx"], c["ly"], c["lz"]), (c["nx"], c["ny"], c["nz"])
        self.exps, self.mean, self.spec = _spectra_of(c)
        self.parts = parts
        self.rsd = (1.0 + REDSHIFT) / (100.0 * math.sqrt(OMEGA_M * (1.0 + REDSHIFT) ** 3 + 1.0 - OMEGA_M))
        self.dev = parts[0].device

    def columns(self, a, b):
        pos = [t[a:b].double() for t in self.parts[:3]]
        v = self.parts[3][a:b].double()
        w = self.parts[4][a:b].double() if self.parts[4] is not None else torch.ones_like(v)
        if self.c["los"]:
            pos[self.c["los"] - 1] = pos[self.c["los"] - 1] + v * self.rsd
        return pos, v, w

    def stencil(self, pos, st):
        accs, taps = [], []
        for k in range(3):
            acc, t = _axis(self.c["order"], k == 0, self.N[k], self.c["los"], pos[k] + (0.5 * self.L[k] / self.N[k] if st else 0.0),
                           0.0, self.L[k], self.L[k])
            accs.append(acc)
            taps.append(t)
        return accs[0] & accs[1] & accs[2], taps

    def paint(self):
        nx, ny, nz = self.N
        ns = 1 + self.c["interlace"]
        grids = [torch.zeros(nx * ny * nz, dtype=torch.float64, device=self.dev) for _ in range(ns * len(self.exps))]
        self.ngrid, self.wsum, mom = 0.0, 0.0, [0.0] * 4
        for a, b in _chunks(len(self.parts[0])):
            pos, v, w = self.columns(a, b)
            self.wsum += float(w.sum())
            for m in range(4):
                mom[m] += float((w * v ** (m + 1)).sum())
            for st in range(ns):
                acc, (tx, ty, tz) = self.stencil(pos, st)
                if st == 0:
                    self.ngrid += float((w * acc).sum())
                vals = [w * v ** e * acc for e in self.exps]
                for ix, wx, _, ox in tx:
                    for iy, wy, _, oy in ty:
                        for iz, wz, _, oz in tz:
                            idx = (ix * ny + iy) * nz + iz
                            wt = wx * wy * wz * (ox & oy & oz)
                            for f, val in enumerate(vals):
                                grids[st * len(self.exps) + f].index_add_(0, idx, val * wt)
        self.moment = [1.0] + [m / self.wsum for m in mom]
        return grids

    def slabs(self):
        """Per run of kx planes: bin, multiplicity x deconvolution, mu, interlace phase of every half-space mode."""
        c, dev = self.c, self.dev
        nx, ny, nz = self.N
        axes = []
        for n, L, half in ((nx, self.L[0], False), (ny, self.L[1], False), (nz, self.L[2], True)):
            d = L / n
            sc = 1.0 / (n * d)
            i = torch.arange(n // 2 + 1 if half else n, device=dev, dtype=torch.float64)
            f = (i if half else torch.where(i <= n // 2, i, i - n)) * sc
            arg = math.pi * f * d
            sinc = torch.where(f != 0, torch.sin(arg) / torch.where(f != 0, arg, torch.ones_like(arg)), torch.ones_like(arg))
            axes.append((f, sinc ** (-2 * c["order"]), torch.polar(torch.ones_like(arg), arg)))
        (fx, cx, ex), (fy, cy, ey), (fz, cz, ez) = axes
        bw = (c["maxk"] - c["mink"]) / c["nk"]
        nyq = min(math.pi * n / L for n, L in zip(self.N, self.L))
        j = torch.arange(ny, device=dev)[None, :, None]
        k = torch.arange(nz // 2 + 1, device=dev)[None, None, :]
        step = max(1, (1 << 24) // (ny * (nz // 2 + 1)))
        for a in range(0, nx, step):
            b = min(nx, a + step)
            s = (fx[a:b, None, None] ** 2 + fy[None, :, None] ** 2) + fz[None, None, :] ** 2
            kt = 2.0 * math.pi * torch.sqrt(s)
            v = ((torch.log10(kt) if c["log"] else kt) - c["mink"]).float().double() / bw
            ok = (v > -1.0) & (v < c["nk"]) & (kt <= nyq)
            kb = torch.where(ok, v, torch.zeros_like(v)).long()  # towards zero, as a cast does
            i = torch.arange(a, b, device=dev)[:, None, None]
            nm = torch.where(k != 0, 2, torch.where(i == nx // 2, 2, torch.where((j == 0) & (i == 0), 2, 1))).double()
            gc = cx[a:b, None, None] * cy[None, :, None] * cz[None, None, :]
            e = ex[a:b, None, None] * ey[None, :, None] * ez[None, None, :] if c["interlace"] else None
            fl = fx[a:b, None, None] if c["los"] == 1 else (fy[None, :, None] if c["los"] == 2 else fz[None, None, :])
            mu = torch.where(s > 0, fl / torch.sqrt(torch.where(s > 0, s, torch.ones_like(s))), torch.zeros_like(s))
            yield a, b, ok, kb, nm, gc * nm * (0.25 if c["interlace"] else 1.0), mu, e

    def fields(self, grids):
        F = []
        for s, g in enumerate(grids):
            f = torch.fft.rfftn(g.view(self.N))
            if s % len(self.exps) == 0 and self.mean:
                f[0, 0, 0] -= self.ngrid
            F.append(f)
        return F

    @staticmethod
    def legendre(mu, l):
        m2 = mu * mu
        return {0: torch.ones_like(mu), 1: mu, 2: 1.5 * m2 - 0.5, 3: (2.5 * m2 - 1.5) * mu, 4: (4.375 * m2 - 3.75) * m2 + 0.375}[l]

    def spectra(self, F):
        c, nf = self.c, len(self.exps)
        ls = range(5) if c["odd"] else (0, 2, 4)
        nk, nmu, copies = c["nk"], c["nmu"], 2048
        pk = [torch.zeros(5, nk, dtype=torch.float64, device=self.dev) for _ in self.spec]
        p2 = [torch.zeros(nk * nmu, dtype=torch.float64, device=self.dev) for _ in self.spec]

        def binned(idx, val, n):
            t = torch.zeros(n * copies, dtype=torch.float64, device=self.dev)
            t.index_add_(0, idx * copies + torch.arange(idx.numel(), device=self.dev) % copies, val)
            return t.view(n, copies).sum(1)

        self.nmodes = torch.zeros(nk, dtype=torch.float64, device=self.dev)
        self.nmodes2 = torch.zeros(nk * nmu, dtype=torch.float64, device=self.dev)
        for a, b, ok, kb, nm, gc, mu, e in self.slabs():
            A, B = F[0][a:b], F[1][a:b] if nf == 2 else None
            if e is not None:
                A = A + F[nf][a:b] * e
                B = B + F[nf + 1][a:b] * e if nf == 2 else None
            idx, mu, gc, nm, A = kb[ok], mu[ok], gc[ok], nm[ok], A[ok]
            B = B[ok] if nf == 2 else None
            mb = ((mu + 1.0) / 2.0 * nmu).long().clamp_(max=nmu - 1)
            self.nmodes += binned(idx, nm, nk)
            if c["out2d"]:
                self.nmodes2 += binned(idx * nmu + mb, nm, nk * nmu)
            for q, (prod, _) in enumerate(self.spec):
                t = {0: lambda: A.abs() ** 2, 1: lambda: (A.conj() * B).real, 2: lambda: (A.conj() * B).imag,
                     3: lambda: B.abs() ** 2}[prod]() * gc
                for l in ls:
                    pk[q][l] += binned(idx, t * self.legendre(mu, l), nk)
                if c["out2d"]:
                    p2[q] += binned(idx * nmu + mb, t, nk * nmu)
        N, V = self.ngrid, self.L[0] * self.L[1] * self.L[2]
        out = []
        for q, (_, m) in enumerate(self.spec):
            r = {"Pk": pk[q], "Nmodes": None,
                 "scalars": torch.tensor([N * self.moment[m], N * N / V, N / (self.N[0] * self.N[1] * self.N[2])], dtype=torch.float64)}
            if c["out2d"]:
                r["Pk_2D"], r["Nmodes_2D"] = p2[q], None
            out.append(r)
        return out

    def gradient(self, F, raw, dL):
        """dL/d(x, y, z, v, w) of sum_l sum_b dL/dP_l(b) P_l(b) for a density spectrum: P_l = (2l + 1) S_l / (Nmodes
        norm), P_0 less its shot noise, the last filled bin held at 0."""
        c = self.c
        N, V = self.ngrid, self.L[0] * self.L[1] * self.L[2]
        norm = N * N / V
        filled = self.nmodes > 0
        last = int(filled.nonzero().max())
        use = filled.clone()
        use[last] = False
        nm = torch.where(filled, self.nmodes, torch.ones_like(self.nmodes))
        coef, dLdN = {}, 0.0
        for l in (0, 2):
            g = torch.as_tensor(dL["Pk%d" % l], device=self.dev) * use
            coef[l] = g * (2 * l + 1) / (nm * norm)
            S = raw["Pk"][l]
            P = (2 * l + 1) * S / (nm * norm) - (N / norm if l == 0 else 0.0)
            dLdN += float((g * (-2.0 * P / N - (1.0 / norm if l == 0 else 0.0))).sum())
        nx, ny, nz = self.N
        G = [torch.zeros_like(f) for f in F]
        for a, b, ok, kb, _, gc, mu, e in self.slabs():
            A = F[0][a:b] if e is None else F[0][a:b] + F[1][a:b] * e
            t = sum(coef[l][kb] * self.legendre(mu, l) for l in (0, 2)) * gc * ok * 2.0
            G[0][a:b] = t * A
            if e is not None:
                G[1][a:b] = t * A * e.conj()
        dLdN -= sum(float(g[0, 0, 0].real) for g in G)
        back = []
        for g in G:  # dL/dcell = Re sum over the half space of Gamma e^{ikx}
            half = torch.nn.functional.pad(torch.view_as_real(g), (0, 0, 0, nz - nz // 2 - 1))
            back.append(torch.fft.ifftn(torch.view_as_complex(half.contiguous()), norm="forward").real.reshape(-1).contiguous())
        n = len(self.parts[0])
        out = {k: torch.zeros(n, dtype=torch.float64, device=self.dev) for k in ("dx", "dy", "dz", "dvlos", "dw")}
        for a, b in _chunks(n):
            pos, v, w = self.columns(a, b)
            for st in range(1 + c["interlace"]):
                acc, (tx, ty, tz) = self.stencil(pos, st)
                if st == 0:
                    out["dw"][a:b] += acc * dLdN
                for ix, wx, dx, ox in tx:
                    for iy, wy, dy, oy in ty:
                        for iz, wz, dz, oz in tz:
                            g = back[st][(ix * ny + iy) * nz + iz] * (acc & ox & oy & oz)
                            out["dw"][a:b] += g * wx * wy * wz
                            out["dx"][a:b] += g * w * dx * wy * wz * (nx / self.L[0])
                            out["dy"][a:b] += g * w * wx * dy * wz * (ny / self.L[1])
                            out["dz"][a:b] += g * w * wx * wy * dz * (nz / self.L[2])
        if c["los"]:
            out["dvlos"] += self.rsd * out[("dx", "dy", "dz")[c["los"] - 1]]
        return out


def _exact_box(c, parts):
    ex = _Exact(c, parts)
    F = ex.fields(ex.paint())
    out = ex.spectra(F)
    if c["kind"] == "gradient":
        out.append(ex.gradient(F, out[0], _loss_gradient(c)))
    return out


def _products(l):
    """Exponents and multinomial coefficients of (kx x + ky y + kz z)^l."""
    return [(a, b, l - a - b, math.factorial(l) // (math.factorial(a) * math.factorial(b) * math.factorial(l - a - b)))
            for a in range(l + 1) for b in range(l + 1 - a)]


def _exact_survey(c, seed):
    data, rand = _survey_inputs(c, seed)
    dev, n, h = data["x"].device, c["n"], c["L"] / 2
    box = _box("", nx=n, ny=n, nz=n, lx=c["L"], ly=c["L"], lz=c["L"], order=c["order"], interlace=c["interlace"], los=0, odd=c["odd"],
               nk=c["nk"], maxk=c["maxk"], n=0)

    class Cat(_Exact):
        def columns(self, a, b):
            return [t[a:b].double() + h for t in self.parts[:3]], self.parts[3][a:b].double() * 0.0, self.parts[4][a:b].double()

    wd, wr = [(t["w"].double() / (1.0 + t["nbar"].double() * 1e4)).float() for t in (data, rand)]
    alpha = float(wd.double().sum() / wr.double().sum())
    grids = None
    for cat, w, pref in ((data, wd, 1.0), (rand, wr, -alpha)):  # the catalogues lie well inside the box: no edge rules
        ex = Cat(box, [cat["x"], cat["y"], cat["z"], w, w.double() * pref])
        g = ex.paint()
        grids = g if grids is None else [u.add_(v) for u, v in zip(grids, g)]
    ex.ngrid, ex.mean = 0.0, 0
    shot = float((wd.double() ** 2).sum() + (wr.double() ** 2).sum() * alpha ** 2)
    norm = float((wr.double() ** 2 * rand["nbar"].double()).sum() * alpha)
    u = torch.arange(n, device=dev, dtype=torch.float64) * (c["L"] / n) - h
    r2 = u[:, None, None] ** 2 + u[None, :, None] ** 2 + u[None, None, :] ** 2
    r2 = torch.where(r2 == 0, torch.ones_like(r2), r2)
    kf = torch.fft.fftfreq(n, d=1.0 / n, device=dev, dtype=torch.float64)
    kf = torch.where(torch.arange(n, device=dev) == n // 2, kf.abs(), kf)
    kz = torch.arange(n // 2 + 1, device=dev, dtype=torch.float64)
    F0 = None
    pk = torch.zeros(5, c["nk"], dtype=torch.float64, device=dev)
    copies = 2048
    raw = {}
    for l in range(5):
        if l % 2 and not c["odd"]:
            continue
        tot = None
        for a, b, d, m in _products(l):
            acc = None
            F = [torch.fft.rfftn(g.view(n, n, n) * (u[:, None, None] ** a * u[None, :, None] ** b * u[None, None, :] ** d * r2 ** (-0.5 * l)))
                 for g in grids]
            for s0, s1, ok, kb, _, gc, mu, e in ex.slabs():
                X = F[0][s0:s1] if e is None else F[0][s0:s1] + F[1][s0:s1] * e
                k2 = kf[s0:s1, None, None] ** 2 + kf[None, :, None] ** 2 + kz[None, None, :] ** 2
                k2 = torch.where(k2 == 0, torch.ones_like(k2), k2)
                X = X * (m * kf[s0:s1, None, None] ** a * kf[None, :, None] ** b * kz[None, None, :] ** d * k2 ** (-0.5 * l))
                if acc is None:
                    acc = torch.empty(n, n, n // 2 + 1, dtype=torch.complex128, device=dev)
                acc[s0:s1] = X
            tot = acc if tot is None else tot.add_(acc)
            del F, acc
        if l == 0:
            F0 = tot
        out = torch.zeros(c["nk"] * copies, dtype=torch.float64, device=dev)
        for s0, s1, ok, kb, _, gc, mu, e in ex.slabs():
            X = tot[s0:s1] * F0[s0:s1].conj()
            val = (X.real if l % 2 == 0 else -X.imag) * gc  # odd l: the imaginary part of conj(F_l) F_0
            idx = kb[ok]
            out.index_add_(0, idx * copies + torch.arange(idx.numel(), device=dev) % copies, val[ok])
        raw[l] = out.view(c["nk"], copies).sum(1)
        del tot
    pk[0] = raw[0]
    pk[2] = 1.5 * raw[2] - 0.5 * raw[0]
    pk[4] = (35.0 * raw[4] - 30.0 * raw[2] + 3.0 * raw[0]) / 8.0
    if c["odd"]:
        pk[1] = raw[1]
        pk[3] = 2.5 * raw[3] - 1.5 * raw[1]
    return {"Pk": pk, "Nmodes": None, "scalars": torch.tensor([shot, norm, alpha], dtype=torch.float64)}


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_box(c, _box_inputs(c, seed * 1000 + i))[0] for i, c in enumerate(_mock_cases(case))]
    if case["kind"] == "survey":
        return _exact_survey(case, seed)
    return _exact_box(case, _box_inputs(case, seed))
