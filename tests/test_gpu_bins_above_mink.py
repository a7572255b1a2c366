"""Linear bins that begin above k = 0: columns whose first modes lie below the first edge (and, by the reference's truncation
towards zero, in bin 0 within one bin width of it), in the mode counts, the FP32 blocked pass, the FP64 bin kernel and the
survey's pass; and a blocked context whose planes run in chunks of unequal length."""
import numpy as np
import pytest

import capow_gb300 as cg
from parity_util import TOL, assert_spectrum, gpu_run, oracle_run, params_pair, particles

pytestmark = pytest.mark.gpu

BOX = dict(XMIN=-3.0, XMAX=997.0, YMIN=0.0, YMAX=1000.0, ZMIN=10.0, ZMAX=510.0, NMU=5)


@pytest.mark.parametrize("precision", ["fp32", "det", "fp64"])
@pytest.mark.parametrize("shape,los,odd,bins", [((64, 64, 64), 3, 1, dict(NK=7, Mink=0.08, Maxk=0.19)),
                                                ((128, 64, 32), 1, 0, dict(NK=24, Mink=0.05, Maxk=0.2)),
                                                ((32, 32, 64), 2, 1, dict(NK=3, Mink=0.06, Maxk=0.5)),
                                                ((60, 50, 42), 0, 0, dict(NK=9, Mink=0.07, Maxk=0.14))])
def test_periodic_bins(gpu, precision, shape, los, odd, bins):
    po, pc = params_pair(NX=shape[0], NY=shape[1], NZ=shape[2], InterpOrder=3, LOS=los, DoInterlacing=1, Momentum=0,
                         Odd_Multipoles=odd, **BOX, **bins)
    parts = particles(po, 6000, seed=sum(shape))
    raw = oracle_run(po, parts, 0)["raw"]
    res, _, _, _ = gpu_run(pc, parts, precision)
    assert_spectrum(res[0], raw, np.abs(raw["Pk0"]), precision, odd=bool(odd), label=f"{precision} {shape} {bins}")


@pytest.mark.parametrize("n,odd,bins", [(64, 1, dict(NK=9, Mink=0.06, Maxk=0.17)), (128, 0, dict(NK=5, Mink=0.15, Maxk=0.3))])
def test_survey_bins(gpu, n, odd, bins):
    import torch

    g = torch.Generator(device=gpu)
    g.manual_seed(n)
    cats = []
    for m in (20000, 90000):
        x = torch.rand(3, m, generator=g, device=gpu) * 900.0 - 450.0
        ones = torch.ones(m, device=gpu)
        cats.append(dict(x=x[0].contiguous(), y=x[1].contiguous(), z=x[2].contiguous(), w=ones, nbar=1e-4 * ones))
    p = cg.Params(NX=n, NY=n, NZ=n, XMIN=-500.0, XMAX=500.0, YMIN=-500.0, YMAX=500.0, ZMIN=-500.0, ZMAX=500.0, InterpOrder=3,
                  DoInterlacing=1, LOS=0, Odd_Multipoles=odd, **bins)
    sv = cg.SurveyParams(X_Origin=0.25, Y_Origin=0.5, Z_Origin=0.125, FKP_Column=-1, FKP_Pk=1e4, NBAR_Column=5)
    res = {}
    for precision in ("fp32", "fp64"):
        with cg.SurveySpectrum(p, sv, precision=precision) as ss:
            res[precision] = ss.power(*cats)
    a, b = res["fp32"], res["fp64"]
    assert np.array_equal(a["Nmodes"], b["Nmodes"]) and (b["Nmodes"] > 0).all()
    t0, t2 = TOL["fp32"]
    assert (np.abs(a["Pk0"] - b["Pk0"]) <= t0 * np.abs(b["Pk0"])).all()
    for l in (1, 2, 3, 4):
        if odd or l % 2 == 0:
            assert ((2 * l + 1) * np.abs(a[f"Pk{l}"] - b[f"Pk{l}"]) <= t2 * np.abs(b["Pk0"])).all(), l


def test_planes_in_unequal_chunks(gpu):
    """Four slots of 256 x 1024 x 1024: 16.8 MB a plane, so the z and y passes take 192 planes, then 64."""
    _, pc = params_pair(NX=256, NY=1024, NZ=1024, InterpOrder=2, LOS=3, DoInterlacing=1, Momentum=1, NK=32, Maxk=0.7, **BOX)
    parts = particles(pc, 300000, seed=78)
    res, st, _, _ = gpu_run(pc, parts, "fp32", spectra=["dd", "dp", "pp"])
    res3, st3, _, _ = gpu_run(pc, parts, "fp32", spectra=["dd", "dp", "pp"], fft_path="3d")
    assert st["ngrid"] == st3["ngrid"]
    dd, pp = (np.abs(res3[k]["Pk0"]) for k in (0, 2))
    for a, b, n0 in zip(res, res3, (dd, np.sqrt(dd * pp), pp)):
        assert_spectrum(a, b, n0, "fp32", odd=False, label=a["kind"])
