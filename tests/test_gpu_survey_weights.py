"""The float catalogue's FKP weights, their sums and the painted counters of Momentum 0 against the same numbers formed
with numpy: weights rounded from the double expression (one wrong rounding in a sum of 300,000 weights is 2e-13 of it, in
one of 31 weights 2e-9), products in float, sums in double (1e-14: additions in another order)."""
import math

import numpy as np
import pytest

import capow_gb300 as cg
from test_gpu_survey import _write_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pk", [0.0, 1e-3, 4000.0, 123456.789, 3e9])
@pytest.mark.parametrize("n", [1, 31, 300001])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_survey_float_weights(gpu, tmp_path, n, pk, precision):
    p, prm, sv = _write_params(tmp_path, NX=16, NY=16, NZ=32, XMIN=0.0, XMAX=800.0, YMIN=0.0, YMAX=800.0, ZMIN=0.0,
                               ZMAX=800.0, InterpOrder=3, DoInterlacing=1, NK=8, Maxk=0.1, Periodic=0, X_Origin=-10.0,
                               REDMININ=0.0, REDMAXIN=5.0, NOBJ_Max=1000000, NBAR_Column=5, FKP_Column=-1, FKP_Pk=pk)
    rng = np.random.default_rng(n)

    def cat(m):
        c = {k: rng.uniform(-10.0, 830.0, m).astype(np.float32) for k in ("x", "y", "z")}  # some outside the box
        c["w"] = rng.uniform(0.25, 3.0, m).astype(np.float32)
        c["nbar"] = (10.0 ** rng.uniform(-7, -2, m)).astype(np.float32)
        return c

    data, rand = cat(n), cat(2 * n + 3)
    with cg.SurveySpectrum(prm, sv, precision=precision) as ss:
        st = ss.power(data, rand)["stats"]
    alpha = st["data_nbw"] / st["rand_nbw"]  # the randoms' w^2 and w^2 nbar sums are reported times alpha^2 and alpha
    for tag, c in (("data", data), ("rand", rand)):
        nb = c["nbar"]
        w = (c["w"].astype(np.float64) * (1.0 / (1.0 + nb.astype(np.float64) * pk))).astype(np.float32)
        ww = w * w
        for key, v, e in (("nbw", w, 0), ("nbwsq", ww, 2), ("nbsqwsq", ww * nb, 1)):
            s = math.fsum(v.astype(np.float64)) * (alpha ** e if tag == "rand" else 1.0)
            assert abs(st[f"{tag}_{key}"] - s) <= 1e-14 * s, (tag, key)
    for tag, c in (("ngrid_data", data), ("ngrid_rand", rand)):
        top = (850.0, 800.0, 800.0)  # the TSC x axis accepts one cell beyond the box
        count = np.logical_and.reduce([(c[k] >= 0.0) & (c[k] < t) for k, t in zip("xyz", top)]).sum()
        assert abs(st[tag] - count) <= 1e-13 * count, tag


@pytest.mark.parametrize("il", [0, 1])
def test_survey_many_objects_on_many_tiles(gpu, tmp_path, il):
    """More than a million objects on a grid of more than 4096 tiles: the FP32 paint takes them ordered by blocks of the
    box. Grids cell by cell against the FP64 context's (5e-5 of the largest cell, the FP32 survey paint's bound), the
    counters and sums to 1e-12; some objects lie outside the box on either side."""
    p, prm, sv = _write_params(tmp_path, NX=264, NY=256, NZ=512, XMIN=0.0, XMAX=800.0, YMIN=-100.0, YMAX=700.0, ZMIN=0.0,
                               ZMAX=1600.0, InterpOrder=2, DoInterlacing=il, NK=8, Maxk=0.1, Periodic=0, X_Origin=-10.0,
                               REDMININ=0.0, REDMAXIN=5.0, NOBJ_Max=3000000, NBAR_Column=5, FKP_Column=-1, FKP_Pk=4000.0)
    rng = np.random.default_rng(8)

    def cat(m):
        c = {"x": rng.uniform(-30.0, 830.0, m), "y": rng.uniform(-130.0, 730.0, m), "z": rng.uniform(-9.0, 1610.0, m)}
        c["w"], c["nbar"] = rng.uniform(0.25, 3.0, m), 10.0 ** rng.uniform(-5, -3, m)
        return {k: v.astype(np.float32) for k, v in c.items()}

    data, rand = cat(50001), cat((1 << 20) + 5)
    out = {}
    for precision in ("fp64", "fp32"):
        with cg.SurveySpectrum(prm, sv, precision=precision) as ss:
            st = ss.power(data, rand)["stats"]
            out[precision] = (st, [ss.grid(k).reshape(264, 256, -1)[:, :, :512] for k in range(1 + il)])
    for k, v in out["fp64"][0].items():
        assert abs(out["fp32"][0][k] - v) <= 1e-12 * abs(v), k
    for a, b in zip(out["fp32"][1], out["fp64"][1]):
        assert np.abs(a - b).max() <= 5e-5 * np.abs(b).max()
