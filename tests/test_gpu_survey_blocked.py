"""The FP32 survey estimator for power-of-two NX (32 to 1024), NY and NZ (weighted z pass, k_yfft, k_xrow_survey) against
the oracle at the suite's tolerances: every row length, one, two and four slots, every (l, m), the observer off the grid
and on a cell corner inside it, top edges below and beyond the Nyquist frequency, linear and logarithmic bins."""
import pytest

import oracle as orc
from test_gpu_survey import _catalogues, _gpu, _write_params, assert_survey

pytestmark = pytest.mark.gpu

# (NX, NY, NZ), Momentum, order, interlacing, odd multipoles, observer on a corner, bins
CASES = [((64, 16, 32), 0, 3, 1, 1, 0, dict(NK=20, Maxk=1.2)), ((64, 64, 32), 2, 2, 1, 1, 1, dict(NK=16, Maxk=0.48)),
         ((128, 32, 64), 3, 3, 0, 1, 0, dict(NK=30, Maxk=0.8)), ((128, 16, 32), 1, 2, 1, 1, 0, dict(NK=500, Maxk=0.8)),
         ((256, 32, 32), 0, 1, 0, 1, 1, dict(NK=12, OutputLog=1, Mink=-1.6, Maxk=-0.2)),
         ((256, 16, 64), 2, 3, 1, 0, 0, dict(NK=10, Maxk=0.32)), ((512, 16, 32), 0, 3, 1, 1, 1, dict(NK=20, Maxk=0.6)),
         ((512, 32, 32), 3, 2, 1, 1, 0, dict(NK=16, Maxk=1.2)), ((1024, 32, 32), 0, 2, 1, 1, 0, dict(NK=9, Maxk=0.12)),
         ((1024, 16, 32), 2, 1, 1, 0, 1, dict(NK=24, Maxk=0.8)), ((64, 256, 32), 1, 3, 0, 0, 1, dict(NK=1, Maxk=0.2)),
         ((32, 32, 32), 0, 2, 1, 1, 1, dict(NK=16, Maxk=0.5)), ((32, 64, 64), 2, 3, 0, 1, 0, dict(NK=11, Maxk=0.4))]


@pytest.mark.parametrize("shape,momentum,order,il,odd,corner,bins", CASES)
def test_survey_blocked_path_matches_oracle(gpu, tmp_path, shape, momentum, order, il, odd, corner, bins):
    half = [2.5 * n for n in shape]  # cells of 5
    off = [0.0, 0.0, 0.0] if corner else [1.5 * half[0] + 100.0, 50.0, -30.0]
    p, prm, sv = _write_params(tmp_path, NX=shape[0], NY=shape[1], NZ=shape[2], XMIN=off[0] - half[0], XMAX=off[0] + half[0],
                               YMIN=off[1] - half[1], YMAX=off[1] + half[1], ZMIN=off[2] - half[2], ZMAX=off[2] + half[2],
                               InterpOrder=order, DoInterlacing=il, Odd_Multipoles=odd, Periodic=0, X_Origin=0.0,
                               Y_Origin=0.0, Z_Origin=0.0, REDMININ=0.0, REDMAXIN=50.0, NOBJ_Max=100000, NBAR_Column=5,
                               FKP_Column=-1, FKP_Pk=4000.0, FKP_Pk_mom=5e9, FKP_Pk_cross=5e5, Momentum=momentum, **bins)
    df, rf = _catalogues(tmp_path, p, 4000, 25000, seed=sum(shape) + momentum)
    if corner:  # a heavy object next to the observer, so that its cell carries weight
        with open(df, "a") as f:
            f.write("1.0 2.0 -1.5 40 0.0002 0 0.5 0.07 0 0 0 0\n")
    r = orc.survey_run(p, df, rf)
    res, _ = _gpu(prm, sv, df, rf, "fp32")
    assert_survey(res, r["raw"], p, "fp32", label=f"{shape} Momentum {momentum} il={il} odd={odd} corner={corner} {bins}")
