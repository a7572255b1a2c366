"""k_bin64 (up to four mirror modes at a time) and k_paint64 (shared products away from the edges) against the oracle at
the suite's FP64 tolerance: odd and even axes, axes of one to four cells, the three interpolation orders, every line of
sight, one and two fields, odd multipoles, linear and logarithmic bins."""
import numpy as np
import pytest

from parity_util import assert_spectrum, gpu_run, grid_close, oracle_run, params_pair, particles

pytestmark = pytest.mark.gpu

CASES = [((9, 7, 5), 2, 1, 1, 1, dict(NK=6, Maxk=0.1)), ((16, 9, 8), 3, 2, 2, 1, dict(NK=20, Maxk=0.2)),
         ((65, 34, 33), 3, 3, 1, 1, dict(NK=40, Maxk=0.3)), ((34, 65, 16), 1, 0, 0, 0, dict(NK=1, Maxk=0.05)),
         ((31, 31, 31), 2, 2, 1, 1, dict(NK=13, OutputLog=1, Mink=-2.4, Maxk=-0.7)), ((8, 4, 4), 3, 3, 0, 1, dict(NK=5, Maxk=0.05)),
         ((64, 32, 64), 2, 0, 1, 0, dict(NK=300, Maxk=0.2)), ((5, 130, 6), 3, 1, 2, 0, dict(NK=9, Maxk=0.04))]


@pytest.mark.parametrize("il", [0, 1])
@pytest.mark.parametrize("shape,order,los,mom,odd,bins", CASES)
def test_fp64_bins_and_paint(gpu, shape, order, los, mom, odd, bins, il):
    po, pc = params_pair(NX=shape[0], NY=shape[1], NZ=shape[2], XMIN=-3.0, XMAX=997.0, YMIN=0.0, YMAX=1000.0, ZMIN=10.0,
                         ZMAX=510.0, InterpOrder=order, LOS=los, DoInterlacing=il, Momentum=mom, Odd_Multipoles=odd, NMU=5,
                         **bins)
    parts = particles(po, 5000, seed=sum(shape) + il)
    ref = oracle_run(po, parts, mom)
    res, st, grids, _ = gpu_run(pc, parts, "fp64", grids=True)
    label = f"{shape} order={order} los={los} mom={mom} il={il} odd={odd} {bins}"
    for k in ("ngrid", "nread", "nout"):
        assert st[k] == ref["stats"][k], label
    for k, g in grids.items():
        grid_close(g, ref["painted"][k], po, "fp64", f"{label} {k}")
    if mom == 1:
        norm0 = np.sqrt(np.abs(oracle_run(po, parts, 0)["raw"]["Pk0"] * oracle_run(po, parts, 2)["raw"]["Pk0"]))
    else:
        norm0 = np.abs(ref["raw"]["Pk0"])
    assert_spectrum(res[0], ref["raw"], norm0, "fp64", odd=bool(odd), label=label)
