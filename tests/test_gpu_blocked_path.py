"""Power-of-two NX (32 to 1024), NY and NZ: z by k_zfft, y by k_yfft, the x axis and the binning by k_xrow_bin.
Held to the oracle and to the 3-D cuFFT + k_bin path on the same catalogue, at the suite's FP32 tolerances, over
every row length of the three kernels, one to four slots, even and odd multipoles, linear and logarithmic bins from one
bin to several hundred, the lines of sight, and top edges from beyond the Nyquist frequency (nothing left out) to a small
part of it (most rows and columns left out)."""
import numpy as np
import pytest

from parity_util import assert_spectrum, gpu_run, oracle_run, params_pair, particles

pytestmark = pytest.mark.gpu

BOX = dict(XMIN=-3.0, XMAX=997.0, YMIN=0.0, YMAX=1000.0, ZMIN=10.0, ZMAX=510.0, NMU=5)

# (NX, NY, NZ), order, LOS, interlacing, Momentum, odd, bins
CASES = [((64, 16, 32), 3, 3, 1, 1, 1, dict(NK=24, Maxk=0.55)),
         ((64, 1024, 32), 2, 0, 1, 0, 0, dict(NK=1, Maxk=0.2)),
         ((128, 64, 128), 3, 1, 1, 1, 0, dict(NK=40, Maxk=0.2)),
         ((128, 32, 64), 1, 0, 0, 0, 1, dict(NK=300, Maxk=0.1)),
         ((256, 128, 64), 3, 2, 1, 1, 0, dict(NK=24, Maxk=0.06)),
         ((256, 16, 32), 2, 0, 0, 1, 1, dict(NK=10, OutputLog=1, Mink=-2.5, Maxk=-0.3)),
         ((512, 32, 128), 2, 3, 1, 2, 1, dict(NK=33, OutputLog=1, Mink=-2.2, Maxk=-1.1)),
         ((512, 64, 32), 3, 1, 1, 1, 1, dict(NK=16, Maxk=0.55)),
         ((1024, 32, 64), 3, 1, 1, 0, 0, dict(NK=64, Maxk=0.1)),
         ((1024, 16, 128), 2, 3, 1, 1, 1, dict(NK=20, Maxk=0.05)),
         ((64, 256, 1024), 2, 2, 0, 1, 0, dict(NK=12, Maxk=0.02)),
         ((64, 512, 2048), 1, 0, 1, 0, 0, dict(NK=500, Maxk=0.2)),
         ((32, 32, 32), 3, 3, 1, 1, 1, dict(NK=16, Maxk=0.1)), ((32, 16, 64), 2, 1, 1, 0, 0, dict(NK=100, Maxk=0.05)),
         ((32, 1024, 32), 1, 0, 0, 1, 1, dict(NK=9, Maxk=0.02)), ((32, 64, 32), 3, 2, 0, 0, 0, dict(NK=1, Maxk=0.2))]


@pytest.mark.parametrize("precision", ["fp32", "det"])
@pytest.mark.parametrize("shape,order,los,il,mom,odd,bins", CASES)
def test_blocked_path_parity(gpu, precision, shape, order, los, il, mom, odd, bins):
    po, pc = params_pair(NX=shape[0], NY=shape[1], NZ=shape[2], InterpOrder=order, LOS=los, DoInterlacing=il, Momentum=mom,
                         Odd_Multipoles=odd, **BOX, **bins)
    parts = particles(po, 6000, seed=40 + sum(shape) + mom)
    raw = oracle_run(po, parts, mom)["raw"]
    res, _, _, _ = gpu_run(pc, parts, precision)
    res3, _, _, _ = gpu_run(pc, parts, precision, fft_path="3d")
    if mom == 1:
        norm0 = np.sqrt(np.abs(oracle_run(po, parts, 0)["raw"]["Pk0"] * oracle_run(po, parts, 2)["raw"]["Pk0"]))
    else:
        norm0 = np.abs(raw["Pk0"])
    label = f"{precision} {shape} order={order} los={los} il={il} mom={mom} odd={odd} {bins}"
    assert_spectrum(res[0], raw, norm0, precision, odd=bool(odd), label=label)
    assert_spectrum(res[0], res3[0], norm0, precision, odd=bool(odd), label=label + " vs 3d")


def test_blocked_path_in_plane_chunks(gpu):
    """Four slots of 256 x 1024 x 2048: the z and y passes run on two chunks of planes."""
    _, pc = params_pair(NX=256, NY=1024, NZ=2048, InterpOrder=2, LOS=3, DoInterlacing=1, Momentum=1, NK=32, Maxk=0.7, **BOX)
    parts = particles(pc, 300000, seed=77)
    res, st, _, _ = gpu_run(pc, parts, "fp32", spectra=["dd", "dp", "pp"])
    res3, st3, _, _ = gpu_run(pc, parts, "fp32", spectra=["dd", "dp", "pp"], fft_path="3d")
    assert st["ngrid"] == st3["ngrid"]
    dd, pp = (np.abs(res3[k]["Pk0"]) for k in (0, 2))
    for a, b, n0 in zip(res, res3, (dd, np.sqrt(dd * pp), pp)):
        assert_spectrum(a, b, n0, "fp32", odd=False, label=a["kind"])
