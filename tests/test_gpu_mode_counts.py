"""Nmodes counted a column at a time (kx and -kx, ky and -ky together), equal to the oracle's: odd, even and power-of-two
axes around the 32 kx of a warp, linear and logarithmic bins, one bin to several hundred, top edges below and
beyond the Nyquist frequency, cubic cells (many modes exactly on edges) and uneven ones."""
import numpy as np
import pytest

from parity_util import gpu_run, oracle_run, params_pair, particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [dict(NK=1, Maxk=0.5), dict(NK=16, Maxk=0.5), dict(NK=400, Maxk=0.2),
                                  dict(NK=13, OutputLog=1, Mink=-2.4, Maxk=-0.7)])
@pytest.mark.parametrize("shape", [(5, 7, 9), (2, 2, 2), (31, 32, 33), (32, 31, 64), (63, 16, 10), (64, 64, 64), (65, 6, 8),
                                   (130, 9, 4), (96, 100, 36)])
@pytest.mark.parametrize("cubic", [0, 1])
def test_mode_counts_equal_the_oracle(gpu, shape, bins, cubic):
    size = [float(10 * n) for n in shape] if cubic else [973.0, 1000.0, 511.0]
    po, pc = params_pair(NX=shape[0], NY=shape[1], NZ=shape[2], XMIN=0.0, XMAX=size[0], YMIN=0.0, YMAX=size[1], ZMIN=0.0,
                         ZMAX=size[2], InterpOrder=2, LOS=3, DoInterlacing=1, Momentum=0, NMU=5, **bins)
    parts = particles(po, 100, seed=3)
    ref = oracle_run(po, parts, 0)["raw"]["Nmodes"]
    res, _, _, _ = gpu_run(pc, parts, "fp32" if min(shape) >= 4 else "fp64")  # (the FP32 paths take 4 cells and more)
    assert np.array_equal(np.asarray(res[0]["Nmodes"], np.int64), np.asarray(ref, np.int64))
