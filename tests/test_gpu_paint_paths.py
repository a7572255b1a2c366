"""The FP32 paint's variants by size, held to the oracle exactly. Particles lie on quarters of cells of size 1 with
integer velocities, so every deposit is a multiple of 2^-6 (CIC) or 2^-15 (TSC) that FP32, the tiles' int32
fixed point (scale 2^15 or finer up to 16384 unit records) and their two-limb cells hold exactly: cells and
counters are equal, whatever the order of the additions.

Covered: bucketing by CTA (few tiles) and by warp (more than 4096 tiles), random order, chunks that are not
full, more entries than a chunk holds; tiles smaller than the default ones, tiles shared by a cluster's CTAs,
and dense tiles (two limbs, several carry rounds) for one, two and four painted slots."""
import numpy as np
import pytest

import capow_gb300 as cg
import oracle as orc
from parity_util import gpu_run, params_pair

pytestmark = pytest.mark.gpu

# (NX, NY, NZ), particles, order, LOS, Momentum, interlacing
CASES = [
    # buckets: few tiles, a chunk that is not full, NN (every particle takes the full rules), many tiles
    ((64, 48, 40), 30011, 3, 0, 0, 1), ((64, 48, 40), 513, 2, 3, 0, 1), ((40, 36, 33), 70001, 1, 0, 0, 1),
    ((20, 20, 20), 40000, 2, 0, 1, 1), ((8, 1024, 2112), 60007, 3, 0, 0, 0), ((8, 1024, 2112), 60007, 2, 3, 0, 1),
    # few and dense tiles: one CTA, clusters, two limbs
    ((32, 32, 32), 5000, 3, 3, 0, 1), ((32, 32, 32), 400000, 2, 0, 1, 1), ((16, 32, 32), 300000, 3, 0, 0, 0),
    ((33, 17, 65), 250000, 3, 2, 0, 1), ((8, 8, 8), 200000, 2, 0, 0, 1), ((64, 64, 64), 900000, 2, 0, 1, 0),
    ((4, 300, 4), 150000, 3, 1, 0, 1), ((64, 64, 64), 2000000, 3, 3, 0, 1),
    # tiles away from the grid's faces: every order, periodic and not, one and two fields
    ((64, 64, 128), 200000, 3, 0, 1, 1), ((64, 64, 128), 200000, 3, 2, 0, 0), ((64, 64, 128), 200000, 2, 0, 0, 1),
    ((64, 64, 128), 200000, 2, 3, 0, 1), ((64, 64, 128), 200000, 2, 0, 1, 1), ((64, 64, 128), 50000, 1, 0, 1, 1),
    ((40, 60, 112), 1000, 3, 3, 0, 1)]


@pytest.mark.parametrize("shape,n,order,los,mom,il", CASES)
def test_paint_variants_equal_the_oracle(gpu, shape, n, order, los, mom, il):
    po, pc = params_pair(NX=shape[0], NY=shape[1], NZ=shape[2], XMIN=0.0, XMAX=float(shape[0]), YMIN=0.0, YMAX=float(shape[1]),
                         ZMIN=0.0, ZMAX=float(shape[2]), InterpOrder=order, LOS=los, DoInterlacing=il, Momentum=mom, NK=8,
                         Maxk=1.0)
    rng = np.random.default_rng(n)
    x, y, z = (rng.integers(0, 4 * m, n) * 0.25 for m in shape)
    v = rng.integers(-3, 4, n).astype(np.float64) if mom else np.zeros(n)
    parts = (x, y, z, v, v, v)
    ref, stats = orc.paint(po, *parts, momentum=mom)[:2]
    _, st, grids, _ = gpu_run(pc, parts, "fp32", grids=True)
    assert st["ngrid"] == stats["ngrid"] and st["nread"] == n and st["nout"] == stats["nout"]
    row = 2 * (shape[2] // 2 + 1)
    for k, g in grids.items():
        a = g.reshape(shape[0], shape[1], row)[:, :, :shape[2]]
        b = ref[k][: shape[0] * shape[1] * row].reshape(shape[0], shape[1], row)[:, :, :shape[2]]
        assert np.array_equal(a, b), f"{shape} {k}: largest difference {np.abs(a - b).max()}"
