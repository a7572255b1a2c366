"""Dense FP32 tiles (many records a tile), held to the oracle exactly. Positions lie on odd eighths of cells of size 1 (TSC:
on quarters), weights on eighths and velocities on integers, so every deposit is a multiple of 2^-18 or coarser whose sums
FP32 holds: cells and counters are equal, whatever the order of the additions.

Covered: tiles just above the dense limit whose records are shared by a cluster's CTAs (a few hundred records and fewer per
CTA, each of them a large part of the CTA's sum), one, two and four painted slots; one record far above the others of
its tile (int64 cells), in a cluster and by one CTA over many carry rounds."""
import numpy as np
import pytest

import capow_gb300 as cg
import oracle as orc
from parity_util import params_pair

pytestmark = pytest.mark.gpu

# (NX, NY, NZ), particles, order, Momentum, interlacing. Tiles of 8^3: 8, 27, 64, 80 and 96 of them, of about 1.4 (NN), 2.6
# (CIC, TSC) records per particle
CASES = [((32, 32, 32), 48000, 1, 0, 0), ((32, 32, 32), 50000, 1, 0, 1), ((32, 32, 32), 60000, 1, 0, 0),
         ((32, 32, 32), 80000, 1, 0, 0), ((32, 32, 32), 125000, 1, 0, 0), ((24, 24, 24), 21000, 1, 0, 0),
         ((16, 16, 16), 6300, 1, 0, 0), ((16, 16, 16), 8000, 1, 0, 1), ((32, 32, 48), 75000, 1, 0, 0),
         ((32, 32, 40), 55000, 2, 0, 0), ((32, 32, 32), 36000, 2, 0, 0), ((32, 32, 32), 50000, 2, 0, 1),
         ((24, 24, 24), 15000, 2, 0, 0), ((16, 16, 16), 5000, 2, 0, 1), ((32, 32, 32), 30000, 3, 0, 0),
         ((32, 32, 32), 94000, 1, 1, 1), ((16, 16, 16), 6500, 2, 1, 1), ((24, 24, 24), 22000, 2, 1, 1)]


def catalogue(shape, n, order, seed, lo=(0, 0, 0), hi=None):
    rng = np.random.default_rng(seed)
    hi = hi or shape
    if order == 3:
        pos = [rng.integers(4 * a, 4 * b, n) * 0.25 for a, b in zip(lo, hi)]
    else:
        pos = [rng.integers(4 * a, 4 * b, n) * 0.25 + 0.125 for a, b in zip(lo, hi)]
    return pos, rng.integers(-3, 4, n).astype(np.float64), rng.integers(4, 13, n) * 0.125


def paint(shape, order, los, mom, il, pos, v, w):
    po, pc = params_pair(NX=shape[0], NY=shape[1], NZ=shape[2], XMIN=0.0, XMAX=float(shape[0]), YMIN=0.0, YMAX=float(shape[1]),
                         ZMIN=0.0, ZMAX=float(shape[2]), InterpOrder=order, LOS=los, DoInterlacing=il, Momentum=mom, NK=8,
                         Maxk=1.0)
    ref, stats = orc.paint(po, *pos, v, v, v, w=w, momentum=mom)
    with cg.PowerSpectrum(pc, precision="fp32") as ps:
        ps.paint(*pos, v, w)
        st = ps.stats()
        assert st["nread"] == len(w) and st["nout"] == stats["nout"]
        row = 2 * (shape[2] // 2 + 1)
        names = ["ddg", "ddg_interlace", "ddg_mom", "ddg_mom_interlace"]
        for which in [k for k in range(4) if (il or k % 2 == 0) and (mom or k < 2)]:
            a = ps.grid(which).reshape(shape[0], shape[1], row)[:, :, :shape[2]]
            b = ref[names[which]][: shape[0] * shape[1] * row].reshape(shape[0], shape[1], row)[:, :, :shape[2]]
            yield f"{shape} {names[which]}", a, b


@pytest.mark.parametrize("shape,n,order,mom,il", CASES)
def test_shared_dense_tiles_equal_the_oracle(gpu, shape, n, order, mom, il):
    pos, v, w = catalogue(shape, n, order, n)
    for name, a, b in paint(shape, order, 0, mom, il, pos, v if mom else np.zeros(n), w):
        assert np.array_equal(a, b), f"{name}: largest difference {np.abs(a - b).max()}, {np.mean(a != b):.3f} of the cells"


@pytest.mark.parametrize("shape,n,lo,hi,order,il", [((32, 32, 32), 150000, (0, 0, 0), None, 1, 1),
                                                   ((32, 32, 32), 300000, (0, 0, 0), None, 2, 0),
                                                   ((128, 128, 256), 200000, (17, 18, 34), (30, 30, 60), 1, 0),
                                                   ((128, 128, 256), 200000, (17, 18, 34), (30, 30, 60), 2, 0)])
def test_one_record_far_above_the_others(gpu, shape, n, lo, hi, order, il):
    """A weight of 2^36 among weights of about 1: the cells that it does not touch are exact, the others within the rounding
    of the cell."""
    pos, v, w = catalogue(shape, n, order, n + order, lo, hi)
    w[n // 2] = 2.0 ** 36
    for name, a, b in paint(shape, order, 3, 0, il, pos, np.zeros(n), w):
        light = b < 2.0 ** 20
        assert np.array_equal(a[light], b[light]), f"{name}: largest difference {np.abs(a - b)[light].max()}"
        assert np.abs(a / np.where(light, 1.0, b) - 1.0)[~light].max(initial=0.0) <= 2.0 ** -23, name


@pytest.mark.parametrize("shape,n,order", [((16, 16, 16), 1200, 2), ((16, 16, 16), 1900, 2), ((16, 16, 16), 2600, 1),
                                           ((16, 16, 16), 4000, 1), ((32, 32, 32), 14000, 2), ((64, 64, 64), 155648, 2),
                                           ((64, 64, 64), 155649, 3), ((64, 64, 64), 467000, 1),
                                           ((64, 64, 64), 16383, 1), ((64, 64, 64), 16383, 3), ((64, 64, 64), 16384, 2)])
def test_one_slot_around_the_bucket_limits(gpu, shape, n, order):
    """One slot with buckets that end below and above the dense limit, half of the catalogue in one tile (beyond its bucket);
    catalogues of one and more particles a thread of the bucketing, and at the line between its two forms."""
    pos, v, w = catalogue(shape, n, order, n)
    half, _, _ = catalogue(shape, n, order, n + 1, (1, 1, 1), (7, 7, 7))
    pos = [np.where(np.arange(n) % 2 == 0, h, p) if n < 20000 else p for h, p in zip(half, pos)]
    for name, a, b in paint(shape, order, 0, 0, 0, pos, np.zeros(n), w):
        assert np.array_equal(a, b), f"{name}: largest difference {np.abs(a - b).max()}"
