"""A device that is nearly full: what fits the layouts without the blocked path's buffers still runs. Each workload runs once
with all of the memory, which measures what it holds, then with less than that by a part of the blocked path's extra buffers
(a bounded filler allocation takes the rest), so that an allocation after the context's creation finds no room."""
import numpy as np
import pytest

import capow_gb300 as cg
from parity_util import TOL

pytestmark = pytest.mark.gpu

N = 256
GRID = 4 * N * N * (N + 2)  # bytes of one painted slot


def params(**kw):
    base = dict(NX=N, NY=N, NZ=N, NK=40, Maxk=0.6, XMIN=0.0, XMAX=1000.0, YMIN=0.0, YMAX=1000.0, ZMIN=0.0, ZMAX=1000.0,
                InterpOrder=3, DoInterlacing=1, LOS=3, Momentum=0)
    return cg.Params(**{**base, **kw})


def particles(dev, n):
    import torch

    g = torch.Generator(device=dev)
    g.manual_seed(5)
    pos = [torch.rand(n, generator=g, device=dev) * 999.0 for _ in range(3)]
    return (*pos, 300.0 * torch.randn(n, generator=g, device=dev))


def same(a, b):
    for r, q in zip(a, b):
        assert np.array_equal(r["Nmodes"], q["Nmodes"])
        for k in ("Pk0", "Pk2", "Pk4"):
            assert np.abs(r[k] - q[k]).max() <= TOL["fp32"][0] * max(np.abs(q["Pk0"]).max(), np.abs(q["Pk2"]).max()), k


def both(run, less):
    """run(held), held() the bytes held since the start of it, with all of the memory and with `less` bytes less than it
    needs."""
    import torch

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    f0 = free()
    need = [0]

    def held():
        need[0] = f0 - torch.cuda.mem_get_info()[0]
        return need[0]

    first = run(held)
    f0 = free()
    filler = torch.empty(f0 - (need[0] - less), dtype=torch.uint8, device="cuda")
    f0 = torch.cuda.mem_get_info()[0]
    try:
        return first, run(held)
    finally:
        del filler
        torch.cuda.empty_cache()


@pytest.mark.parametrize("host", [False, True])
def test_paint_after_a_blocked_context(gpu, host):
    parts = particles(gpu, 8000000)
    if host:
        parts = [t.cpu().numpy() for t in parts]

    def run(held):
        with cg.PowerSpectrum(params(), precision="fp32", spectra=["dd", "pp"]) as ps:
            assert held() > 11 * GRID  # grids, planes and columns: the blocked path
            ps.paint(*parts)
            r = ps.power()
            ps.paint(*parts)
            again = ps.power()
            held()
            same(again, r)
            return r

    a, b = both(run, 2 * GRID)
    same(b, a)


def test_backward_after_a_blocked_forward(gpu):
    parts = [t.cpu().numpy() for t in particles(gpu, 4000000)]
    dL = {"Pk0": np.linspace(1.0, 2.0, 40), "Pk2": np.linspace(-1.0, 1.0, 40)}

    def run(held):
        with cg.PowerSpectrum(params(), precision="fp32") as ps:
            assert held() > 5 * GRID
            ps.paint(*parts)
            ps.power()
            ps.paint(*parts)
            r = ps.power()
            g = ps.backward(dL)
            held()
            return r, {k: np.array(v.cpu() if hasattr(v, "cpu") else v) for k, v in g.items()}

    (r0, g0), (r1, g1) = both(run, GRID // 2)
    same(r1, r0)
    for k in ("dx", "dy", "dz"):
        assert np.abs(g1[k] - g0[k]).max() <= 1e-3 * np.abs(g0[k]).max(), k


def test_batch_of_blocked_contexts(gpu):
    parts = (*particles(gpu, 4000000), None)

    def run(held):
        cg.release_batch()
        out = cg.run_batch([(params(), parts), (params(NZ=N // 2), parts)], precision="fp32")
        held()
        cg.release_batch()
        assert all(status == cg.OK for status, _ in out)
        return [r[0] for _, r in out]

    a, b = both(run, GRID)
    same(b, a)


def test_survey_after_a_blocked_context(gpu):
    import torch

    x, y, z, _ = particles(gpu, 4000000)
    ones = torch.ones_like(x)
    cats = [dict(x=x[a], y=y[a], z=z[a], w=ones[a], nbar=1e-3 * ones[a]) for a in (slice(0, 400000), slice(400000, None))]
    sv = cg.SurveyParams(X_Origin=500.5, Y_Origin=500.25, Z_Origin=499.0, FKP_Column=-1, FKP_Pk=1e4, NBAR_Column=5)

    def run(held):
        with cg.SurveySpectrum(params(LOS=0), sv, precision="fp32") as ss:
            created = held()
            r = ss.power(*cats)
            held()
            return created, r

    (c0, a), (c1, b) = both(run, GRID // 2)
    assert abs(c0 - c1) < GRID // 8  # the blocked path in both contexts
    same([b], [a])


def test_records_of_small_tiles(gpu):
    """A grid of few tiles takes smaller ones, which list a particle more often: where their records do not fit, the default
    tiles are taken."""
    parts = particles(gpu, 8000000)

    def run(held):
        with cg.PowerSpectrum(params(NX=32, NY=32, NZ=32, Maxk=0.09, NK=10), precision="fp32") as ps:
            ps.paint(*parts)
            r = ps.power()
            ps.paint(*parts)
            ps.stats()
            held()
            return r, ps.tile_kernel_ms()[1]

    (a, small), (b, default) = both(run, 100 << 20)
    assert default < 0.8 * small  # records listed
    same(b, a)
