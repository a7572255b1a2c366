"""The FP32 readout's listed particles (near a face of the reference's rules: exact FP64 taps, eight lanes a particle or, for
a long list, one) against the FP64 path's gradients: a few of them, one, none, and more than the lanes share; every order, the
wrapping and the open line of sight, one field and two, with and without interlacing, float and double columns. Bound: the
suite's relative L2 difference of FP32 gradients, over the listed particles and over all."""
import numpy as np
import pytest

import capow_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nface", [0, 1, 37, 40001])
@pytest.mark.parametrize("order,los,il,spectra,precision,dtype", [
    (1, 3, 1, None, "fp32", "f4"), (2, 0, 1, None, "fp32", "f8"), (2, 1, 0, ["dd", "dp", "pp"], "fp32", "f4"),
    (3, 0, 0, None, "fp32", "f4"), (3, 2, 1, ["dd", "dp", "pp"], "fp32", "f8"), (3, 3, 1, None, "det", "f4")])
def test_listed_particles(gpu, nface, order, los, il, spectra, precision, dtype):
    import torch

    p = cg.Params(NX=48, NY=40, NZ=64, XMIN=0.0, XMAX=480.0, YMIN=0.0, YMAX=400.0, ZMIN=0.0, ZMAX=640.0, InterpOrder=order,
                  DoInterlacing=il, NK=14, Maxk=0.3, LOS=los, Momentum=0)
    rng = np.random.default_rng(nface + order)
    n = 50000
    pos = [rng.uniform(30.0, s - 30.0, n) for s in (480.0, 400.0, 640.0)]
    face = rng.permutation(n)[:nface]
    for k, i in enumerate(face):  # the first and second cell's steps, the low and the high faces, both stencils' halves
        s = (480.0, 400.0, 640.0)[k % 3]
        pos[k % 3][i] = (5.0, 10.0, 0.0, s - 10.0, s - 5.0, s - 1e-3)[k // 3 % 6]
    v = rng.normal(0.0, 0.3, n)
    w = rng.uniform(0.5, 1.5, n)
    parts = [torch.tensor(a.astype(dtype), device=gpu) for a in (*pos, v, w)]
    dl = {"Pk0": np.cos(0.4 * np.arange(14)), "Pk2": 0.5 * np.sin(0.3 * np.arange(14))}
    out = {}
    for prec in (precision, "fp64"):
        with cg.PowerSpectrum(p, precision=prec, spectra=spectra) as ps:
            ps.paint(*parts)
            ps.power()
            g = {k: torch.empty_like(parts[0]) for k in ("dx", "dy", "dz", "dvlos", "dw")}
            ps.backward([dl] * 3 if spectra else dl, out=g)
            out[prec] = {k: a.double().cpu().numpy() for k, a in g.items()}
    # CIC's derivative jumps at a node, and a particle put on one along the line of sight is moved off it by 1e-3 cells a unit
    # of velocity: under 0.02 (5 steps of a float at 47) the two precisions may differ in the side, and each is a derivative
    keep = np.ones(n, bool)
    if order == 2 and los:
        keep = ~(((pos[los - 1] % 10.0) == 0) & (np.abs(v) < 0.02))
        face = face[keep[face]]
    for k, b in out["fp64"].items():
        a, b = out[precision][k] * keep, b * keep
        for sel in (slice(None), face):
            # (against the mean gradient of all particles where a few listed ones have a smaller one)
            scale = max(np.linalg.norm(b[sel]), np.linalg.norm(b) * np.sqrt(np.size(b[sel]) / n))
            assert np.linalg.norm(a[sel] - b[sel]) <= 2e-3 * scale, (k, np.linalg.norm(a[sel] - b[sel]), scale)
