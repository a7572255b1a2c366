"""A batch whose mocks of one shape differ widely in their number of bins: the shape's contexts take a layout whose x pass
holds all of them (the blocked x pass keeps 76 bytes a bin of shared memory where the transposed one keeps 52, for one field
without interlacing), and every mock equals its own context."""
import numpy as np
import pytest

import capow_gb300 as cg
from parity_util import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nks", [(40, 3000, 25), (3000, 40), (25, 40, 60)])
def test_batch_of_many_and_few_bins(gpu, nks):
    import torch

    rng = np.random.default_rng(5)
    mocks = []
    for nk in nks:
        p = cg.Params(NX=64, NY=64, NZ=64, XMIN=0.0, XMAX=500.0, YMIN=0.0, YMAX=500.0, ZMIN=0.0, ZMAX=500.0, InterpOrder=2,
                      DoInterlacing=0, NK=nk, Maxk=0.4, LOS=3, Momentum=0)
        pos = [torch.tensor(rng.uniform(0.0, 500.0, 20000), device=gpu) for _ in range(3)]
        mocks.append((p, (*pos, torch.tensor(rng.normal(0.0, 200.0, 20000), device=gpu), None)))
    out = cg.run_batch(mocks, precision="fp32")
    for (p, parts), (status, res) in zip(mocks, out):
        assert status == cg.OK, p.NK
        with cg.PowerSpectrum(p, precision="fp32") as ps:
            ps.paint(*parts[:4])
            ref = ps.power()[0]
        assert np.array_equal(res[0]["Nmodes"], ref["Nmodes"])
        scale = np.abs(ref["Pk0"]).max()
        for k in ("Pk0", "Pk2", "Pk4"):
            assert np.abs(res[0][k] - ref[k]).max() <= TOL["fp32"][0] * scale, (p.NK, k)
