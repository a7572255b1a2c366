"""The batch autotuner's tile shapes are kept per number of painted slots: batches of one grid with four, two and one of
them, in either order, each equal their own contexts."""
import numpy as np
import pytest

import capow_gb300 as cg
from parity_util import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [(["dd", "dp", "pp"], ["dd"], ["pp"]), (["pp"], ["dd", "dp", "pp"], ["dd"])])
@pytest.mark.parametrize("interlace", [1, 0])
def test_tuned_tiles_of_other_slot_counts(gpu, order, interlace):
    import torch

    rng = np.random.default_rng(11)
    n = 150000
    p = cg.Params(NX=128, NY=128, NZ=128 + 32 * interlace, XMIN=0.0, XMAX=500.0, YMIN=0.0, YMAX=500.0, ZMIN=0.0, ZMAX=500.0,
                  InterpOrder=3, DoInterlacing=interlace, NK=30, Maxk=0.6, LOS=3, Momentum=0)
    pos = [torch.tensor(rng.uniform(0.0, 500.0, n), device=gpu) for _ in range(3)]
    parts = (*pos, torch.tensor(rng.normal(0.0, 200.0, n), device=gpu), None)
    for spectra in order:
        (status, res), = cg.run_batch([(p, parts)], precision="fp32", spectra=spectra, autotune=True)
        assert status == cg.OK
        with cg.PowerSpectrum(p, precision="fp32", spectra=spectra) as ps:
            ps.paint(*parts[:4])
            ref = ps.power()
        auto = {r["kind"]: np.abs(r["Pk0"]).max() for r in ref}
        for a, b in zip(res, ref):
            assert np.array_equal(a["Nmodes"], b["Nmodes"])
            scale = np.sqrt(auto["dd"] * auto["pp"]) if b["kind"] == "dp" else auto[b["kind"]]
            for k in ("Pk0", "Pk2", "Pk4"):
                assert np.abs(a[k] - b[k]).max() <= TOL["fp32"][0] * scale, (spectra, b["kind"], k)
