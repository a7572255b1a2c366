"""Host threads with contexts of different grids at once: their kernels are the same functions with other amounts of shared
memory, and no thread's launches are refused or changed by another's."""
import threading

import numpy as np
import pytest

import capow_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,order", [("fp32", 3), ("fp32", 2), ("det", 3)])
def test_threads_with_different_grids(gpu, precision, order):
    import torch

    # (grid, particles): many and few tiles, tiles of 64 KB and of 10 KB a CTA, long and short axes
    grids = [((64, 64, 64), 3000), ((256, 256, 256), 3000), ((128, 128, 128), 3000), ((64, 64, 512), 3000),
             ((96, 64, 64), 3000), ((128, 128, 256), 3000)]
    errors = []

    def work(shape, n, seed):
        try:
            rng = np.random.default_rng(seed)
            p = cg.Params(NX=shape[0], NY=shape[1], NZ=shape[2], XMIN=0.0, XMAX=100.0, YMIN=0.0, YMAX=100.0, ZMIN=0.0,
                          ZMAX=100.0, InterpOrder=order, DoInterlacing=1, NK=20, Maxk=1.0, LOS=3, Momentum=0)
            parts = [torch.tensor(a, device=gpu) for a in (*(rng.uniform(0.0, 100.0, n) for _ in range(3)),
                                                           rng.normal(0.0, 100.0, n))]
            torch.cuda.synchronize()
            first = None
            with cg.PowerSpectrum(p, precision=precision, spectra=["dd", "dp", "pp"]) as ps:
                for _ in range(30):
                    for _ in range(40):  # (launches only, nothing waits for them)
                        ps.paint(*parts)
                    pk = ps.power()[0]["Pk0"]
                    first = pk if first is None else first
                    assert np.abs(pk - first).max() <= 1e-4 * np.abs(first).max()
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append((shape, repr(e)))

    ts = [threading.Thread(target=work, args=(*g, k)) for k, g in enumerate(grids)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[:2]
