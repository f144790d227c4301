"""The grouped CIC push of a layer whose particle arrays are 4 GB each, past
the reach of a 32-bit byte offset: both widths, with the regrouping."""
import numpy as np
import pytest

from tertia_b200.abi import (QS_F_DENS, QS_F_JX, QS_LAYER_C, QS_SHAPE_CIC)
from gpu_helpers import cfg_for

pytestmark = pytest.mark.gpu


def available_gb():
    with open("/proc/meminfo") as f:
        kb = next(int(line.split()[1]) for line in f if line.startswith("MemAvailable"))
    return kb / 2**20


@pytest.mark.parametrize("prec,ppc", [("fp64fft", 2048), ("fp32", 4096)])
def test_row_push_of_4gb_arrays(oracle_lib, monkeypatch, prec, ppc):
    import torch
    from tertia_b200.mesh import Mesh
    n = 512 * 512 * ppc
    free, _ = torch.cuda.mem_get_info()
    if free < 96 * 2**30 or available_gb() < 24 * n / 2**30 + 16:
        pytest.skip("needs 96 GB on the device and three arrays of the particles on the host")
    monkeypatch.setenv("QS_CIC_REGROUP", "1")
    cfg = cfg_for(prec, n=512, layers=2, shape=QS_SHAPE_CIC)
    # every particle in the middle of its cell with px = 0.5: no field, no
    # move, and every node gets what one particle per cell would, ppc times
    half = np.full(n, 0.5)
    zero = np.zeros(n)   # never written: its pages take no memory
    small = cfg_for(prec, n=32, layers=2, shape=QS_SHAPE_CIC)
    dt = np.float32 if prec == "fp32" else np.float64
    one = np.full(32 * 32, 0.5)
    F = np.zeros((6, 32, 32))
    r = oracle_lib.push_layer(small, np.arange(32 * 32), one, one, one, 0 * one, 0 * one, one, F, F,
                              precise=True, dtype=dt)
    # sums of ppc equal terms one after another: half an ulp each
    tol = ppc * np.finfo(dt).eps
    with Mesh(cfg) as m:
        m.load_front_plasma(dict(cell=np.repeat(np.arange(512 * 512, dtype=np.int32), ppc),
                                 y=half, z=half, px=half, py=zero, pz=zero, w=half))
        del half, zero
        for full in (0, 1, 0):   # the last one behind a regrouping
            m.move_particles_layer(1, 0, full)
            for f, q in ((QS_F_JX, 0), (QS_F_DENS, 3)):
                want = ppc * float(r["dep"][q][16, 16])
                assert want != 0
                np.testing.assert_allclose(m.get_layer(QS_LAYER_C, f), want, rtol=tol)
        m.sync()
