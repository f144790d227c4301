"""The map kernels between the halves of the transforms, at every row width
they are compiled for: marches over a few layers with no, one and two inner
iterations and with split layers, against the oracle."""
import numpy as np
import pytest

from tertia_b200 import workload as wl
from tertia_b200.abi import QS_SHAPE_CIC, QS_SHAPE_NGP
from gpu_helpers import cfg_for, rel_l2

pytestmark = pytest.mark.gpu

# the tolerances of the whole-march tests: rounding in FP64, the benchmark's
# 1e-5 in FP32
TOL = {"fp64fft": 1e-10, "fp32": 1e-5}


@pytest.mark.parametrize("prec,ny,nz", [("fp32", 32, 64), ("fp32", 64, 32), ("fp32", 128, 32),
                                        ("fp32", 256, 64), ("fp32", 512, 32), ("fp32", 1024, 32),
                                        ("fp64fft", 64, 32), ("fp64fft", 128, 64),
                                        ("fp64fft", 256, 32), ("fp64fft", 512, 32)])
def test_march_matches_oracle_at_every_row_width(oracle_lib, prec, ny, nz):
    from tertia_b200.mesh import Mesh
    for n_iter, split, shape in ((0, 1, QS_SHAPE_CIC), (2, 1, QS_SHAPE_CIC), (1, 2, QS_SHAPE_CIC),
                                 (1, 1, QS_SHAPE_NGP)):
        cfg = cfg_for(prec, n=32, layers=7, shape=shape, n_iter=n_iter, nx_split=split)
        cfg.ny, cfg.nz = ny, nz
        cfg.hy, cfg.hz = 6.4 / ny, 6.4 / nz
        # (fine cells: enough particles that no cell's beam current passes the solver's limit)
        beam = wl.small_beam(cfg, n=100_000, nb=0.2)
        front = wl.front_plasma(cfg, seed=ny)
        o = oracle_lib.Oracle(cfg)
        o.load_beam(beam)
        o.load_front_plasma(front)
        o.step()
        with Mesh(cfg) as m:
            m.load_beam(beam)
            m.load_front_plasma(front)
            m.step()
            got = np.stack([np.stack([m.get_field3d(f, i) for f in range(6)])
                            for i in range(cfg.nx)])
        ref = np.stack([np.stack([o.get_field3d(f, i) for f in range(6)]) for i in range(cfg.nx)])
        assert np.max(np.abs(ref)) > 0
        assert rel_l2(got, ref) < TOL[prec], (n_iter, split, shape, rel_l2(got, ref))
