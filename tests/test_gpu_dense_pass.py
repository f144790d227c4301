"""The dense transform pass (plain FP64, and FP32 at sizes that are no power of
two) at the edges of its tiles: one value group, less and more than a 32-wide
output tile, around one and two 64-deep stages and beyond, rectangular, and
planes that start off a 16-byte boundary."""
import numpy as np
import pytest

from gpu_helpers import cfg_for, rel_l2

pytestmark = pytest.mark.gpu

# a sum of n products of 2 cos with unit normals: rounding of order sqrt(n) eps
# relative to the result (n <= 264), with a margin of 30
TOL = {"fp64": 1e-13, "fp32": 2e-6}


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("nz,ny,off", [(8, 8, 0), (8, 24, 0), (24, 40, 1), (40, 64, 0), (56, 72, 1),
                                       (72, 120, 0), (136, 128, 1), (264, 8, 0), (200, 264, 0)])
def test_dense_pass_edges(oracle_lib, prec, nz, ny, off):
    import torch
    from tertia_b200.mesh import Mesh
    cfg = cfg_for(prec, n=8, layers=2)
    cfg.ny, cfg.nz = ny, nz
    rng = np.random.default_rng(ny * 7 + nz)
    x = rng.standard_normal((3, nz, ny))
    dt = torch.float64 if prec == "fp64" else torch.float32
    n = x.size
    # `off` values past the start of an allocation: no 16-byte boundary
    d_in = torch.zeros(n + off, dtype=dt, device="cuda")
    d_out = torch.zeros(n + off, dtype=dt, device="cuda")
    d_in[off:] = torch.as_tensor(x.reshape(-1), device="cuda").to(dt)
    torch.cuda.synchronize()
    with Mesh(cfg) as m:
        for kz, ky in ((0, 0), (0, 1), (1, 0), (1, 1)):
            m.transform2d_dev(kz, ky, 3, d_in[off:].data_ptr(), d_out[off:].data_ptr())
            m.sync()
            y = d_out[off:].cpu().double().numpy().reshape(x.shape)
            ref = oracle_lib.transform2d(d_in[off:].cpu().double().numpy().reshape(x.shape), kz, ky)
            assert rel_l2(y, ref) < TOL[prec], (kz, ky, rel_l2(y, ref))
