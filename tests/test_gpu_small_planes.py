"""The one-launch transform of small planes: all sizes and kinds, a batch of one,
of eight and of more than a launch takes, in place, and planes whose output
overlaps the next plane's input (which takes the two-pass form)."""
import numpy as np
import pytest

from gpu_helpers import cfg_for, rel_l2

pytestmark = pytest.mark.gpu

TOL = {"fp64fft": 1e-13, "fp32": 2e-6}   # those of the transforms' own tests


@pytest.mark.parametrize("prec", ["fp32", "fp64fft"])
@pytest.mark.parametrize("nz,ny,batch", [(32, 32, 1), (32, 64, 8), (32, 128, 3), (64, 32, 11),
                                         (64, 64, 2), (64, 128, 8), (128, 32, 1), (128, 64, 5),
                                         (128, 128, 9)])
def test_small_planes(oracle_lib, prec, nz, ny, batch):
    import torch
    from tertia_b200.mesh import Mesh
    cfg = cfg_for(prec, n=8, layers=2)
    cfg.ny, cfg.nz = ny, nz
    rng = np.random.default_rng(ny * 5 + nz + batch)
    x = rng.standard_normal((batch, nz, ny))
    dt = torch.float32 if prec == "fp32" else torch.float64
    dev = torch.as_tensor(x, device="cuda").to(dt)
    exact_in = dev.cpu().double().numpy()
    plane = nz * ny
    with Mesh(cfg) as m:
        for kz, ky in ((0, 0), (0, 1), (1, 0), (1, 1)):
            ref = oracle_lib.transform2d(exact_in, kz, ky)
            for shift in (None, 0, plane, 7 * plane):   # apart, in place, one and more planes on
                n = batch * plane
                buf = torch.zeros(3 * n + 8 * plane, dtype=dt, device="cuda")
                buf[:n] = dev.reshape(-1)
                at = 2 * n if shift is None else shift
                torch.cuda.synchronize()
                if shift and batch > 8:
                    continue   # a later launch's input is overwritten by an earlier one's output
                m.transform2d_dev(kz, ky, batch, buf.data_ptr(), buf[at:].data_ptr())
                m.sync()
                y = buf[at:at + n].cpu().double().numpy().reshape(x.shape)
                assert rel_l2(y, ref) < TOL[prec], (kz, ky, shift, rel_l2(y, ref))
