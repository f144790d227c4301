"""A handle whose march was captured, then given another front: another number
of particles, another layout of the same number, or single pushes between the
front and the march.  The march by graph equals the march launch by launch."""
import numpy as np
import pytest

from tertia_b200 import workload as wl
from tertia_b200.abi import (QS_F_EY, QS_F_RHOBEAM, QS_LAYER_C, QS_SHAPE_CIC, QS_SHAPE_NGP)
from gpu_helpers import cfg_for, rel_l2

pytestmark = pytest.mark.gpu

# FP32: the order of the atomic additions over 6 layers; FP64 likewise
TOL = {"fp32": 1e-4, "fp64fft": 1e-11, "fp64": 1e-11}


def fronts(cfg):
    """A front of ppc particles per cell, the same with every fifth particle
    left out, and as many particles as the first with some cells crowded."""
    a = wl.front_plasma(cfg, seed=5)
    n = len(a["y"])
    b = {k: np.asarray(v)[np.arange(n) % 5 != 0] for k, v in a.items()}
    cell = np.asarray(a["cell"]).copy()
    cell[:n // 2] = np.sort(np.random.default_rng(3).integers(0, cell[n // 2], n // 2))
    c = dict(a, cell=cell.astype(np.int32))
    return a, b, c


def marches(cfg, graph, every=0):
    from tertia_b200.mesh import Mesh
    cfg = cfg.copy()
    cfg.use_graph = graph
    a, b, c = fronts(cfg)
    out = []
    with Mesh(cfg) as m:
        m.load_beam(wl.small_beam(cfg, n=2000))
        m.move_beam_particles()
        for front, pushes in ((a, 0), (b, 0), (c, 0), (a, 1), (b, 2), (c, 4), (a, 5), (a, 0)):
            m.load_front_plasma(front)
            for _ in range(pushes):
                m.move_particles_layer(0, 0, 1)
            m.move_all_split_layers()
            m.sync()
            out.append((m.onaxis_ex(), m.get_field3d(QS_F_EY, 1), m.get_plasma()["w"]))
    return out


@pytest.mark.parametrize("prec,shape,n", [("fp32", QS_SHAPE_CIC, 32), ("fp32", QS_SHAPE_CIC, 64),
                                          ("fp64fft", QS_SHAPE_CIC, 64), ("fp32", QS_SHAPE_NGP, 64),
                                          ("fp64", QS_SHAPE_NGP, 32), ("fp64", QS_SHAPE_CIC, 32)])
def test_captured_march_with_another_front(prec, shape, n):
    cfg = cfg_for(prec, n=n, layers=6, shape=shape, ts=0.0, synchrotron=0)
    plain, graph = marches(cfg, 0), marches(cfg, 1)
    for i, (p, g) in enumerate(zip(plain, graph)):
        assert np.max(np.abs(p[0])) > 0
        for x, y in zip(p, g):
            assert x.shape == y.shape
            assert rel_l2(y, x) < TOL[prec], i


@pytest.mark.parametrize("store", ["", "0"])
def test_captured_adjoint_with_another_layout(monkeypatch, store):
    """NGP's kernel for particles in lattice order is not replayed for others."""
    from tertia_b200.mesh import Mesh
    if store:
        monkeypatch.setenv("QS_ADJ_FIELDS", store)
    base = cfg_for("fp64", n=32, layers=6, shape=QS_SHAPE_NGP, ts=0.0, synchrotron=0)
    grads = []
    for prec in ("fp64", "fp32"):
        cfg = cfg_for(prec, n=32, layers=6, shape=QS_SHAPE_NGP, ts=0.0, synchrotron=0)
        a, _, c = fronts(base)
        with Mesh(cfg) as m:
            m.load_beam(wl.small_beam(cfg, n=2000))
            m.load_front_plasma(a)
            m.adjoint_checkpoints(3)
            m.move_beam_particles()
            g = np.zeros(cfg.nx)
            g[:2] = 1.0
            for front in (a, c):
                m.load_front_plasma(front)
                m.move_all_split_layers()
                grads.append(m.adjoint(g))
    for x, y in zip(grads[:2], grads[2:]):
        assert np.linalg.norm(x) > 0
        assert rel_l2(y, x) < 1e-4


def test_layer_after_a_replayed_march():
    """After a march by graph the C layer is layer 0, whichever layer single
    calls stopped at before."""
    from tertia_b200.mesh import Mesh
    cfg = cfg_for("fp64", n=32, layers=6, shape=QS_SHAPE_NGP, ts=0.0, synchrotron=0)
    with Mesh(cfg) as m:
        m.load_beam(wl.small_beam(cfg, n=2000))
        m.move_beam_particles()
        m.move_all_split_layers()
        first = m.get_layer(QS_LAYER_C, QS_F_RHOBEAM)
        m.begin_march()
        m.layer_begin(cfg.nx - 2, 0)
        assert np.any(m.get_layer(QS_LAYER_C, QS_F_RHOBEAM) != first)
        m.move_all_split_layers()
        np.testing.assert_array_equal(m.get_layer(QS_LAYER_C, QS_F_RHOBEAM), first)
