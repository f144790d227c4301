"""The counting sort that regroups the plasma by cell every few full pushes of
the grouped CIC push: at each interval, over crowded cells, and around an
adjoint that recomputes from its checkpoints."""
import numpy as np
import pytest

from tertia_b200 import workload as wl
from tertia_b200.abi import (PRECISIONS, QS_F_JX, QS_F_JY, QS_F_JZ, QS_LAYER_C, QS_LAYER_P,
                             QS_SHAPE_CIC)
from gpu_helpers import cfg_for, rel_l2
from test_gpu_push_rows import TOL, crowd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [1, 2, 4])
@pytest.mark.parametrize("prec,ny,nz,hy", [("fp32", 32, 32, 0.2), ("fp32", 64, 8, 0.01),
                                           ("fp32", 96, 40, 0.01), ("fp64fft", 64, 32, 0.2),
                                           ("fp64fft", 32, 64, 0.01)])
def test_pushes_through_regroupings(oracle_lib, monkeypatch, prec, ny, nz, hy, every):
    """Each of six full pushes and a half one against the oracle's push of the
    state before it, particle by particle (load order); the launches show
    where a regrouping (a scan and a scatter) ran."""
    from tertia_b200.mesh import Mesh
    monkeypatch.setenv("QS_CIC_REGROUP", str(every))
    cfg = cfg_for(prec, n=32, layers=4, shape=QS_SHAPE_CIC)
    cfg.ny, cfg.nz, cfg.hy, cfg.hz = ny, nz, hy, hy
    p, P, C = crowd(cfg, 5 * ny + nz)
    tp, tx, td = TOL[prec]
    dt = np.float32 if prec == "fp32" else np.float64
    with Mesh(cfg) as m:
        m.load_front_plasma(p)
        for c in range(6):
            m.set_layer(QS_LAYER_P, c, P[c])
            m.set_layer(QS_LAYER_C, c, C[c])
        for i in range(7):
            full = i < 6
            a = m.get_plasma()
            k0 = m.kernel_launches()
            m.move_particles_layer(0, 0, int(full))
            ran = m.kernel_launches() - k0
            # a first push counts and scans; one behind a counting push scans and scatters
            assert ran == (3 if i % every == 0 else 1), (i, ran)
            q = m.get_plasma()
            m.sync()
            dep = np.stack([m.get_layer(QS_LAYER_C, f) for f in (QS_F_JX, QS_F_JY, QS_F_JZ)])
            np.testing.assert_array_equal(q["w"], p["w"])
            a = {k: (np.asarray(v, dt) if k != "cell" else v) for k, v in a.items()}
            r = oracle_lib.push_layer(cfg, a["cell"], a["y"], a["z"], a["px"], a["py"], a["pz"],
                                      a["w"], P.astype(dt), C.astype(dt), full=full, precise=True,
                                      dtype=dt)
            for k in ("px", "py", "pz"):
                np.testing.assert_allclose(q[k], r[k], rtol=tp, atol=tp)
            for axis, at, size in (("y", lambda c: c % ny, ny), ("z", lambda c: c // ny, nz)):
                d = ((at(q["cell"]) + q[axis]) -
                     (at(np.asarray(r["cell"])) + np.asarray(r[axis], float)))
                d -= size * np.round(d / size)   # periodic
                assert np.max(np.abs(d)) < tx, (i, axis)
            assert rel_l2(dep, np.asarray(r["dep"], float)[:3]) < td, i


@pytest.mark.parametrize("prec", ["fp32", "fp64fft"])
@pytest.mark.parametrize("profile", [True, False])
def test_pushes_after_an_adjoint(monkeypatch, prec, profile):
    """A regrouping left due before the adjoint (by the march where every
    kernel is profiled, else by single pushes) does not count its particles
    into the first regrouping after it."""
    from tertia_b200.mesh import Mesh
    monkeypatch.setenv("QS_ADJ_FIELDS", "0")
    cfg = wl.small_config(n=64, layers=8, ts=0.0, synchrotron=0, shape=QS_SHAPE_CIC)
    cfg.precision = PRECISIONS[prec]
    front = wl.front_plasma(cfg, seed=3)
    with Mesh(cfg) as m:
        m.load_beam(wl.small_beam(cfg, n=2000))
        m.load_front_plasma(front)
        m.adjoint_checkpoints(4)
        m.move_beam_particles()
        m.profile_enable(profile)
        m.move_all_split_layers()
        if not profile:
            for _ in range(4):
                m.move_particles_layer(0, 0, 1)
        g = np.zeros(cfg.nx)
        g[:2] = 1.0
        assert np.any(m.adjoint(g))
        for _ in range(5):   # the fifth one follows a regrouping
            m.move_particles_layer(0, 0, 1)
        m.sync()
        np.testing.assert_array_equal(m.get_plasma()["w"],
                                      np.asarray(front["w"], np.float32 if prec == "fp32" else float))


def test_pushes_after_a_replayed_adjoint(monkeypatch):
    """The same when the sweep is replayed: single pushes leave a regrouping
    due, and the replay restores checkpoints like the captured run did."""
    from tertia_b200.mesh import Mesh
    monkeypatch.setenv("QS_ADJ_FIELDS", "0")
    cfg = wl.small_config(n=64, layers=8, ts=0.0, synchrotron=0, shape=QS_SHAPE_CIC)
    cfg.precision = PRECISIONS["fp32"]
    front = wl.front_plasma(cfg, seed=3)
    g = np.zeros(cfg.nx)
    g[:2] = 1.0
    with Mesh(cfg) as m:
        m.load_beam(wl.small_beam(cfg, n=2000))
        m.load_front_plasma(front)
        m.adjoint_checkpoints(4)
        m.move_beam_particles()
        for _ in range(3):
            m.load_front_plasma(front)
            m.move_all_split_layers()
            for _ in range(4):
                m.move_particles_layer(0, 0, 1)
            assert np.any(m.adjoint(g))
            for _ in range(5):
                m.move_particles_layer(0, 0, 1)
            m.sync()
