"""The grouped CIC push at the edges of its windows and tiles: crowded cells
(more particles than a lane's list of moved ones, more than one window of
slots), empty rows, moves of more than one cell per layer (sub-steps), sizes
that are and are not powers of two, and a full push whose cells the next
regrouping counts."""
import numpy as np
import pytest

from tertia_b200.abi import QS_F_JX, QS_F_JY, QS_F_JZ, QS_LAYER_C, QS_LAYER_P, QS_SHAPE_CIC
from gpu_helpers import cfg_for, rel_l2

pytestmark = pytest.mark.gpu


def crowd(cfg, seed):
    """Particles grouped by cell: most cells hold 0 to 6, a few 40, one 300;
    the second row of cells is empty."""
    rng = np.random.default_rng(seed)
    ncell = cfg.ny * cfg.nz
    count = rng.integers(0, 7, ncell)
    count[rng.integers(0, ncell, 6)] = 40
    count[cfg.ny:2 * cfg.ny] = 0
    count[ncell // 2 + 3] = 300
    cell = np.repeat(np.arange(ncell, dtype=np.int32), count)
    n = len(cell)
    p = dict(cell=cell, y=rng.uniform(0, 1, n), z=rng.uniform(0, 1, n),
             w=rng.uniform(0.1, 0.4, n))
    for k in ("px", "py", "pz"):
        p[k] = 0.2 * rng.standard_normal(n)
    p = {k: (np.asarray(v, np.float32).astype(np.float64) if k != "cell" else v)
         for k, v in p.items()}
    F = [np.asarray(0.3 * rng.standard_normal((6, cfg.nz, cfg.ny)), np.float32).astype(np.float64)
         for _ in range(2)]
    return p, F[0], F[1]


# FP32 against FP32 in another order and with other reciprocals: a few ulp in
# the momenta, times the move (up to 8 cells here) in the positions; a deposit
# node is a sum of up to 1200 terms of one sign per particle
TOL = {"fp32": (4e-6, 2e-5, 1e-5), "fp64fft": (1e-13, 1e-12, 1e-12)}


@pytest.mark.parametrize("prec,ny,nz,hy", [("fp32", 32, 32, 0.2), ("fp32", 64, 8, 0.01),
                                           ("fp32", 96, 24, 0.2), ("fp32", 96, 40, 0.01),
                                           ("fp64fft", 64, 32, 0.2), ("fp64fft", 32, 64, 0.01)])
def test_row_push_edges(oracle_lib, prec, ny, nz, hy):
    from tertia_b200.mesh import Mesh
    cfg = cfg_for(prec, n=32, layers=4, shape=QS_SHAPE_CIC)
    cfg.ny, cfg.nz, cfg.hy, cfg.hz = ny, nz, hy, hy
    p, P, C = crowd(cfg, ny + nz)
    tp, tx, td = TOL[prec]
    dt = np.float32 if prec == "fp32" else np.float64
    for full in (0, 1):
        with Mesh(cfg) as m:
            m.load_front_plasma(p)
            for c in range(6):
                m.set_layer(QS_LAYER_P, c, P[c])
                m.set_layer(QS_LAYER_C, c, C[c])
            m.move_particles_layer(0, 0, full)
            q = m.get_plasma()
            dep = np.stack([m.get_layer(QS_LAYER_C, f) for f in (QS_F_JX, QS_F_JY, QS_F_JZ)])
            sums = None
            if full:   # two more pushes: the second one is counted and regrouped before the third
                m.move_particles_layer(0, 0, 1)
                m.move_particles_layer(0, 0, 0)
                m.sync()
                sums = m.get_plasma()["w"]
        a = {k: (np.asarray(v, dt) if k != "cell" else v) for k, v in p.items()}
        r = oracle_lib.push_layer(cfg, a["cell"], a["y"], a["z"], a["px"], a["py"], a["pz"], a["w"],
                                  P.astype(dt), C.astype(dt), full=bool(full), precise=True,
                                  dtype=dt)
        for k in ("px", "py", "pz"):
            np.testing.assert_allclose(q[k], r[k], rtol=tp, atol=tp)
        for axis, at, size in (("y", lambda c: c % ny, ny), ("z", lambda c: c // ny, nz)):
            d = (at(q["cell"]) + q[axis]) - (at(np.asarray(r["cell"])) + np.asarray(r[axis], float))
            d -= size * np.round(d / size)   # periodic
            assert np.max(np.abs(d)) < tx, axis
        assert rel_l2(dep, np.asarray(r["dep"], float)[:3]) < td
        if sums is not None:   # each particle keeps its own weight through the regrouping
            np.testing.assert_array_equal(sums, p["w"])


# the second push starts from the first one's positions, TOL's tx off at most:
# so are its weights, and a node's sum is off by about as much relative to it
TOL2 = {"fp32": 1e-4, "fp64fft": 1e-11}


@pytest.mark.parametrize("prec,ny,nz,hy", [("fp32", 32, 32, 0.2), ("fp32", 64, 8, 0.01),
                                           ("fp32", 96, 24, 0.2), ("fp32", 96, 40, 0.01),
                                           ("fp64fft", 64, 32, 0.2), ("fp64fft", 32, 64, 0.01)])
def test_row_push_after_a_move(oracle_lib, prec, ny, nz, hy):
    """Particles that left the cell they are grouped by: into the cells around
    their tile, across the periodic edges and further."""
    from tertia_b200.mesh import Mesh
    cfg = cfg_for(prec, n=32, layers=4, shape=QS_SHAPE_CIC)
    cfg.ny, cfg.nz, cfg.hy, cfg.hz = ny, nz, hy, hy
    p, P, C = crowd(cfg, 3 * ny + nz)
    dt = np.float32 if prec == "fp32" else np.float64
    with Mesh(cfg) as m:
        m.load_front_plasma(p)
        for c in range(6):
            m.set_layer(QS_LAYER_P, c, P[c])
            m.set_layer(QS_LAYER_C, c, C[c])
        m.move_particles_layer(0, 0, 1)
        m.move_particles_layer(0, 0, 0)
        dep = np.stack([m.get_layer(QS_LAYER_C, f) for f in (QS_F_JX, QS_F_JY, QS_F_JZ)])
    r = {k: (np.asarray(v, dt) if k != "cell" else v) for k, v in p.items()}
    w = r["w"]
    for full in (True, False):
        r = oracle_lib.push_layer(cfg, r["cell"], r["y"], r["z"], r["px"], r["py"], r["pz"], w,
                                  P.astype(dt), C.astype(dt), full=full, precise=True, dtype=dt)
    assert np.mean(np.asarray(r["cell"]) != p["cell"]) > 0.05
    assert rel_l2(dep, np.asarray(r["dep"], float)[:3]) < TOL2[prec]
