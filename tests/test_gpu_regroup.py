"""The counting sort that regroups the plasma by cell every few full pushes of
the grouped CIC push, around an adjoint that recomputes from its checkpoints."""
import numpy as np
import pytest

from tertia_b200 import workload as wl
from tertia_b200.abi import PRECISIONS, QS_SHAPE_CIC

pytestmark = pytest.mark.gpu


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
