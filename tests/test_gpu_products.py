"""Meshes large enough to form their products on the integer pipe, with
operands inside its range, at its edges and outside (velocities down to the
subnormals, whose edges and cells are evaluated again with FP64 instructions):
bit for bit the oracle's, for both flux plugins, with and without Coriolis."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from swe_fvm_gb300 import Fluxes, Solvers, SpaceDisc, TimeDisc, Wavespeeds, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flux,cor", [("HLLC", 0.0), ("HLL", 0.0), ("HLLC", 0.4)])
def test_large_mesh_equals_oracle(gpu, flux, cor):
    m, prim = scenarios.random_front_case(146, seed=3)
    assert m.num_cells >= 40000
    rng = np.random.default_rng(1)
    wet = np.flatnonzero(prim[:, 0] - m.centroids()[:, 2] > 1e-12)
    for tiny in (0.0, 2.0 ** -511, 2.0 ** -512, 1e-200, 1e-300, 5e-324):
        some = rng.choice(wet, 600, replace=False)
        prim[some, 1:] = tiny * rng.choice([-1.0, 1.0], (600, 2))
    o = Oracle(m, prim, flux=flux, cor=cor)
    sd = SpaceDisc(getattr(Fluxes, flux)(Wavespeeds.Einfeldt), m, prim, cor=cor)
    td = TimeDisc(sd)
    o.compute_interface_values()
    o.compute_fluxes()
    for _ in range(2):
        dt = 0.15 * o.min_len_to_wavespeed()
        assert td.CFLdt() == dt
        o.step("SSPRK2", dt)
        Solvers.SSPRK2(td, dt)
        assert np.array_equal(sd.GetVolField(), o.prim())
    assert np.array_equal(sd.GetFluxes(), o.edge_fields()[2])
