"""The full interface values after steps: a step of several stages leaves the
depths only, and the getters make the rest from the last stage's input.  They
equal the oracle's (which holds the last stage's) bit for bit, also after the
state was replaced, and making them leaves the state, the fluxes and the CFL
ratio alone."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from swe_fvm_gb300 import Fluxes, Solvers, SpaceDisc, TimeDisc, Wavespeeds, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cor", [0.0, 0.7])
@pytest.mark.parametrize("scheme", ["Euler", "SSPRK2", "SSPRK3"])
def test_interface_values_after_steps(gpu, scheme, cor):
    m, prim = scenarios.random_front_case(20, seed=4)
    o = Oracle(m, prim, cor=cor)
    sd = SpaceDisc(Fluxes.HLLC(Wavespeeds.Einfeldt), m, prim, cor=cor)
    td = TimeDisc(sd)
    for _ in range(3):
        o.step(scheme, 2e-3)
        getattr(Solvers, scheme)(td, 2e-3)
    edg, src, f, _ = o.edge_fields()
    ratio = sd.GetMinLenToWavespeed()
    sd.SetVolField(prim)
    assert np.array_equal(sd.GetEdgField(), edg)
    assert np.array_equal(sd.GetSrcField()[:, 1:], src[:, 1:])
    assert np.array_equal(sd.GetFluxes(), f)
    assert sd.GetMinLenToWavespeed() == ratio == o.min_len_to_wavespeed()
    assert np.array_equal(sd.GetVolField(), prim)
    # the run continues from the replaced state as one that never looked
    other = SpaceDisc(Fluxes.HLLC(Wavespeeds.Einfeldt), m, prim, cor=cor)
    for s in (sd, other):
        t = TimeDisc(s)
        for _ in range(2):
            getattr(Solvers, scheme)(t, 2e-3)
    assert np.array_equal(sd.GetVolField(), other.GetVolField())


def test_fluxes_from_the_last_interface_values(gpu):
    """ComputeFluxes reads the interface values there are, not the state set since."""
    m, prim = scenarios.random_front_case(20, seed=4)
    sd = SpaceDisc(Fluxes.HLL(Wavespeeds.Davis), m, prim)
    Solvers.SSPRK2(TimeDisc(sd), 2e-3)
    inner = m.edge_cells[:, 1] >= 0
    f = sd.GetFluxes()[inner]
    sd.SetVolField(np.tile([9.0, 0.0, 0.0], (m.num_cells, 1)))
    sd.ComputeFluxes()
    assert np.array_equal(sd.GetFluxes()[inner], f)
