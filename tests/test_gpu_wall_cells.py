"""Wet wall cells that stand above their vertices, below and above the size from
which they are listed: the interface values of a state and the step from the list
that making them left, bit for bit the oracle's and those of a step that lists
its cells itself."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from swe_fvm_gb300 import Fluxes, Solvers, SpaceDisc, TimeDisc, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["Euler", "SSPRK2"])
@pytest.mark.parametrize("basin", [True, False])
@pytest.mark.parametrize("lattice", [3, 16, 150])
def test_wall_cells(gpu, lattice, basin, scheme):
    m, prim = scenarios.random_front_case(lattice, seed=7)
    if basin:  # wet everywhere: its rim is all that is partially wet
        prim[:, 0] = 1.0 + 0.01 * np.random.default_rng(1).random(m.num_cells)
    o = Oracle(m, prim)
    o.compute_interface_values()
    o.compute_fluxes()
    edg, src, f, mx = o.edge_fields()
    sd, other = (SpaceDisc(Fluxes.HLLC(), m, prim) for _ in range(2))
    for s in (sd, other):
        s.SetVolField(prim)
    sd.ComputeInterfaceValues()
    assert np.array_equal(sd.GetNodeMax(), mx)
    sd.ComputeFluxes()
    assert np.array_equal(sd.GetEdgField(), edg)
    assert np.array_equal(sd.GetSrcField()[:, 1:], src[:, 1:])
    assert np.array_equal(sd.GetFluxes(), f)
    o.step(scheme, 1e-4)
    for s in (sd, other):
        getattr(Solvers, scheme)(TimeDisc(s), 1e-4)
        assert np.array_equal(s.GetVolField(), o.prim())
    sd.prime()  # a list from the priming pass too
    o.step(scheme, 1e-4)
    getattr(Solvers, scheme)(TimeDisc(sd), 1e-4)
    assert np.array_equal(sd.GetVolField(), o.prim())
