"""A new bed leaves the interface values and source slots of the last
reconstruction as they are, whatever scheme ran before it; the flux pass reads
them."""
import numpy as np
import pytest

from swe_fvm_gb300 import Fluxes, SpaceDisc, scenarios

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cor", [0.0, 0.7])
@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_interface_values_outlast_a_new_bed(gpu, scheme, cor):
    m, prim = scenarios.random_front_case(20, seed=4)
    # (lower everywhere: no depth at the old interface values turns negative)
    z = m.geometry[:, 2] - 0.05 * np.random.default_rng(2).random(m.num_nodes)
    sd, ref = (SpaceDisc(Fluxes.HLLC(), m, prim, cor=cor) for _ in range(2))
    for s in (sd, ref):
        s.run(scheme, 2e-3, 3)
    edg, src = ref.GetEdgField(), ref.GetSrcField()  # made before the bed changes
    for s in (sd, ref):
        s.set_bathymetry(z)
    assert np.array_equal(sd.GetEdgField(), edg)
    assert np.array_equal(sd.GetSrcField(), src)
    # (again, for values that nothing asked for before the flux pass)
    other = SpaceDisc(Fluxes.HLLC(), m, prim, cor=cor)
    other.run(scheme, 2e-3, 3)
    other.set_bathymetry(z)
    for s in (other, ref):
        s.ComputeFluxes()
    assert np.array_equal(other.GetFluxes(), ref.GetFluxes())
    # and the run goes on alike from a new state
    prim2 = prim.copy()
    prim2[:, 0] = np.maximum(prim[:, 0], z[m.cell_nodes].max(axis=1))
    for s in (sd, ref, other):
        s.SetVolField(prim2)
        s.run(scheme, 1e-3, 2)
    assert np.array_equal(sd.GetVolField(), ref.GetVolField())
    assert np.array_equal(other.GetVolField(), ref.GetVolField())
