"""Partially-wet cells: their list (left by the update, or made anew for a new
state or bed) and the kernels over it, with 8 lanes a cell or one, on meshes of
a few listed cells up to lists too long for the groups: bit for bit the oracle's."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from swe_fvm_gb300 import Batch, Fluxes, Solvers, SpaceDisc, TimeDisc, Wavespeeds, scenarios
from swe_fvm_gb300.adjoint import Rollout

pytestmark = pytest.mark.gpu


def films(m, rng, share):
    """Thin films and moving water over the mesh's bed."""
    bc = m.centroids()[:, 2]
    w = np.maximum(bc, 0.15 + 0.05 * rng.random())
    thin = rng.random(m.num_cells) < share
    w[thin] = bc[thin] + 10.0 ** rng.uniform(-11, -2, thin.sum())
    prim = np.stack([w, 0.1 * rng.standard_normal(w.size), 0.1 * rng.standard_normal(w.size)], 1)
    prim[w - bc <= 1e-12, 1:] = 0.0
    return prim


def follow(sd, o, scheme, steps, dt):
    td = TimeDisc(sd)
    for _ in range(steps):
        o.step(scheme, dt)
        getattr(Solvers, scheme)(td, dt)
    assert np.array_equal(sd.GetVolField(), o.prim())


@pytest.mark.parametrize("lattice,share", [(4, 0.3), (5, 0.5), (7, 0.2), (9, 1.0), (12, 0.1), (30, 0.6), (190, 0.25)])
def test_lists_of_every_length(gpu, lattice, share):
    """190 lists more cells than the groups take (8000)."""
    rng = np.random.default_rng(lattice)
    m, _ = scenarios.random_front_case(lattice, seed=lattice)
    sd = SpaceDisc(Fluxes.HLLC(Wavespeeds.Einfeldt), m, films(m, rng, share))
    for scheme in ("SSPRK2", "Euler", "SSPRK3"):
        prim = films(m, rng, share)
        o = Oracle(m, prim)
        sd.SetVolField(prim)
        follow(sd, o, scheme, 2, 1e-4)


def test_list_follows_the_state(gpu):
    """Steps after every way to change or look at the state in between."""
    rng = np.random.default_rng(2)
    m, prim = scenarios.random_front_case(16, seed=6)
    ro = Rollout(m, prim)
    sd = ro.sd
    o = Oracle(m, prim)
    follow(sd, o, "SSPRK2", 2, 1e-3)
    sd.ComputeInterfaceValues()
    sd.ComputeInterfaceValues()
    follow(sd, o, "SSPRK2", 1, 1e-3)
    sd.GetEdgField()
    follow(sd, o, "SSPRK3", 1, 1e-3)
    prim = films(m, rng, 0.3)
    o = Oracle(m, prim)
    sd.SetVolField(prim)
    follow(sd, o, "Euler", 1, 1e-3)
    gauges = np.arange(4)
    traces = ro.forward(1, 4, 2, gauges, 2)
    ro.backward(np.ones_like(traces))
    state = sd.GetVolField()
    o = Oracle(m, state)
    follow(sd, o, "SSPRK2", 2, 1e-3)
    z = m.geometry[:, 2] + 0.01 * rng.random(m.num_nodes)
    m2 = type(m)(np.column_stack([m.geometry[:, :2], z]), m.edge_nodes, m.edge_cells, m.cell_nodes, m.cell_edges,
                 m.cell_neighbours)
    prim = sd.GetVolField()
    prim[:, 0] = np.maximum(prim[:, 0], m2.centroids()[:, 2])
    sd.SetVolField(prim)
    sd.set_bathymetry(z)
    follow(sd, Oracle(m2, prim), "SSPRK2", 2, 1e-3)


def test_batch_list_follows_one_instance(gpu):
    """A new state in one instance of a batch."""
    rng = np.random.default_rng(3)
    meshes = [scenarios.random_front_case(n, seed=n)[0] for n in (6, 11, 14)]
    prims = [films(m, rng, 0.3) for m in meshes]
    b = Batch(meshes, prims, Fluxes.HLL(Wavespeeds.Davis))
    oracles = [Oracle(m, p, flux="HLL", wavespeed="Davis") for m, p in zip(meshes, prims)]

    def step():
        b.run(1, 1e-4, 2)
        for q, o in enumerate(oracles):
            o.step("SSPRK2", 1e-4)
            o.step("SSPRK2", 1e-4)
            assert np.array_equal(b.prim(q), o.prim())

    step()
    prims[1] = films(meshes[1], rng, 0.6)
    b.set_prim(1, prims[1])
    oracles[1] = Oracle(meshes[1], prims[1], flux="HLL", wavespeed="Davis")
    step()
