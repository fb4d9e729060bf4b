"""The bathymetry-dependent records computed on the device: after a new bed the
interface values, fluxes and steps equal the oracle's on that bed, bit for bit,
on meshes from two cells (all walls) up and beds with flat cells, equal nodes
and steep faces."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from swe_fvm_gb300 import Fluxes, Solvers, SpaceDisc, TimeDisc
from swe_fvm_gb300.mesh import Mesh, build_topology, jittered_delaunay, structured_square

pytestmark = pytest.mark.gpu

MESHES = {"square1": lambda: structured_square(1, 0.0, 1.0), "square3": lambda: structured_square(3, -1.0, 2.0),
          "square8": lambda: structured_square(8, 0.0, 1.0),
          "delaunay14": lambda: build_topology(*jittered_delaunay(14, 3))}


def beds(mesh, rng):
    x, y = mesh.geometry[:, 0], mesh.geometry[:, 1]
    n = x.size
    yield np.zeros(n)
    yield np.where(x > x.mean(), 0.25, 0.0)  # flat cells either side of a step
    yield np.round(4 * rng.random(n)) / 8.0  # many equal nodes
    yield 0.3 * rng.random(n) - 0.1


@pytest.mark.parametrize("name", list(MESHES))
def test_new_bed_equals_oracle(gpu, name):
    mesh = MESHES[name]()
    rng = np.random.default_rng(5)
    sd = SpaceDisc(Fluxes.HLLC(), mesh, np.tile([1.0, 0.0, 0.0], (mesh.num_cells, 1)))
    for z in beds(mesh, rng):
        g = mesh.geometry.copy()
        g[:, 2] = z
        m = Mesh(g, mesh.edge_nodes, mesh.edge_cells, mesh.cell_nodes, mesh.cell_edges, mesh.cell_neighbours)
        bc = m.centroids()[:, 2]
        w = np.maximum(bc, 0.12 + 0.1 * rng.random(m.num_cells))
        prim = np.stack([w, 0.1 * rng.standard_normal(w.size), 0.1 * rng.standard_normal(w.size)], 1)
        prim[w - bc <= 1e-12, 1:] = 0.0
        o = Oracle(m, prim)
        sd.set_bathymetry(z)
        sd.SetVolField(prim)
        o.compute_interface_values()
        o.compute_fluxes()
        sd.ComputeInterfaceValues()
        sd.ComputeFluxes()
        edg, src, f, mx = o.edge_fields()
        assert np.array_equal(sd.GetEdgField(), edg)
        assert np.array_equal(sd.GetSrcField()[:, 1:], src[:, 1:])
        assert np.array_equal(sd.GetNodeMax(), mx)
        assert np.array_equal(sd.GetFluxes(), f)
        td = TimeDisc(sd)
        for _ in range(3):
            dt = 0.15 * o.min_len_to_wavespeed()
            o.step("SSPRK2", dt)
            Solvers.SSPRK2(td, dt)
            assert np.array_equal(sd.GetVolField(), o.prim())
