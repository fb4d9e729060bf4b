"""The backward pass's kept workspace and graphs: passes of changing shape on one
context (segment length, scheme, gauges, observation stride, regularisation,
step count, bed, custom scheme, stream) give what a fresh context gives."""
import numpy as np
import pytest

from swe_fvm_gb300 import scenarios
from swe_fvm_gb300.adjoint import Rollout
from swe_fvm_gb300.mesh import Mesh

pytestmark = pytest.mark.gpu


def passes(ro, scheme, steps, keep, gauges, every, depth, weight):
    ro.set_regularisation(depth)
    tr = ro.forward(scheme, steps, keep, gauges, every)
    return tr, ro.backward(weight * np.cos(np.arange(tr.size)).reshape(tr.shape))


def test_changing_shapes_equal_fresh_contexts(gpu):
    import torch

    m, prim = scenarios.random_front_case(14, seed=8)
    rng = np.random.default_rng(1)
    z = m.geometry[:, 2] + 0.005 * rng.random(m.num_nodes)
    m2 = Mesh(np.column_stack([m.geometry[:, :2], z]), m.edge_nodes, m.edge_cells, m.cell_nodes, m.cell_edges,
              m.cell_neighbours)
    prim2 = prim.copy()
    prim2[:, 0] = np.maximum(prim[:, 0], m2.centroids()[:, 2])
    base = Rollout(m, prim2)
    table = ([1.0, 0.5], [0.0, 0.5], [1.0, 0.5])
    g1, g2 = rng.integers(0, m.num_cells, 5), rng.integers(0, m.num_cells, 9)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    shapes = [(1, 8, 2, g1, 2, 1e-3, 1.0), (1, 8, 2, g1, 2, 1e-3, 2.0), (1, 8, 2, g1, 2, 1e-2, 1.0),
              (1, 9, 2, g1, 3, 1e-3, 1.0), (2, 6, 3, g1, 2, 1e-3, 1.0), (0, 6, 6, g2, 1, 1e-3, 1.0),
              (3, 8, 2, g2, 4, 1e-3, 1.0), (1, 12, 5, g2, 4, 1e-3, 1.0), (1, 8, 2, g1, 2, 1e-3, 1.0)]
    for q, shape in enumerate(shapes):
        bed, mesh = (m.geometry[:, 2], m) if q % 3 else (z, m2)
        base.sd.set_stream(streams[q % 2].cuda_stream)
        base.sd.set_bathymetry(bed)
        base.sd.SetVolField(prim2)
        base.sd.prime()
        fresh = Rollout(mesh, prim2)
        for ro in (base, fresh):
            ro.sd.set_scheme(*table)
        tr, (gp, gz) = passes(base, *shape)
        tf, (fp, fz) = passes(fresh, *shape)
        assert np.array_equal(tr, tf), q
        # (node sums are atomic: their order varies by rounding)
        assert np.allclose(gp, fp, rtol=1e-9, atol=1e-11 * np.abs(fp).max()), q
        assert np.allclose(gz, fz, rtol=1e-9, atol=1e-11 * np.abs(fz).max()), q
