"""Taped run and reverse on meshes with an odd number of cells (one triangle,
three, a lattice with one cell cut off): the kept intermediates stay aligned,
and the gradient is the finite difference's."""
import numpy as np
import pytest

from swe_fvm_gb300.adjoint import BatchRollout, Rollout
from swe_fvm_gb300.mesh import build_topology, jittered_delaunay

pytestmark = pytest.mark.gpu


def mesh(cells):
    xyz, tri = jittered_delaunay(9, 4)
    tri = tri[: cells or (len(tri) - 1 + len(tri) % 2)]
    used = np.unique(tri)
    new = np.zeros(len(xyz), dtype=np.int64)
    new[used] = np.arange(used.size)
    xyz = xyz[used]
    xyz[:, 2] = 0.05 * xyz[:, 0] + 0.03 * xyz[:, 1] ** 2
    m = build_topology(xyz, new[tri])
    assert m.num_cells % 2 == 1
    prim = np.zeros((m.num_cells, 3))
    c = m.centroids()
    prim[:, 0] = 0.4 + 0.05 * np.sin(5 * c[:, 0]) * np.cos(4 * c[:, 1])
    prim[:, 1:] = [0.04, -0.03]
    return m, prim


@pytest.mark.parametrize("cells", [1, 3, 0])
def test_odd_cells(gpu, cells):
    m, prim = mesh(cells)
    g = np.array([0, m.num_cells // 2])
    ro = Rollout(m, prim)
    tr = ro.forward(1, 6, 2, g, 3)
    gp, gz = ro.backward(np.ones_like(tr))
    assert np.isfinite(gp).all() and np.isfinite(gz).all()
    dts = ro.dts(6)
    d = np.zeros_like(prim)
    i = m.num_cells // 2
    d[i, 0] = 1e-6
    traces = []
    for s in (1.0, -1.0):
        ro.sd.SetVolField(prim + s * d)
        traces.append(ro.sd.run_traces(1, dts, g, 3).sum())
    fd = (traces[0] - traces[1]) / 2e-6
    assert gp[i, 0] == pytest.approx(fd, rel=1e-5, abs=1e-8)


def test_odd_batch(gpu):
    cases = [mesh(3), mesh(1), mesh(0)]
    g = [np.array([0]) for _ in cases]
    br = BatchRollout([m for m, _ in cases], [p for _, p in cases])
    tr = br.forward(1, 4, 2, g, 2)
    grads = br.backward([np.ones_like(t) for t in tr])
    for (m, p), (gp, gz), gq, t in zip(cases, grads, g, tr):
        ro = Rollout(m, p)
        assert np.array_equal(ro.forward(1, 4, 2, gq, 2), t)
        gp1, gz1 = ro.backward(np.ones_like(t))
        assert np.allclose(gp, gp1, rtol=1e-12, atol=1e-14) and np.allclose(gz, gz1, rtol=1e-12, atol=1e-14)
