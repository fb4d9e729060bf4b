"""A caller's own CUDA graph over the state upload, the reconstruction or the
flux pass: its replays change what the next call starts from without a call, and
the steps, the interface values and the fluxes follow."""
import numpy as np
import pytest

from swe_fvm_gb300 import Fluxes, SpaceDisc, scenarios

pytestmark = pytest.mark.gpu


def contexts(torch):
    m, prim = scenarios.random_front_case(16, seed=3)
    sd, ref = SpaceDisc(Fluxes.HLLC(), m, prim), SpaceDisc(Fluxes.HLLC(), m, prim)
    stream = torch.cuda.Stream()
    sd.set_stream(stream.cuda_stream)
    sd.run(1, 1e-3, 2)
    ref.run(1, 1e-3, 2)
    sd.synchronize()
    return m, prim, sd, ref, stream


def test_replayed_upload(gpu):
    import torch

    m, prim, sd, ref, stream = contexts(torch)
    rng = np.random.default_rng(0)
    buf = torch.empty((m.num_cells, 3), dtype=torch.float64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sd.set_prim_device(buf.data_ptr())
    bc = m.centroids()[:, 2]
    for scale in (0.0, 0.05, 0.1):  # other cells partly wet each time
        p = prim.copy()
        p[:, 0] = np.maximum(bc, prim[:, 0] - scale * rng.random(m.num_cells))
        p[p[:, 0] - bc <= 1e-12, 1:] = 0.0
        buf.copy_(torch.as_tensor(p))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        ref.SetVolField(p)
        for s in (sd, ref):
            s.run(1, 1e-4, 2)
        assert np.array_equal(sd.GetVolField(), ref.GetVolField())
        assert np.array_equal(sd.GetEdgField(), ref.GetEdgField())


def test_replayed_reconstruction(gpu):
    import torch

    m, prim, sd, ref, stream = contexts(torch)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sd.ComputeInterfaceValues()
    for scheme in (1, 0, 2):
        for s in (sd, ref):
            s.run(scheme, 1e-4, 2)
        assert np.array_equal(sd.GetSrcField(), ref.GetSrcField())
        with torch.cuda.stream(stream):
            graph.replay()
        ref.ComputeInterfaceValues()
        assert np.array_equal(sd.GetEdgField(), ref.GetEdgField())
        for s in (sd, ref):
            s.ComputeFluxes()
        assert np.array_equal(sd.GetFluxes(), ref.GetFluxes())
    for s in (sd, ref):
        s.run(1, 1e-4, 1)
    assert np.array_equal(sd.GetVolField(), ref.GetVolField())


@pytest.mark.parametrize("first", [0, 1])  # interface values left by the last stage, or made when asked for
def test_replayed_fluxes(gpu, first):
    import torch

    m, prim, sd, ref, stream = contexts(torch)
    for s in (sd, ref):
        s.run(first, 1e-4, 2)
    sd.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sd.ComputeFluxes()
    for scheme in (None, 1, 0, 2):
        for primed in (False, True):
            for s in (sd, ref):
                if scheme is not None:
                    s.run(scheme, 1e-4, 2)
                if primed:
                    s.ComputeInterfaceValues()
            with torch.cuda.stream(stream):
                graph.replay()
            ref.ComputeFluxes()
            assert np.array_equal(sd.GetFluxes(), ref.GetFluxes())
            assert np.array_equal(sd.GetEdgField(), ref.GetEdgField())
    for s in (sd, ref):
        s.run(1, 1e-4, 1)
    assert np.array_equal(sd.GetVolField(), ref.GetVolField())
