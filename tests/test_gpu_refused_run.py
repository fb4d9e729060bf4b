"""A run that the runtime refuses (its stream is being captured by the caller)
leaves the context as it was: the interface values, the state and the CFL ratio
stay, and the next call goes through."""
import numpy as np
import pytest

from swe_fvm_gb300 import Fluxes, SpaceDisc, SweError, scenarios

pytestmark = pytest.mark.gpu


def refused(torch, sd, stream, call):
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(RuntimeError):  # the capture is broken off
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            with pytest.raises(SweError):
                call(sd)


@pytest.mark.parametrize("primed", [True, False])
@pytest.mark.parametrize("scheme", [0, 1, 2])
def test_context_is_as_before(gpu, scheme, primed):
    import torch

    m, prim = scenarios.random_front_case(16, seed=3)
    sd, ref = (SpaceDisc(Fluxes.HLLC(), m, prim) for _ in range(2))
    stream = torch.cuda.Stream()
    sd.set_stream(stream.cuda_stream)
    other = prim.copy()
    other[:, 0] = np.maximum(m.centroids()[:, 2], prim[:, 0] - 0.03)
    other[other[:, 0] - m.centroids()[:, 2] <= 1e-12, 1:] = 0.0
    for s in (sd, ref):
        s.run(1, 1e-3, 2)
        s.run(scheme, 1e-3, 1)  # (its step graph exists)
        s.SetVolField(other)
        if primed:
            s.ComputeInterfaceValues()
            s.ComputeFluxes()
    sd.synchronize()
    refused(torch, sd, stream, lambda s: s.run(scheme, 1e-3, 1))
    # the first call after it steps
    for s in (sd, ref):
        s.run(scheme, 1e-4, 1)
    assert np.array_equal(sd.GetVolField(), ref.GetVolField())
    for s in (sd, ref):
        s.SetVolField(other)
        if primed:
            s.ComputeInterfaceValues()
            s.ComputeFluxes()
    sd.synchronize()
    refused(torch, sd, stream, lambda s: s.run(scheme, 1e-3, 1))
    assert np.array_equal(sd.GetEdgField(), ref.GetEdgField())
    assert np.array_equal(sd.GetSrcField(), ref.GetSrcField())
    assert np.array_equal(sd.GetFluxes(), ref.GetFluxes())
    assert sd.GetMinLenToWavespeed() == ref.GetMinLenToWavespeed()
    assert np.array_equal(sd.GetVolField(), ref.GetVolField())
