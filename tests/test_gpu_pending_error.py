"""Errors of the runtime that a step, a getter or a new bed has nothing to do
with: one that an earlier call reported leaves nothing behind, one of the
program's own is neither reported nor consumed."""
import ctypes

import numpy as np
import pytest

from swe_fvm_gb300 import Fluxes, SpaceDisc, SweError, scenarios
from swe_fvm_gb300.adjoint import Rollout

pytestmark = pytest.mark.gpu


def test_goes_on_after_a_tape_that_does_not_fit(gpu):
    m, prim = scenarios.random_front_case(12, seed=1)
    ro, ref = Rollout(m, prim), Rollout(m, prim)
    n = 1 << 40  # 8 TB of recorded time steps
    with pytest.raises(SweError):
        ro.forward(1, n, n, np.zeros(0, dtype=np.int64), n)
    for r in (ro, ref):
        r.sd.run(1, 1e-4, 2)
    assert np.array_equal(ro.sd.GetVolField(), ref.sd.GetVolField())


def test_error_of_the_program(gpu):
    rt = ctypes.CDLL("libcudart.so.13")
    m, prim = scenarios.random_front_case(12, seed=1)
    sd, ref = (SpaceDisc(Fluxes.HLLC(), m, prim) for _ in range(2))
    for s in (sd, ref):
        s.run(1, 1e-4, 1)  # (the step's graph exists)
        s.SetVolField(prim)
    p = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(1 << 60)) == 2  # out of memory
    got = []
    for s in (sd, ref):
        s.run(1, 1e-4, 2)
        got.append((s.GetEdgField(), s.GetFluxes(), s.GetNodeMax()))
        s.set_bathymetry(m.geometry[:, 2])
        pending = rt.cudaPeekAtLastError()
        if s is sd:
            assert pending == 2
            rt.cudaGetLastError()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert np.array_equal(sd.GetVolField(), ref.GetVolField())
