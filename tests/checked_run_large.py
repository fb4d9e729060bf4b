"""Runs steps, getters, new beds and an adjoint pass on a mesh and a batch whose
products go through the integer pipe and whose part-wet lists are longer than the
lane groups take, and prints one JSON line of state digests; run once with the
product library and once with SWE_GB300_CHECKED=1 by test_gpu_checked_large."""
import json
import sys

import numpy as np

from checked_run import digest
from swe_fvm_gb300 import Batch, Fluxes, SpaceDisc, Wavespeeds, _lib, scenarios
from swe_fvm_gb300.adjoint import Rollout


def look(sd):
    return [digest(f()) for f in (sd.GetVolField, sd.GetEdgField, sd.GetSrcField, sd.GetFluxes, sd.GetNodeMax)]


def main():
    out = {"checked": _lib.checked(), "library": _lib.library_path()}
    rng = np.random.default_rng(0)
    m, prim = scenarios.random_front_case(160, 3)
    bc = m.centroids()[:, 2]
    thin = rng.random(m.num_cells) < 0.3
    prim[thin, 0] = bc[thin] + 10.0 ** rng.uniform(-11, -2, thin.sum())
    prim[prim[:, 0] - bc <= 1e-12, 1:] = 0.0
    z = m.geometry[:, 2] - 0.01 * rng.random(m.num_nodes)
    for reorder in ("keep", "morton"):
        for flux in (Fluxes.HLLC(Wavespeeds.Einfeldt), Fluxes.HLL(Wavespeeds.Davis)):
            for cor in (0.0, 0.5):
                sd = SpaceDisc(flux, m, prim, cor=cor, reorder=reorder)
                key = f"{reorder}/{flux.kind}{flux.wavespeed}/{cor}/"
                for scheme in (0, 1, 2):
                    sd.run(scheme, 1e-5, 3)
                    out[key + str(scheme)] = look(sd)
                sd.set_bathymetry(z)
                sd.prime()
                sd.run(1, 1e-5, 3)
                sd.synchronize()  # raises on any device error bit
                out[key + "bed"] = look(sd)
    small = [scenarios.random_front_case(n, n) for n in (100, 110, 3)]
    b = Batch([c[0] for c in small], [c[1] for c in small], Fluxes.HLLC(Wavespeeds.Einfeldt))
    b.run_cfl(1, 5)
    b.set_bathymetry([c[0].geometry[:, 2] - 0.01 for c in small])
    b.prime()
    b.run_cfl(2, 3)
    b.synchronize()
    out["batch"] = [digest(b.prim(q)) for q in range(len(small))]
    ro = Rollout(m, prim)
    tr = ro.forward(1, 6, 2, rng.integers(0, m.num_cells, 8), 2)
    gp, gz = ro.backward(np.ones_like(tr))
    ro.sd.synchronize()
    out["adjoint_traces"] = digest(tr)
    out["adjoint_grads"] = [float(np.abs(g).sum()) for g in (gp, gz)]
    print(json.dumps(out))
    return 0


if __name__ == "__main__":
    sys.exit(main())
