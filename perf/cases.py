"""What the performance of this framework is measured on.

Each case is one pass of work that a user's program does through the public
entry points: the reference driver's host loop on small meshes, CFL-stepped
runs whose state stays on the device, an ensemble of instances in one batch,
iterations of a gauge inversion (forward, gradient, new bed, forward), and the
diagnostic getters.  Sizes are those of the scenarios, the tests and the
benchmark: bowls of a few hundred cells, the 8192-cell Thacker bowl, coasts of
tens of thousands of cells, the dam break with about a million.

``exact`` restates the explicit step in plain torch, in 64 bits, from the mesh
arrays alone; its gradients come from torch's autograd.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from swe_fvm_gb300 import Batch, Fluxes, Solvers, SpaceDisc, TimeDisc, Wavespeeds
from swe_fvm_gb300.adjoint import batch_gauge_rollout, gauge_rollout
from swe_fvm_gb300.mesh import Mesh, build_topology, gaussian_bumps, jittered_delaunay, structured_square

SCHEMES = {"Euler": 0, "SSPRK2": 1, "SSPRK3": 2}


def listed():
    return [
        # The reference driver's own loop (dt = CFLdt(); step) on a bowl of its size, four steps between two
        # looks at the state: what an interactive or coupled program does; all latency.
        {"name": "driver_bowl_512", "kind": "driver", "scene": "bowl", "side": 16, "flux": "HLL", "speed": "Einfeldt",
         "scheme": "Euler", "cor": 0.0, "cfl": 0.15, "steps": 4},
        # The same loop on an irregular wet/dry mesh with Coriolis and the three-stage scheme.
        {"name": "driver_front_2k_coriolis", "kind": "driver", "scene": "front", "side": 33, "flux": "HLLC",
         "speed": "Davis", "scheme": "SSPRK3", "cor": 0.7, "cfl": 0.15, "steps": 3},
        # The Thacker bowl with its moving shoreline, the usual verification run, stepped on the device.
        {"name": "thacker_8192", "kind": "run", "scene": "thacker", "side": 64, "flux": "HLLC", "speed": "Einfeldt",
         "scheme": "SSPRK2", "cor": 0.0, "cfl": 0.4, "steps": 20},
        # A coast with films and emerging bumps, odd cell count, Coriolis: a regional model's ordinary size.
        {"name": "coast_25k_coriolis", "kind": "run", "scene": "front", "side": 113, "flux": "HLLC",
         "speed": "Rusanov", "scheme": "SSPRK3", "cor": 0.3, "cfl": 0.3, "steps": 10},
        # A dam break over bumps, ordinary size, the other flux plugin and one stage a step.
        {"name": "dam_72k_hll_euler", "kind": "run", "scene": "dam", "side": 191, "flux": "HLL", "speed": "Davis",
         "scheme": "Euler", "cor": 0.0, "cfl": 0.15, "steps": 20},
        # A coast of the size that whole estuaries have, water moving everywhere.
        {"name": "coast_250k", "kind": "run", "scene": "front", "side": 355, "flux": "HLLC", "speed": "Einfeldt",
         "scheme": "SSPRK2", "cor": 0.0, "cfl": 0.15, "steps": 8},
        # The benchmark's dam break, about a million cells: throughput.
        {"name": "dam_1m", "kind": "run", "scene": "dam", "side": 708, "flux": "HLLC", "speed": "Einfeldt",
         "scheme": "SSPRK2", "cor": 0.0, "cfl": 0.15, "steps": 8},
        # Many small basins stepped together, each with its own time step, as in Monte-Carlo studies.
        {"name": "ensemble_32", "kind": "ensemble", "count": 32, "low": 2000, "high": 16000, "flux": "HLLC",
         "speed": "Einfeldt", "scheme": "SSPRK2", "cfl": 0.4, "steps": 12},
        # One iteration of an offshore gauge inversion: traces, both gradients, the bed moved along its gradient,
        # traces again.
        {"name": "inversion_20k", "kind": "inversion", "side": 101, "gauges": 16, "steps": 40, "every": 10,
         "keep": 10, "cfl": 0.15},
        # The same for several basins with shores, batched.
        {"name": "inversions_6", "kind": "inversions", "count": 6, "low": 2000, "high": 9000, "gauges": 8,
         "steps": 20, "every": 5, "keep": 5, "cfl": 0.4},
        # Reconstruction, fluxes and every getter of one state, as a plotting or debugging program reads them.
        {"name": "fields_18k", "kind": "fields", "scene": "front", "side": 97, "flux": "HLLC", "speed": "Einfeldt",
         "cor": 0.2},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["driver", "run", "run", "run", "ensemble", "inversion", "inversions", "fields"])
    plugin = {"flux": rng.choice(["HLL", "HLLC", "HLLC"]), "speed": rng.choice(["Rusanov", "Davis", "Einfeldt"])}
    cor = rng.choice([0.0, 0.0, round(rng.uniform(0.1, 1.0), 2)])
    scheme = rng.choice(["Euler", "SSPRK2", "SSPRK2", "SSPRK3"])
    if kind == "driver":
        return {"kind": kind, "scene": rng.choice(["bowl", "front", "thacker", "dam"]), "side": _log_int(rng, 13, 60),
                **plugin, "scheme": scheme, "cor": cor, "cfl": 0.15, "steps": rng.randint(1, 6)}
    if kind == "run":
        side = _log_int(rng, 40, 480)
        return {"kind": kind, "scene": rng.choice(["front", "dam", "thacker"]), "side": side, **plugin,
                "scheme": scheme, "cor": cor, "cfl": rng.choice([0.15, 0.3]), "steps": rng.randint(3, 12)}
    if kind == "ensemble":
        low = _log_int(rng, 1000, 6000)
        return {"kind": kind, "count": rng.randint(3, 32), "low": low, "high": low * rng.randint(2, 4),
                "flux": plugin["flux"], "speed": plugin["speed"], "scheme": scheme, "cfl": rng.choice([0.15, 0.4]),
                "steps": rng.randint(3, 12)}
    if kind == "inversion":
        every = rng.randint(2, 8)
        return {"kind": kind, "side": _log_int(rng, 25, 110), "gauges": rng.randint(3, 40),
                "steps": every * rng.randint(2, 5), "every": every, "keep": rng.randint(3, 10), "cfl": 0.15}
    if kind == "inversions":
        every = rng.randint(2, 5)
        return {"kind": kind, "count": rng.randint(2, 6), "low": 1500, "high": _log_int(rng, 2500, 9000),
                "gauges": rng.randint(3, 12), "steps": every * rng.randint(2, 4), "every": every,
                "keep": rng.randint(3, 7), "cfl": 0.4}
    return {"kind": kind, "scene": rng.choice(["front", "dam"]), "side": _log_int(rng, 30, 110), **plugin, "cor": cor}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=80)
def _mesh(shape: str, side: int, variant: int = 0) -> Mesh:
    """A flat mesh: a program makes or reads its mesh once.  "square" is side x side squares of two triangles,
    "delaunay" a triangulated side x side lattice with moved points."""
    if shape == "square":
        return structured_square(side, -2.0, 2.0)
    return build_topology(*jittered_delaunay(side, 40 + variant))


def _with_bed(mesh: Mesh, z) -> Mesh:
    g = mesh.geometry.copy()
    g[:, 2] = z
    return Mesh(g, mesh.edge_nodes, mesh.edge_cells, mesh.cell_nodes, mesh.cell_edges, mesh.cell_neighbours)


def _scene(scene: str, side: int, seed: int):
    """(mesh with its bed, initial (w, u, v) per cell)."""
    rng = np.random.default_rng(seed)
    if scene in ("thacker", "bowl"):
        flat = _mesh("square", side)
        x, y = flat.geometry[:, 0], flat.geometry[:, 1]
        mesh = _with_bed(flat, 0.1 * (x * x + y * y))
        c = mesh.centroids()
        if scene == "thacker":  # a paraboloid of water in the bowl, its middle and curvature drawn
            mid, curve = rng.uniform(0.1, 0.18), rng.uniform(0.08, 0.14)
            w = c[:, 2] + np.maximum(0.0, mid - curve * (c[:, 0] ** 2 + c[:, 1] ** 2))
        else:  # a hump in a bowl full to the brim
            a, b = rng.uniform(-0.5, 0.5, 2)
            w = 1.0 + 0.2 * np.exp(-5.0 * ((c[:, 0] - a) ** 2 + (c[:, 1] - b) ** 2))
        prim = np.zeros((mesh.num_cells, 3))
        prim[:, 0] = w
        return mesh, prim
    flat = _mesh("delaunay", side)
    x, y = flat.geometry[:, 0], flat.geometry[:, 1]
    if scene == "dam":  # two levels over eight bumps, some of which stand out of the water
        z = gaussian_bumps(x, y, rng.uniform(0.05, 0.3, 8), rng.uniform(0.02, 0.1, 8), rng.uniform(0.0, 1.0, (8, 2)))
        mesh = _with_bed(flat, z)
        c = mesh.centroids()
        w = np.where(c[:, 0] < rng.uniform(0.25, 0.4), 0.5, 0.2)
    else:  # "front": a sloped shore with bumps, films and water that moves
        z = gaussian_bumps(x, y, rng.uniform(0.1, 0.4, 5), rng.uniform(0.05, 0.15, 5), rng.uniform(0.1, 0.9, (5, 2)))
        mesh = _with_bed(flat, z + 0.3 * np.maximum(0.0, x - 0.6))
        c = mesh.centroids()
        w = 0.15 + 0.1 * np.exp(-((c[:, 0] - 0.3) ** 2 + (c[:, 1] - rng.uniform(0.3, 0.7)) ** 2) / 0.02)
    w = np.maximum(w, c[:, 2])
    prim = np.zeros((mesh.num_cells, 3))
    if scene == "front":
        thin = rng.random(mesh.num_cells) < 0.02
        w[thin] = c[thin, 2] + rng.uniform(0.0, 2e-3, int(thin.sum()))
        wet = w - c[:, 2] > 1e-12
        kx, ky, ph = rng.uniform(4, 9), rng.uniform(4, 9), rng.uniform(0, 6)
        prim[wet, 1] = 0.2 * np.sin(kx * c[wet, 0] + ky * c[wet, 1] + ph)
        prim[wet, 2] = 0.2 * np.cos(ky * c[wet, 0] - kx * c[wet, 1] + ph)
    prim[:, 0] = w
    return mesh, prim


def _basins(case, seed):
    """The instances of an ensemble: still water with a hump over one to four bumps."""
    rng = np.random.default_rng(seed)
    sizes = np.exp(np.random.default_rng(7).uniform(math.log(case["low"]), math.log(case["high"]), case["count"]))
    out = []
    for q, cells in enumerate(sizes):
        flat = _mesh("delaunay", max(8, int(round(math.sqrt(cells / 2.0))) + 1), q)
        x, y = flat.geometry[:, 0], flat.geometry[:, 1]
        nb = int(rng.integers(1, 5))
        z = gaussian_bumps(x, y, rng.uniform(0.05, 0.3, nb), rng.uniform(0.02, 0.1, nb), rng.uniform(0, 1, (nb, 2)))
        mesh = _with_bed(flat, z)
        c = mesh.centroids()
        p, s = rng.uniform(0.2, 0.8, 2), rng.uniform(0.05, 0.2)
        w = 0.1 + rng.uniform(0.01, 0.2) * np.exp(-((c[:, 0] - p[0]) ** 2 + (c[:, 1] - p[1]) ** 2) / (2 * s * s))
        prim = np.zeros((mesh.num_cells, 3))
        prim[:, 0] = np.maximum(w, c[:, 2])
        out.append((mesh, prim))
    return out


def _offshore(case, seed):
    """A submerged sloped bed with a bump, a current and a hump; gauges and the traces they recorded."""
    rng = np.random.default_rng(seed)
    flat = _mesh("delaunay", case["side"])
    x, y = flat.geometry[:, 0], flat.geometry[:, 1]
    p = rng.uniform(0.3, 0.7, 4)
    z = 0.08 * x + 0.05 * y + 0.12 * np.exp(-((x - p[0]) ** 2 + (y - p[1]) ** 2) / (2 * 0.12 ** 2))
    mesh = _with_bed(flat, z)
    c = mesh.centroids()
    w = 0.5 + 0.04 * np.exp(-((c[:, 0] - p[2]) ** 2 + (c[:, 1] - p[3]) ** 2) / (2 * 0.1 ** 2))
    uv = np.tile([0.05, 0.03], (mesh.num_cells, 1))
    gauges = rng.integers(0, mesh.num_cells, case["gauges"])
    seen = 0.5 + 0.01 * rng.standard_normal((case["steps"] // case["every"], case["gauges"]))
    return flat, mesh, w, uv, z, gauges, seen


def _shores(case, seed):
    rng = np.random.default_rng(seed + 1)
    basins = _basins(case, seed)
    gauges = [rng.integers(0, m.num_cells, case["gauges"]) for m, _ in basins]
    seen = 0.1 + 0.01 * rng.standard_normal((case["steps"] // case["every"], case["gauges"] * case["count"]))
    return basins, gauges, seen


def _fluxer(case):
    return getattr(Fluxes, case["flux"])(getattr(Wavespeeds, case["speed"]))


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "stream": torch.cuda.Stream()}
    if kind in ("driver", "run", "fields"):
        mesh, prim = _scene(case["scene"], case["side"], seed)
        state["sd"] = SpaceDisc(_fluxer(case), mesh, prim, cor=case["cor"], cfl=case.get("cfl", 0.15))
        state["prim"] = prim if kind != "run" else _dev(prim)
    elif kind == "ensemble":
        basins = _basins(case, seed)
        state["batch"] = Batch([m for m, _ in basins], [p for _, p in basins], _fluxer(case), cfl=case["cfl"])
        state["prim"] = [_dev(p) for _, p in basins]
    elif kind == "inversion":
        flat, mesh, w, uv, z, gauges, seen = _offshore(case, seed)
        state.update(mesh=flat, w=_dev(w), uv=_dev(uv), z=_dev(z), gauges=gauges, seen=_dev(seen))
    else:
        basins, gauges, seen = _shores(case, seed)
        flat = [_mesh("delaunay", _lattice(m), q) for q, (m, _) in enumerate(basins)]
        state.update(mesh=flat, w=_dev(np.concatenate([p[:, 0] for _, p in basins])),
                     z=_dev(np.concatenate([m.geometry[:, 2] for m, _ in basins])), gauges=gauges, seen=_dev(seen))
    holder = state.get("sd") or state.get("batch")
    if holder is not None:
        holder.set_stream(state["stream"].cuda_stream)
    return state


def _lattice(mesh):
    return int(round(math.sqrt(mesh.num_nodes)))


def run(state):
    case, stream = state["case"], state["stream"]
    here = torch.cuda.current_stream()
    stream.wait_stream(here)
    with torch.cuda.stream(stream):
        out = _RUN[case["kind"]](state, case)
    here.wait_stream(stream)
    return out


def _run_driver(state, case):
    sd = state["sd"]
    sd.SetVolField(state["prim"])
    sd.prime()
    td, step = TimeDisc(sd), getattr(Solvers, case["scheme"])
    for _ in range(case["steps"]):
        step(td, td.CFLdt())
    return {"state": sd.GetVolField(), "ratio": sd.GetMinLenToWavespeed()}


def _run_run(state, case):
    sd = state["sd"]
    sd.set_prim_device(state["prim"].data_ptr())
    sd.prime()
    sd.set_time(0.0)
    t = sd.run_cfl(SCHEMES[case["scheme"]], case["steps"])
    out = torch.empty_like(state["prim"])
    sd.get_prim_device(out.data_ptr())
    return {"state": out, "time": t}


def _run_ensemble(state, case):
    b, prims = state["batch"], state["prim"]
    for q, p in enumerate(prims):
        b.set_prim_device(q, p.data_ptr())
    b.prime()
    b.run_cfl(SCHEMES[case["scheme"]], case["steps"])
    return {"state": np.concatenate([b.prim(q) for q in range(len(prims))])}


def _run_inversion(state, case):
    def traces(w, z):
        return gauge_rollout(w, z, state["mesh"], state["gauges"], case["steps"], case["every"], case["keep"],
                             uv0=state["uv"], cfl=case["cfl"])

    return _iteration(state, traces)


def _run_inversions(state, case):
    def traces(w, z):
        return batch_gauge_rollout(w, z, state["mesh"], state["gauges"], case["steps"], case["every"], case["keep"],
                                   cfl=case["cfl"])

    return _iteration(state, traces)


def _iteration(state, traces):
    w, z = state["w"].clone().requires_grad_(True), state["z"].clone().requires_grad_(True)
    first = traces(w, z)
    (0.5 * (first - state["seen"]).square().sum()).backward()
    with torch.no_grad():
        moved = z - 1e-3 * z.grad / z.grad.abs().max()
        second = traces(w, moved)
    return {"first": first.detach(), "grad_w": w.grad, "grad_z": z.grad, "second": second}


def _run_fields(state, case):
    sd = state["sd"]
    sd.SetVolField(state["prim"])
    sd.ComputeInterfaceValues()
    sd.ComputeFluxes()
    return {"edges": sd.GetEdgField(), "sources": sd.GetSrcField(), "fluxes": sd.GetFluxes(),
            "node_max": sd.GetNodeMax(), "ratio": sd.GetMinLenToWavespeed(), "integrals": sd.integrals()}


_RUN = {"driver": _run_driver, "run": _run_run, "ensemble": _run_ensemble, "inversion": _run_inversion,
        "inversions": _run_inversions, "fields": _run_fields}


# -------------------------------------------------------------------- work
_STAGES = {"Euler": 1, "SSPRK2": 2, "SSPRK3": 3}


def _cells(case):
    """Cells of a case (a triangulated side x side lattice has about 2 (side - 1)^2)."""
    kind = case["kind"]
    if kind in ("ensemble", "inversions"):
        s = np.exp(np.random.default_rng(7).uniform(math.log(case["low"]), math.log(case["high"]), case["count"]))
        return int(sum(2 * max(7, int(round(math.sqrt(c / 2.0)))) ** 2 for c in s))
    if case.get("scene") in ("thacker", "bowl"):
        return 2 * case["side"] ** 2
    return 2 * (case["side"] - 1) ** 2


def work(case):
    """Bytes that cannot be done without: per cell and stage the state in and out (48), the six ids (24) and its
    share of the node coordinates (12); per step the step's first state once more (24); each state in and out.  An
    adjoint pass reads and writes the state and its adjoint over the same mesh, after one recomputed forward.
    flops: the flux (about 62 an edge), the update (about 73 a cell) and the reconstruction (about 13) of a stage."""
    c, kind = _cells(case), case["kind"]
    stage_bytes, stage_flops = 84.0 * c, (1.5 * 62 + 73 + 13) * c
    if kind == "fields":
        return {"bytes": c * (24.0 + 36 + 1.5 * (2 * 48 + 24) + 4), "flops": (1.5 * 62 + 13) * c}
    if kind in ("inversion", "inversions"):
        sweep = 2 * case["steps"]  # SSPRK2 stages; two forwards, a recomputed one, and the reverse at twice the work
        return {"bytes": 5 * (stage_bytes * sweep + 24.0 * c * case["steps"]), "flops": 5 * stage_flops * sweep}
    n = _STAGES[case["scheme"]] * case["steps"]
    return {"bytes": stage_bytes * n + 24.0 * c * (case["steps"] if n > case["steps"] else 0) + 48.0 * c,
            "flops": stage_flops * n}


# ------------------------------------------------------------------- exact
WET, TOL, CAPTURE = 1e-12, 1e-13, 1e-10


def _sel(c, a, b):
    return torch.where(c, a, b)


def _smin(a, b):
    return torch.where(b < a, b, a)


def _smax(a, b):
    return torch.where(a < b, b, a)


def _slope(p0, p1, p2):
    """Slope of the plane through three points (rows x, y, z), by elimination with the larger pivot."""
    a00, a01, b0 = p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2]
    a10, a11, b1 = p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2]
    sw = a00.abs() < a10.abs()
    a00, a10 = _sel(sw, a10, a00), _sel(sw, a00, a10)
    a01, a11 = _sel(sw, a11, a01), _sel(sw, a01, a11)
    b0, b1 = _sel(sw, b1, b0), _sel(sw, b0, b1)
    m = a10 / a00
    gy = (b1 - m * b0) / (a11 - m * a01)
    return (b0 - a01 * gy) / a00, gy


def _cubic_root(d, c, b, lo, hi):
    """The reference's bisection on x^3 + b x^2 + c x + d, whose iteration count follows the interval."""
    f = lambda x: x * x * x + b * x * x + c * x + d  # noqa: E731
    flo, fhi = f(lo), f(hi)
    same = torch.signbit(flo) == torch.signbit(fhi)
    ends = _sel(flo.abs() < fhi.abs(), lo, hi)
    mant, ex = torch.frexp((hi - lo).clamp_min(1e-300))
    ex = ex.to(torch.int64)
    n = 50 + torch.where(mant == 0.5, ex - 1, torch.where(ex >= 1, ex - 1, ex))
    x, neg = torch.zeros_like(d), torch.signbit(flo)
    a, z = lo.clone(), hi.clone()
    for it in range(int(n.max()) + 1 if n.numel() else 0):
        on = it <= n
        mid = 0.5 * (a + z)
        cut = torch.signbit(f(mid)) != neg
        x = _sel(on, mid, x)
        z, a = _sel(on & cut, mid, z), _sel(on & ~cut, mid, a)
    return _sel(same, ends, x)


class _Plain:
    """The explicit step in plain torch (float64), every read of a stage from its first state."""

    def __init__(self, mesh, z, case, device):
        ix = lambda a: torch.as_tensor(np.asarray(a), device=device)  # noqa: E731
        self.cn, self.ce, self.ct = ix(mesh.cell_nodes).T, ix(mesh.cell_edges).T, ix(mesh.cell_neighbours).T
        self.en, self.ec = ix(mesh.edge_nodes).T, ix(mesh.edge_cells).T
        self.hllc, self.speed, self.cor = case.get("flux", "HLLC") == "HLLC", case.get("speed", "Einfeldt"), case.get("cor", 0.0)
        geo = torch.as_tensor(mesh.geometry, device=device)
        self.x, self.y, self.z = geo[:, 0], geo[:, 1], z
        nodes = (self.x, self.y, self.z)
        self.P = [[c[self.cn[k]] for c in nodes] for k in range(3)]
        k3 = 1.0 / 3.0
        self.T = [self.P[0][r] * k3 + self.P[1][r] * k3 + self.P[2][r] * k3 for r in range(3)]
        self.E = [(c[self.en[0]] + c[self.en[1]]) * 0.5 for c in nodes]
        self.Ek = [[c[self.ce[k]] for c in self.E] for k in range(3)]
        dx, dy = (self.x[self.en[0]] - self.x[self.en[1]]), (self.y[self.en[0]] - self.y[self.en[1]])
        self.L = (dx * dx + dy * dy).sqrt()
        ba = [self.P[1][r] - self.P[0][r] for r in (0, 1)]
        ca = [self.P[2][r] - self.P[0][r] for r in (0, 1)]
        self.A = 0.5 * (ba[0] * ca[1] - ca[0] * ba[1]).abs()
        self.own, self.nb = self.ec[0], self.ec[1]
        self.inner = self.nb >= 0
        self.nbs = self.nb.clamp_min(0)
        self.tx, self.ty = self._tangent(torch.arange(self.L.numel(), device=device), self.own)
        self.nx, self.ny = self.ty, -self.tx
        self.mine = [self.own[self.ce[k]] == torch.arange(self.A.numel(), device=device) for k in range(3)]
        self.wall = [self.ct[k] < 0 for k in range(3)]
        self.nbr = [self.ct[k].clamp_min(0) for k in range(3)]
        bound = (self.nb[self.ce] < 0).any(0)
        top = _smax(_smax(self.P[0][2], self.P[1][2]), self.P[2][2])
        self.brim = _sel(bound, torch.full_like(top, math.inf), top)
        reach = [2.0 * self.A[c] / self.L for c in (self.own, self.nbs)]
        self.reach = _smin(reach[0], reach[1])
        # each edge's slot in its owner and in its neighbour: local index * cells + cell
        C = self.A.numel()
        self.slot = torch.zeros((2, self.L.numel()), dtype=torch.int64, device=device)
        for k in range(3):
            cells = torch.arange(C, device=device)
            for side, sel in ((0, self.mine[k]), (1, ~self.mine[k])):
                self.slot[side, self.ce[k][sel]] = k * C + cells[sel]
        self.dry = _slope(self.P[0], self.P[1], self.P[2])

    def _tangent(self, e, t):
        x0, y0 = self.x[self.en[0]][e], self.y[self.en[0]][e]
        tx = (self.x[self.en[1]][e] - x0) / self.L[e]
        ty = (self.y[self.en[1]][e] - y0) / self.L[e]
        flip = (self.T[0][t] - x0) * ty - tx * (self.T[1][t] - y0) > 0.0
        return _sel(flip, -tx, tx), _sel(flip, -ty, ty)

    def _assign(self, b, w, u, v):
        h = w - b
        wet, thin = h > WET, (h > WET) & (h < 1e-3)
        hs = _sel(thin, h, torch.ones_like(h))
        s = math.sqrt(2.0) * hs / (hs * hs + 1e-6).sqrt()
        u, v = _sel(thin, u * s, u), _sel(thin, v * s, v)
        zero = torch.zeros_like(h)
        return _sel(wet, w, b), _sel(wet, u, zero), _sel(wet, v, zero)

    def _planes(self, W, U, V):
        """(level, gx, gy, u, v) of every cell after the first pass, and which cells are partly wet."""
        C = self.A.numel()
        h = W - self.T[2]
        dry, full = ~(h > WET), self.brim < W
        full = full & ~dry
        part = ~dry & ~full
        near_dry = torch.zeros(C, dtype=torch.bool, device=W.device)
        pts = []
        for k in range(3):
            j = self.nbr[k]
            far = full[j]
            near_dry = near_dry | (~far & dry[j])
            # (cells that take no such plane get their own corners, so that every slope is finite)
            pts.append([_sel(full, _sel(far, self.T[r][j], self.Ek[k][r]), self.P[k][r]) for r in range(3)])
        gx, gy = _slope(*pts)
        off = lambda p: gx * (p[0] - self.T[0]) + gy * (p[1] - self.T[1])  # noqa: E731
        third = 1.0 / 3.0
        hold = torch.ones(C, dtype=torch.bool, device=W.device)
        for k in range(3):
            m = [1.0 - third if q == k else -third for q in range(3)]
            d = [self.P[0][r] * m[0] + self.P[1][r] * m[1] + self.P[2][r] * m[2] for r in (0, 1)]
            hold = hold & (((gx * d[0] + gy * d[1]) + W) - self.P[k][2] > WET)
        tvd = torch.ones_like(hold)
        for k in range(3):
            ek, wj = W + off(self.Ek[k]), W[self.nbr[k]]
            tvd = tvd & (_smin(W, wj) <= ek) & (ek <= _smax(W, wj))
        keep = full & ~near_dry & hold & tvd
        zero = torch.zeros_like(W)
        level = _sel(dry, self.T[2], W)
        gx = _sel(dry, self.dry[0], _sel(keep, gx, zero))
        gy = _sel(dry, self.dry[1], _sel(keep, gy, zero))
        u, v = _sel(dry, zero, U), _sel(dry, zero, V)
        if bool(part.any()):
            i = part.nonzero()[:, 0]
            level = level.index_put((i,), self._level1(i, W[i]))
        return level, gx, gy, u, v, part

    def _level1(self, i, w):
        zs = torch.stack([self.P[k][2][i] for k in range(3)])
        b13, b23 = zs.max(0).values, zs.min(0).values
        b12 = 3.0 * self.T[2][i] - b23 - b13
        mid = b12 + (1.0 / 3.0) * (b13 - b12) * (b13 - b12) / (b13 - b23)
        h = w - self.T[2][i]
        low = 3.0 * h * (b13 - b23) * (b12 - b23)
        root = np.cbrt(low.detach().cpu().numpy().astype(np.longdouble)).astype(np.float64)
        cube = b23 + torch.as_tensor(root, device=w.device)
        d = (b13 - b23) * (3.0 * h * (b13 - b12) - b12 * (b12 + b23)) - b23 * b23 * b13
        c = 3.0 * (b12 * b13 + b13 * b23 - b12 * b23)
        two = _cubic_root(d, c, -3.0 * b13, b12, b13)
        return _sel(w >= b13, w, _sel(w <= mid, cube, two))

    def _part2(self, i, W, level, top):
        """Second pass over partly wet cells i: (level, gx, gy)."""
        P = [torch.stack([self.P[k][r][i] for k in range(3)]) for r in range(3)]
        o = torch.zeros((3, i.numel()), dtype=torch.int64, device=W.device)
        o[0], o[1], o[2] = 0, 1, 2
        for a in (0, 1, 0):
            sw = torch.gather(P[2], 0, o[a:a + 1])[0] > torch.gather(P[2], 0, o[a + 1:a + 2])[0]
            o[a], o[a + 1] = _sel(sw, o[a + 1], o[a]).clone(), _sel(sw, o[a], o[a + 1]).clone()
        p = [[torch.gather(P[r], 0, o[k:k + 1])[0] for r in range(3)] for k in range(3)]
        b23, b12, b13 = p[0][2], p[1][2], p[2][2]
        w, l1 = W[i], level[i]
        w23 = top[torch.gather(torch.stack([self.cn[k][i] for k in range(3)]), 0, o[0:1])[0]]
        h23, ratio = w23 - b23, (b12 - b23) / (b13 - b23)
        one, three = 1.0 / 3.0 * h23 * ratio, 1.0 / 3.0 * h23 * (2.0 * b13 - b12 - b23) / (b13 - b23)
        h = w - self.T[2][i]
        rh = h / h23
        k2, k3 = (3.0 * rh / ratio).sqrt(), (3.0 * rh * ratio).sqrt()
        alpha, beta = 3.0 * rh, (b13 - b12) / (b13 - b23)
        zero = torch.zeros_like(h)
        k1 = 1.0 - _cubic_root((1.0 + beta - alpha) / (beta * beta), (alpha - 3.0) / beta, zero, zero, zero + 1.0)
        is1 = h <= one
        is3 = ~is1 & (h >= three)
        q1 = [_sel(is1, k2 * p[1][r] + (1.0 - k2) * p[0][r], p[1][r]) for r in range(3)]
        two = [k1 * p[2][r] + (1.0 - k1) * p[1][r] for r in range(3)]
        two[2] = k1 * b13 + (1.0 - k1) * b12
        up = [p[2][0], p[2][1], p[2][2] + 1.5 * (h - three)]
        q2 = [_sel(is1, k3 * p[2][r] + (1.0 - k3) * p[0][r], _sel(is3, up[r], two[r])) for r in range(3)]
        gx, gy = _slope(p[0], q1, q2)
        lv = w23 + (gx * (self.T[0][i] - p[0][0]) + gy * (self.T[1][i] - p[0][1]))
        skip = (w > b13) | (b13 - b23 < TOL) | (~is1 & ~is3 & (k1 < TOL))
        return _sel(skip, l1, lv), _sel(skip, zero, gx), _sel(skip, zero, gy)

    def _at(self, plane, z, px, py):
        level, gx, gy = plane
        a = level + (gx * (px - self.T[0]) + gy * (py - self.T[1]))
        return _sel(a - z >= 0, a, z), a - z >= 0

    def _node_max(self, level, gx, gy):
        """Per node the highest first-pass value of the cells around it."""
        top = self.z.detach().clone()
        for k in range(3):
            a, _ = self._at((level, gx, gy), self.P[k][2], self.P[k][0], self.P[k][1])
            top = top.scatter_reduce(0, self.cn[k], a.detach(), "amax")
        return top

    def interface(self, W, U, V):
        """Per local edge the values (w, u, v) and the source gradient (x, y) of every cell."""
        level, gx, gy, u, v, part = self._planes(W, U, V)
        if bool(part.any()):
            i = part.nonzero()[:, 0]
            l2, x2, y2 = self._part2(i, W, level, self._node_max(level, gx, gy))
            level, gx, gy = level.index_put((i,), l2), gx.index_put((i,), x2), gy.index_put((i,), y2)
        ew, eu, ev, sx, sy = [], [], [], [], []
        for k in range(3):
            b = self.Ek[k][2]
            a, on = self._at((level, gx, gy), b, self.Ek[k][0], self.Ek[k][1])
            zero = torch.zeros_like(a)
            w_, u_, v_ = self._assign(b, a, _sel(on, u, zero), _sel(on, v, zero))
            ew.append(w_), eu.append(u_), ev.append(v_)
            sx.append(gx + self.cor * (-v_)), sy.append(gy + self.cor * u_)
        return ew, eu, ev, sx, sy

    def _elem(self, nx, ny, h, hu, hv):
        wet = h > WET
        hs = _sel(wet, h, torch.ones_like(h))
        q, zero = (hu * nx + hv * ny), torch.zeros_like(h)
        f = (q, (q / hs) * hu + (0.5 * h * h) * nx, (q / hs) * hv + (0.5 * h * h) * ny)
        return [_sel(wet, x, zero) for x in f]

    def fluxes(self, W, ew, eu, ev):
        """Per edge the three fluxes, and the least length-to-wavespeed ratio."""
        cat = [torch.cat(a) for a in (ew, eu, ev)]
        lw_, lu, lv = (c[self.slot[0]] for c in cat)
        rw, ru, rv = (c[self.slot[1]] for c in cat)
        b, nx, ny, tx, ty = self.E[2], self.nx, self.ny, self.tx, self.ty
        hl, hr = lw_ - b, rw - b
        go = self.inner & (hl + hr > CAPTURE)
        one = torch.ones_like(hl)
        hl, hr = _sel(go, hl, one), _sel(go, hr, one)
        ul, ur = lu * nx + lv * ny, ru * nx + rv * ny
        # sqrt with a zero slope at zero depth, for autograd
        root = lambda h: _sel(h > 0, _sel(h > 0, h, one).sqrt(), torch.zeros_like(h))  # noqa: E731
        cl, cr = root(hl), root(hr)
        if self.speed == "Rusanov":
            ap = _smax(ul.abs() + cl, ur.abs() + cr)
            a0, a1 = -ap, ap
        elif self.speed == "Davis":
            a0, a1 = _smin(ul - cl, ur - cr), _smax(ul + cl, ur + cr)
        else:
            roe, c = (cl * ul + cl * ur) / (cl + cr), (0.5 * (hl + hr)).sqrt()
            a0, a1 = _smin(ul - cl, roe - c), _smax(ur + cr, roe + c)
        zero = torch.zeros_like(hl)
        Ul, Ur = (hl, hl * lu, hl * lv), (hr, hr * ru, hr * rv)
        if self.hllc:
            A, B = hr * (a1 - ur), hl * (a0 - ul)
            us = (a1 - ur) * hr * ur - (a0 - ul) * hl * ul + 0.5 * (hl * hl - hr * hr)
            us = us / (A - B)
            speed = _smax(torch.full_like(a0, TOL), _smax(a0, a1))
            right = ~(us > 0.0)
            h, u, v = _sel(right, hr, hl), _sel(right, ru, lu), _sel(right, rv, lv)
            ax, hx = _sel(right, a1, a0), _sel(right, A, B)
            vt = u * tx + v * ty
            hs = hx / (ax - us)
            star = (hs, hs * (vt * tx + us * ty), hs * (vt * nx + us * ny))
            side = (h, h * u, h * v)
            s = _sel(right, _smax(zero, a1), _smin(zero, a0))
            F = [f + s * (p - q) for f, p, q in zip(self._elem(nx, ny, *side), star, side)]
        else:
            al, ar = _smin(zero, a0), _smax(zero, a1)
            go = go & (ar - al > CAPTURE)
            al, ar = _sel(go, al, -one), _sel(go, ar, one)
            speed = _smax(-al, ar)
            Fl, Fr = self._elem(nx, ny, *Ul), self._elem(nx, ny, *Ur)
            F = [(ar * fl - al * fr + (al * ar) * (q - p)) / (ar - al) for fl, fr, p, q in zip(Fl, Fr, Ul, Ur)]
        ratio = self.reach / (abs(self.cor) + speed)
        ratio = torch.where(go, ratio, torch.full_like(ratio, math.inf)).detach().min().clamp_max(1.0)
        ho = W[self.own] - self.T[2][self.own]
        wall = self._elem(nx, ny, ho, torch.zeros_like(ho), torch.zeros_like(ho))
        return [_sel(go, f, _sel(self.inner, zero, q)) for f, q in zip(F, wall)], ratio

    def stage(self, S, S0, a, b, dt):
        """One Shu-Osher stage: a S0 + b S + RHS(S, dt); a is None for S0 + RHS.  Returns (state, ratio)."""
        W, U, V = S
        ew, eu, ev, sx, sy = self.interface(W, U, V)
        F, ratio = self.fluxes(W, ew, eu, ev)
        h = W - self.T[2]
        wet = h > WET
        zero, inf = torch.zeros_like(h), torch.full_like(h, math.inf)
        out = zero
        for k in range(3):
            f = F[0][self.ce[k]]
            out = out + _smax(zero, _sel(self.mine[k], f, -f))
        runs = out > TOL
        drain = _sel(wet, _sel(runs, self.A * h / _sel(runs, out, torch.ones_like(out)), inf), zero)
        inv = 1.0 / self.A
        r = [zero, zero, zero]
        for k in range(3):
            e = self.ce[k]
            f = [x[e] for x in F]
            theirs = _sel(self.wall[k], inf, drain[self.nbr[k]])
            leaves = _sel(self.mine[k], f[0], -f[0]) > 0.0
            d = torch.full_like(h, float(dt)) if not torch.is_tensor(dt) else dt.expand_as(h)
            dk = _sel(leaves, _smin(d, drain), _smin(d, theirs))
            ck = inv * self.L[e]
            he = ew[k] - self.Ek[k][2]
            s = _sel(self.mine[k], dk, -dk) * ck
            r = [x - s * y for x, y in zip(r, f)]
            q = d * (1.0 / 3.0)
            nx, ny = _sel(self.mine[k], self.nx[e], -self.nx[e]), _sel(self.mine[k], self.ny[e], -self.ny[e])
            p = 0.5 * he * he
            r[1] = r[1] - q * sx[k] * he + dk * (nx * ck * p)
            r[2] = r[2] - q * sy[k] * he + dk * (ny * ck * p)
        cons = lambda s: (s[0] - self.T[2], (s[0] - self.T[2]) * s[1], (s[0] - self.T[2]) * s[2])  # noqa: E731
        if a is None:
            n = [x + y for x, y in zip(cons(S0), r)]
        else:
            n = [a * x + b * p + y for x, p, y in zip(cons(S0), cons(S), r)]
        wet, thin = n[0] > WET, (n[0] > WET) & (n[0] < 1e-3)
        hs = _sel(wet, n[0], torch.ones_like(h))
        ih = _sel(thin, math.sqrt(2.0) * hs / (hs * hs * hs * hs + 1e-12).sqrt(), 1.0 / hs)
        return [_sel(wet, n[0] + self.T[2], self.T[2]), _sel(wet, n[1] * ih, zero), _sel(wet, n[2] * ih, zero)], ratio

    def step(self, S, scheme, dt):
        S1, ratio = self.stage(S, S, None, None, dt)
        if scheme == "SSPRK2":
            S1, ratio = self.stage(S1, S, 0.5, 0.5, 0.5 * dt)
        elif scheme == "SSPRK3":
            S1, ratio = self.stage(S1, S, 0.75, 0.25, 0.25 * dt)
            S1, ratio = self.stage(S1, S, 1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0 * dt)
        return S1, ratio

    def cfl_steps(self, S, scheme, steps, cfl, look=None):
        """CFL-limited steps; look(step number, state) after each.  Returns (state, elapsed time, last ratio)."""
        ew, eu, ev, _, _ = self.interface(*S)
        ratio = self.fluxes(S[0], ew, eu, ev)[1]
        t = 0.0
        for n in range(steps):
            dt = cfl * float(ratio)
            t += dt
            S, ratio = self.step(S, scheme, dt)
            if look:
                look(n + 1, S)
        return S, t, float(ratio)


def _columns(prim, device):
    p = torch.as_tensor(prim, dtype=torch.float64, device=device)
    return [p[:, 0].clone(), p[:, 1].clone(), p[:, 2].clone()]


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "inversion":
        return _exact_inversion(case, seed, device)
    with torch.no_grad():
        if kind in ("driver", "run"):
            mesh, prim = _scene(case["scene"], case["side"], seed)
            plain = _Plain(mesh, torch.as_tensor(mesh.geometry[:, 2].copy(), device=device), case, device)
            S, t, ratio = plain.cfl_steps(_columns(prim, device), case["scheme"], case["steps"], case["cfl"])
            if kind == "run":
                return {"state": torch.stack(S, 1), "time": t}
            return {"state": torch.stack(S, 1), "ratio": ratio}
        if kind == "ensemble":
            got = []
            for mesh, prim in _basins(case, seed):
                plain = _Plain(mesh, torch.as_tensor(mesh.geometry[:, 2].copy(), device=device), case, device)
                S, _, _ = plain.cfl_steps(_columns(prim, device), case["scheme"], case["steps"], case["cfl"])
                got.append(torch.stack(S, 1))
            return {"state": torch.cat(got)}
        if kind == "inversions":
            return _exact_inversions(case, seed, device)
        return _exact_fields(case, seed, device)


def _exact_inversion(case, seed, device):
    flat, mesh, w, uv, z, gauges, seen = _offshore(case, seed)
    at, seen = torch.as_tensor(gauges, device=device), torch.as_tensor(seen, device=device)

    def traces(w, z):
        rows = []

        def look(n, S):
            if n % case["every"] == 0:
                rows.append(S[0][at])

        plain = _Plain(mesh, z, case, device)
        plain.cfl_steps([w] + _columns(np.column_stack([uv[:, :1], uv]), device)[1:], "SSPRK2", case["steps"],
                        case["cfl"], look)
        return torch.stack(rows)

    wt = torch.as_tensor(w, device=device).requires_grad_(True)
    zt = torch.as_tensor(z, device=device).requires_grad_(True)
    first = traces(wt, zt)
    (0.5 * (first - seen).square().sum()).backward()
    with torch.no_grad():
        second = traces(wt, zt - 1e-3 * zt.grad / zt.grad.abs().max())
    return {"first": first.detach(), "grad_w": wt.grad, "grad_z": zt.grad, "second": second}


def _exact_inversions(case, seed, device):
    basins, gauges, _ = _shores(case, seed)
    cols = []
    for (mesh, prim), at in zip(basins, gauges):
        plain, at, rows = _Plain(mesh, torch.as_tensor(mesh.geometry[:, 2].copy(), device=device), case, device), \
            torch.as_tensor(at, device=device), []

        def look(n, S):
            if n % case["every"] == 0:
                rows.append(S[0][at])

        plain.cfl_steps(_columns(prim, device), "SSPRK2", case["steps"], case["cfl"], look)
        cols.append(torch.stack(rows))
    # the gradient at a shore is regularised (the level's slope in a nearly dry cell grows without bound), so it has
    # no plain value; nor do the traces over the bed that it moved
    return {"first": torch.cat(cols, 1), "grad_w": None, "grad_z": None, "second": None}


def _exact_fields(case, seed, device):
    mesh, prim = _scene(case["scene"], case["side"], seed)
    plain = _Plain(mesh, torch.as_tensor(mesh.geometry[:, 2].copy(), device=device), case, device)
    W, U, V = _columns(prim, device)
    ew, eu, ev, sx, sy = plain.interface(W, U, V)
    F, ratio = plain.fluxes(W, ew, eu, ev)
    E, C = plain.L.numel(), W.numel()
    edges, sources = torch.zeros((2 * E, 3), device=device, dtype=W.dtype), torch.zeros((2 * E, 3), device=device,
                                                                                       dtype=W.dtype)
    for k in range(3):  # value of cell i towards its neighbour j: row 2 e + (i < j)
        row = 2 * plain.ce[k] + (torch.arange(C, device=device) < plain.ct[k]).to(torch.int64)
        edges[row] = torch.stack([ew[k], eu[k], ev[k]], 1)
        sources[row, 1], sources[row, 2] = sx[k], sy[k]
    level, gx, gy = plain._planes(W, U, V)[:3]
    h = W - plain.T[2]
    A, wet = plain.A, h > WET
    sums = torch.stack([(q * wet).sum() for q in (A * h, A * (0.5 * h * (U * U + V * V)),
                                                  A * (0.5 * h * h + h * plain.T[2]))])
    return {"edges": edges, "sources": sources, "fluxes": torch.stack(F, 1),
            "node_max": plain._node_max(level, gx, gy), "ratio": float(ratio), "integrals": sums}
