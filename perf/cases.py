"""The workloads whose speed this framework is measured on.

Every case is one pass through the public Python entry points, on the seeded
synthetic circuits of ``neospice_b200.workloads``, at sizes from one small
circuit (latency and launches) to batches and single systems that fill the
GPU:

  lu        batched refactor + solve (+ transposed solve) of given matrices:
            what a caller with its own Newton loop asks for (solver.Batch)
  ac        one complex refactor + solve per frequency point of an AC sweep
  grid      one large power-grid matrix over the whole GPU (AMD-LU)
  dc        DC operating points of diode-clamped resistor meshes (DcBatch),
            with the adjoint gradient of the solutions where ``grad`` is set
  chain     transients of CMOS inverter chains, plain and Monte Carlo
  bsim4     transients of the BSIM4v7 ring + NAND Monte Carlo circuit
  tree      recorded transient of inverter-driven RC trees and the gradient
            of a loss over its timepoints

All arithmetic of this framework is float64, so there is one data type.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from neospice_b200 import workloads as W
from neospice_b200.autodiff import dc_solve, tran_loss
from neospice_b200.circuit import DcBatch, TranBatch
from neospice_b200.solver import Batch, Topology

PULSE = (0.0, 1.8, 0.0, 1e-10, 1e-10, 1e-9, 2e-9)
TSTEP = 1e-12


def listed():
    return [
        # one small circuit's matrix (37 unknowns), factored and solved: the
        # call latency a caller's own Newton loop pays per iteration
        {"name": "lu_one", "kind": "lu", "side_lo": 6, "side_hi": 6, "count": 1,
         "transposed": False},
        # a ragged batch of several hundred circuits (145 .. 577 unknowns),
        # with the transposed solve an adjoint or noise analysis needs
        {"name": "lu_many", "kind": "lu", "side_lo": 12, "side_hi": 24, "count": 592,
         "transposed": True},
        # an AC sweep: 150 frequency points of a 1026-unknown RC mesh
        {"name": "ac_sweep", "kind": "ac", "side": 32, "points": 150},
        # one 16,393-unknown power grid factored and solved by the whole GPU
        {"name": "power_grid", "kind": "grid", "side": 128},
        # one operating point alone (2305 unknowns): interactive use
        {"name": "dc_one", "kind": "dc", "side_lo": 48, "side_hi": 48, "count": 1, "grad": False},
        # the ordinary batch: several hundred ragged meshes (257 .. 1601 unknowns)
        {"name": "dc_many", "kind": "dc", "side_lo": 16, "side_hi": 40, "count": 600,
         "grad": False},
        # large meshes (5185 unknowns), a Monte Carlo sweep of one circuit size
        {"name": "dc_large", "kind": "dc", "side_lo": 72, "side_hi": 72, "count": 148,
         "grad": False},
        # operating points with the gradient of a loss over them (backward)
        {"name": "dc_grad", "kind": "dc", "side_lo": 16, "side_hi": 32, "count": 200,
         "grad": True},
        # one transient of the 32-stage inverter chain: latency of one run
        {"name": "chain_one", "kind": "chain", "stages": 32, "count": 1, "tstop": 0.3e-9},
        # its Monte Carlo over thresholds and transconductances
        {"name": "chain_many", "kind": "chain", "stages": 32, "count": 400, "tstop": 0.2e-9},
        # BSIM4v7 Monte Carlo, 200 MOSFETs per instance
        {"name": "bsim4_many", "kind": "bsim4", "stages": 25, "count": 300, "tstop": 0.06e-9},
        # interconnect optimisation: forward transient + adjoint gradient
        {"name": "tree_grad", "kind": "tree", "nodes": 500, "count": 64, "tstop": 0.1e-9},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lu", "ac", "grid", "dc", "dc", "chain", "bsim4", "tree"])
    if kind == "lu":
        hi = _log_int(rng, 4, 40)
        return {"kind": "lu", "side_lo": max(3, hi - rng.randrange(0, 8)), "side_hi": hi,
                "count": _log_int(rng, 1, 600), "transposed": rng.random() < 0.5}
    if kind == "ac":
        return {"kind": "ac", "side": _log_int(rng, 6, 40), "points": _log_int(rng, 10, 200)}
    if kind == "grid":
        return {"kind": "grid", "side": _log_int(rng, 50, 128)}
    if kind == "dc":
        hi = _log_int(rng, 8, 56)
        most = 600 if hi <= 40 else 200
        return {"kind": "dc", "side_lo": max(6, hi - rng.randrange(0, 9)), "side_hi": hi,
                "count": _log_int(rng, 1, most), "grad": rng.random() < 0.4}
    if kind == "chain":
        return {"kind": "chain", "stages": rng.randrange(5, 41), "count": _log_int(rng, 1, 400),
                "tstop": rng.randrange(60, 201) * 1e-12}
    if kind == "bsim4":
        return {"kind": "bsim4", "stages": 2 * rng.randrange(3, 16) + 1,
                "count": _log_int(rng, 1, 300), "tstop": rng.randrange(20, 61) * 1e-12}
    return {"kind": "tree", "nodes": _log_int(rng, 40, 600), "count": _log_int(rng, 1, 64),
            "tstop": rng.randrange(30, 101) * 1e-12}


# --- inputs --------------------------------------------------------------------------


def _sides(case):
    """One side per instance, the same for every seed; at most eight
    different ones in an lu batch (a caller's handful of circuits)."""
    lo, hi, count = case["side_lo"], case["side_hi"], case["count"]
    if case["kind"] == "lu":
        kinds = np.unique(np.linspace(lo, hi, min(8, count)).round().astype(int))
        return [int(kinds[i % len(kinds)]) for i in range(count)]
    return [int(s) for s in np.random.default_rng([lo, hi, count]).integers(lo, hi + 1, count)]


def _lu_inputs(case, seed):
    """Per side the mesh's matrix at zero bias, and per instance its values
    with the diodes' conductances of some operating point (the diagonals a
    Newton iteration changes) and a process spread on all conductances."""
    rng = np.random.default_rng([seed, 1])
    sides = _sides(case)
    systems = {}
    for s in dict.fromkeys(sides):
        mesh = W.diode_mesh(np.random.default_rng([seed, 2, s]), side=s)
        circ = mesh.build()
        cp, ri = circ.pattern()
        a, _ = circ.initial_matrix(1e-12)
        cols = np.repeat(np.arange(len(cp) - 1), np.diff(cp))
        systems[s] = (len(cp) - 1, cp, ri, cols, a)
    values, rhs = [], []
    for s in sides:
        n, _, ri, cols, a = systems[s]
        v = np.where(np.abs(a) == 1.0, a, a * np.exp(0.05 * rng.standard_normal()))
        clamped = (ri == cols) & (ri < n - 1) & (rng.random(len(ri)) < 0.05)
        v[clamped] += rng.uniform(0.0, 0.04, int(clamped.sum()))
        values.append(v)
        b = np.where(rng.random(n) < 0.02, rng.uniform(0.0, 1e-3, n), 0.0)
        b[-1] = 1.0
        rhs.append(b)
    return sides, systems, values, rhs


def _ac_inputs(case, seed):
    nl = W.rc_mesh(np.random.default_rng([seed, 3]), case["side"])
    n, cp, ri, g, c, b = W.ac_system(nl)
    omegas = 2 * np.pi * np.logspace(3, 11, case["points"])
    ax = np.empty((case["points"], 2 * len(ri)))
    ax[:, 0::2] = g
    ax[:, 1::2] = omegas[:, None] * c
    bz = np.zeros((case["points"], 2 * n))
    bz[:, 0::2] = b.real
    bz[:, 1::2] = b.imag
    return n, cp, ri, ax, bz


def _grid_inputs(case, seed):
    n, cp, ri, v = W.power_grid_transient(case["side"], seed)
    return n, cp, ri, v, np.random.default_rng([seed, 4]).standard_normal(n)


def _meshes(case, seed):
    """Meshes whose layout (where diodes and sources sit) is the case's and
    whose resistances and currents are the seed's."""
    out = []
    for i, s in enumerate(_sides(case)):
        mesh = W.diode_mesh(np.random.default_rng([6, i, s]), side=s)
        rng = np.random.default_rng([seed, 5, i])
        mesh.r_h = 1000.0 * np.exp(0.1 * rng.standard_normal(len(mesh.r_h)))
        mesh.r_v = 1000.0 * np.exp(0.1 * rng.standard_normal(len(mesh.r_v)))
        mesh.isrc_amps = rng.uniform(0.0, 1e-3, len(mesh.isrc_amps))
        out.append(mesh)
    return out


def _dc_weights(size, seed):
    return np.random.default_rng([seed, 7]).standard_normal(size)


def _netlists(case, seed):
    rngs = [np.random.default_rng([seed, 8, i]) for i in range(case["count"])]
    if case["kind"] == "chain":
        return [W.inverter_chain_mc(r, case["stages"], pulse=PULSE) for r in rngs]
    if case["kind"] == "bsim4":
        return [W.bsim4_ring_nand(r, case["stages"]) for r in rngs]
    return [W.rc_tree_driven(r, case["nodes"]) for r in rngs]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lu":
        sides, systems, values, rhs = _lu_inputs(case, seed)
        topo = {s: Topology.order(n, cp, ri, a) for s, (n, cp, ri, _, a) in systems.items()}
        return {"kind": kind, "transposed": case["transposed"],
                "batch": Batch([topo[s] for s in sides]),
                "values": torch.from_numpy(np.concatenate(values)).cuda(),
                "rhs": torch.from_numpy(np.concatenate(rhs)).cuda()}
    if kind == "ac":
        n, cp, ri, ax, bz = _ac_inputs(case, seed)
        topo = Topology.order_complex(n, cp, ri, ax[0])
        return {"kind": kind, "batch": Batch([topo] * case["points"]),
                "values": torch.from_numpy(ax.ravel()).cuda(),
                "rhs": torch.from_numpy(bz.ravel()).cuda()}
    if kind == "grid":
        n, cp, ri, v, b = _grid_inputs(case, seed)
        batch = Batch([Topology.order(n, cp, ri, v, solver="auto-amdlu")])
        batch.set_schedule(2)
        return {"kind": kind, "batch": batch, "values": torch.from_numpy(v).cuda(),
                "rhs": torch.from_numpy(b).cuda()}
    if kind == "dc":
        meshes = _meshes(case, seed)
        batch = DcBatch([m.build() for m in meshes], symbolic=DcBatch.PER_PATTERN)
        params = np.concatenate([m.params() for m in meshes])
        state = {"kind": kind, "grad": case["grad"], "batch": batch,
                 "params": torch.from_numpy(params).cuda()}
        if case["grad"]:
            weights = _dc_weights(int(batch.solution_offsets[-1]), seed)
            state["weights"] = torch.from_numpy(weights).cuda()
        return state
    nls = _netlists(case, seed)
    circuits = [nl.build() for nl in nls]
    if kind == "tree":
        far = case["nodes"] - 1
        points = int(case["tstop"] / TSTEP * 1.3) + 200
        batch = TranBatch(circuits, TSTEP, case["tstop"], np.full(1, far, np.int32),
                          max_points=points)
        batch.record(True)
        _, p_dc, _ = batch.params()
        return {"kind": kind, "batch": batch, "far": np.full(case["count"], far),
                "targets": torch.full((case["count"] * points,), 0.9, dtype=torch.float64,
                                      device="cuda"),
                "params": torch.from_numpy(p_dc).cuda().requires_grad_(True)}
    points = int(case["tstop"] / TSTEP * 1.3) + 400
    probes = np.arange(nls[0].num_nodes) if case["count"] == 1 else np.arange(1, 6)
    return {"kind": kind, "batch": TranBatch(circuits, TSTEP, case["tstop"], probes,
                                             max_points=points)}


# --- one pass ------------------------------------------------------------------------


def run(state):
    kind, batch = state["kind"], state["batch"]
    if kind in ("lu", "grid"):
        status, _ = batch.refactor(state["values"])
        out = {"x": batch.solve(state["rhs"].clone()), "status": status}
        if state.get("transposed"):
            out["xt"] = batch.solve_transposed(state["rhs"].clone())
        return out
    if kind == "ac":
        lu, status = batch.refactor_complex(state["values"])
        return {"x": batch.solve_complex(lu, state["rhs"].clone()), "status": status}
    if kind == "dc":
        if not state["grad"]:
            x, status, iterations = batch.run(state["params"])
            return {"x": x, "status": status, "iterations": iterations}
        params = state["params"].detach().requires_grad_(True)
        x = dc_solve(batch, params)
        (x * state["weights"]).sum().backward()
        return {"x": x.detach(), "grad": params.grad}
    batch.run()
    if kind == "tree":
        params = state["params"].detach().requires_grad_(True)
        loss = tran_loss(batch, state["far"], state["targets"], params)
        loss.sum().backward()
        return {"loss": loss.detach(), "grad": params.grad}
    res = batch.results()
    return {"time": np.concatenate([r["time"] for r in res]),
            "values": np.concatenate([r["values"] for r in res]),
            "points": np.array([len(r["time"]) for r in res]),
            "status": np.array([r["status"] for r in res]),
            "iterations": np.array([r["newton_iters"] for r in res])}


# --- what a pass cannot do without ---------------------------------------------------


def _mesh_flops(n):
    """Multiply-subtracts (two operations each) of one sparse LU of an
    n-unknown mesh under minimum degree (measured 10 .. 28 n^1.5 for 257 ..
    9217 unknowns)."""
    return 3.2 * n ** 1.5 * math.log(n) ** 0.95


def work(case):
    kind = case["kind"]
    if kind == "lu":
        sides = _sides(case)
        solves = 2 if case["transposed"] else 1
        b = f = 0.0
        for s in sides:
            n = s * s + 1
            fill = n * (2 + 3.2 * math.log(n))  # LU entries, measured on these meshes
            b += 8 * 5 * n + 16 * n * solves
            f += _mesh_flops(n) + 2 * fill * solves
        return {"bytes": b, "flops": f}
    if kind == "ac":
        n = case["side"] ** 2 + 2
        return {"bytes": case["points"] * (16 * 5 * n + 32 * n),
                "flops": case["points"] * 4 * _mesh_flops(n)}
    if kind == "grid":
        n = case["side"] ** 2
        return {"bytes": 8 * 5 * n + 16 * n, "flops": 1.6 * _mesh_flops(n)}
    if kind == "dc":
        b = f = 0.0
        mid = (case["side_lo"] + case["side_hi"]) / 2
        n = mid * mid + 1
        # 2 n resistors and 15 values per diode in, n unknowns out; about
        # eight Newton iterations
        b = case["count"] * 8 * (2 * n + 0.75 * n + n) * (2 if case["grad"] else 1)
        f = case["count"] * (9 if case["grad"] else 8) * _mesh_flops(n)
        return {"bytes": b, "flops": f}
    steps = case["tstop"] / TSTEP
    if kind == "chain":
        # per Newton iteration (two per step) 2 MOSFETs a stage, some 300
        # operations each; the time and the probes of each step out
        probes = case["stages"] + 2 if case["count"] == 1 else 5
        return {"bytes": case["count"] * (8 * 90 + steps * 8 * (1 + probes)),
                "flops": case["count"] * steps * 2 * case["stages"] * 600}
    if kind == "bsim4":
        # 6.4e5 operations a Newton iteration with 200 devices (measured)
        return {"bytes": case["count"] * (8 * case["stages"] * 8 * 130 + steps * 8 * 6),
                "flops": case["count"] * steps * 2 * case["stages"] * 25600}
    n = case["nodes"]
    return {"bytes": case["count"] * (8 * 4 * n + 8 * steps), "flops": case["count"] * steps * 7 * 40 * n}


# --- the same in 64 bits without this framework ---------------------------------------


def _dense_batches(mats, rhs, transposed=False, complex_=False):
    """Solutions of the sparse systems (n, rows, cols, values) by dense LU on
    the GPU, a few at a time."""
    out = []
    kind = torch.complex128 if complex_ else torch.float64
    for (n, rows, cols, v), b in zip(mats, rhs):
        m = torch.zeros((n, n), dtype=kind, device="cuda")
        at = (torch.as_tensor(rows, device="cuda").long(), torch.as_tensor(cols, device="cuda").long())
        m[at] = torch.as_tensor(v, device="cuda")
        out.append(torch.linalg.solve(m.T if transposed else m, torch.as_tensor(b, device="cuda")))
    return torch.cat(out).cpu().numpy()


def _mesh_exact(mesh, weights):
    """Operating point of one mesh by a dense Newton iteration, converged to
    the last places, and (given weights) the gradient of weights . x."""
    s, n = mesh.side, mesh.num_nodes
    dev = "cuda"
    grid = np.arange(n).reshape(s, s)
    ends = np.concatenate([np.stack([grid[:, :-1].ravel(), grid[:, 1:].ravel()]),
                           np.stack([grid[:-1, :].ravel(), grid[1:, :].ravel()])], axis=1)
    a, b = (torch.as_tensor(e, device=dev) for e in ends)
    r = torch.as_tensor(np.concatenate([mesh.r_h, mesh.r_v]), device=dev)
    g = torch.zeros((n + 1, n + 1), dtype=torch.float64, device=dev)
    for i, j, sign in ((a, a, 1), (b, b, 1), (a, b, -1), (b, a, -1)):
        g.index_put_((i, j), sign / r, accumulate=True)
    g[0, n] = g[n, 0] = 1.0
    rhs = torch.zeros(n + 1, dtype=torch.float64, device=dev)
    rhs[torch.as_tensor(mesh.isrc_nodes, device=dev).long()] += torch.as_tensor(mesh.isrc_amps, device=dev)
    rhs[n] = mesh.v_corner
    dn = torch.as_tensor(mesh.diode_nodes, device=dev).long()
    vt = mesh.diode_n * 300.15 * 1.38064852e-23 / 1.6021766208e-19
    vcrit = vt * math.log(vt / (math.sqrt(2.0) * mesh.diode_is))
    vd = torch.full((len(dn),), vcrit, dtype=torch.float64, device=dev)
    x = torch.zeros(n + 1, dtype=torch.float64, device=dev)
    for _ in range(100):
        e = torch.exp(vd / vt)
        gd = mesh.diode_is * e / vt + 1e-12
        cur = mesh.diode_is * (e - 1.0) + 1e-12 * vd
        j, c = g.clone(), rhs.clone()
        j[dn, dn] += gd
        c[dn] -= cur - gd * vd
        new = torch.linalg.solve(j, c)
        dv = new[dn] - vd
        up = (new[dn] > vcrit) & (dv > 2 * vt)
        vd = torch.where(up, vd + vt * torch.log1p(torch.clamp(dv, min=0.0) / vt), new[dn])
        done = not bool(up.any()) and float((new - x).abs().max()) < 1e-13
        x = new
        if done:
            break
    if weights is None:
        return x, None
    j = g.clone()
    j[dn, dn] += mesh.diode_is * torch.exp(x[dn] / vt) / vt + 1e-12
    lam = torch.linalg.solve(j.T, torch.as_tensor(weights, device=dev))
    gr = (lam[a] - lam[b]) * (x[a] - x[b]) / r ** 2
    gi = lam[torch.as_tensor(mesh.isrc_nodes, device=dev).long()]
    zero = torch.zeros(len(mesh.params()) - len(gr) - len(gi) - 1, dtype=torch.float64, device=dev)
    return x, torch.cat([gr, zero, gi, lam[n:]])


def exact(case, seed):
    kind = case["kind"]
    if kind == "lu":
        if case["count"] * (case["side_hi"] ** 2 + 1) ** 3 > 1e13:
            return None
        sides, systems, values, rhs = _lu_inputs(case, seed)
        mats = [(systems[s][0], systems[s][2], systems[s][3], v) for s, v in zip(sides, values)]
        out = {"x": _dense_batches(mats, rhs), "status": None}
        if case["transposed"]:
            out["xt"] = _dense_batches(mats, rhs, transposed=True)
        return out
    if kind == "ac":
        n, cp, ri, ax, bz = _ac_inputs(case, seed)
        if case["points"] * n ** 3 > 2e12:
            return None
        cols = np.repeat(np.arange(n), np.diff(cp))
        z = _dense_batches([(n, ri, cols, v[0::2] + 1j * v[1::2]) for v in ax],
                           [b[0::2] + 1j * b[1::2] for b in bz], complex_=True)
        return {"x": z.view(np.float64), "status": None}
    if kind == "grid":
        n, cp, ri, v, b = _grid_inputs(case, seed)
        cols = np.repeat(np.arange(n), np.diff(cp))
        return {"x": _dense_batches([(n, ri, cols, v)], [b]), "status": None}
    if kind == "dc":
        if case["count"] * 10 * max(case["side_hi"], 24) ** 6 > 3e13:
            return None
        meshes = _meshes(case, seed)
        xs, grads, at = [], [], 0
        weights = _dc_weights(sum(m.num_vars for m in meshes), seed) if case["grad"] else None
        for m in meshes:
            w = None if weights is None else weights[at:at + m.num_vars]
            at += m.num_vars
            x, g = _mesh_exact(m, w)
            xs.append(x)
            grads.append(g)
        if case["grad"]:
            return {"x": torch.cat(xs), "grad": torch.cat(grads)}
        return {"x": torch.cat(xs), "status": None, "iterations": None}
    # a transient's discrete steps are the integrator's own: nothing outside
    # it gives their values
    return None
