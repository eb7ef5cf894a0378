"""Performance cases of the particle path, each one pass through the public entry points.

A case is a dict of plain values; `kind` selects one of four families:

  fempic  whole FemPIC steps (inject, push, move + deposit, hole fill / sort) of a box mesh in its
          steady state, through FemPIC.step, FemPIC.run_graph or FemPIC.run_steps
  field   FemPIC's field phase (node charge density, one Newton step, cell field) from given charges
  cabana  CabanaPIC's move + current deposit on a periodic two-stream state
  advec   NESO-advection steps of one instance or of a batch of instances

exact() computes the same pass with plain torch operations in 64 bits.
"""
from __future__ import annotations

import functools
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = Path(__file__).resolve().parent.parent / "op-pic_b200"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

from oppb.advec import AdvecBatchDevice, AdvecMesh  # noqa: E402
from oppb.cabana import CabanaDevice, Deck, HexMesh, synthetic_interp  # noqa: E402
from oppb.fempic import FemPIC, HostMesh  # noqa: E402
from oppb.field import FieldConstants, FieldDevice, boundary_potential  # noqa: E402

DEV = "cuda:0"
REMOVED = 2147483647
FILL_STEPS = 300      # steps to the steady state: ions cross the box in about 230
RESIDENCE = 230       # steady particles per injected particle a step
SIGMA = 0.1           # thermal velocity
FIELD = dict(n0=1.0, phi0=0.0, kte=100.0, qe=1.0, eps0=1.0)


def listed() -> list[dict]:
    return [
        # A small run driven step by step from the host: every launch and readback counts.
        dict(name="fempic_small_step_f64", kind="fempic", nx=10, ny=10, nz=40, inject=2000, precision="f64",
             fill="HoleFill_All", period=10, dh=0.0, api="step", steps=4),
        # The same size replayed as captured sort cycles, mixed precision.
        dict(name="fempic_small_graph_mixed", kind="fempic", nx=10, ny=10, nz=40, inject=2000, precision="mixed",
             fill="Sort_Periodic", period=10, dh=0.0, api="graph", steps=10),
        # An ordinary run on an odd-sized mesh with the global move (direct-hop seed) on.
        dict(name="fempic_mid_dh_f64", kind="fempic", nx=23, ny=19, nz=61, inject=13001, precision="f64",
             fill="HoleFill_All", period=10, dh=0.02, api="step", steps=2),
        # The loops launched one by one (push, move, deposit), sorted every step, as a generated main
        # with opp_fill = Sort_All runs them.
        dict(name="fempic_mid_loops_sort_f64", kind="fempic", nx=24, ny=24, nz=96, inject=30000, precision="f64",
             fill="Sort_All", period=10, dh=0.0, api="loops", steps=2),
        # The benchmark's workload in FP64, one whole sort cycle.
        dict(name="fempic_large_step_f64", kind="fempic", nx=48, ny=48, nz=192, inject=250000, precision="f64",
             fill="Sort_Periodic", period=10, dh=0.0, api="step", steps=10),
        # The benchmark's workload in mixed precision, fed from and returning to pinned host memory.
        dict(name="fempic_large_host_mixed", kind="fempic", nx=48, ny=48, nz=192, inject=250000, precision="mixed",
             fill="Sort_Periodic", period=10, dh=0.0, api="host", steps=10),
        # The field phase of the small and of the benchmark's mesh.
        dict(name="field_small", kind="field", nx=10, ny=10, nz=40),
        dict(name="field_large", kind="field", nx=48, ny=48, nz=192),
        # A small FP32-momentum CabanaPIC run on an odd-sized mesh.
        dict(name="cabana_small_mixed", kind="cabana", nx=15, ny=13, nz=37, nppc=64, precision="mixed", steps=5),
        # The benchmark's two-stream workload, ten steps of a run in progress.
        dict(name="cabana_large_f64", kind="cabana", nx=32, ny=32, nz=256, nppc=400, precision="f64", steps=10),
        # One advection instance whose cells are read from their records (any mesh, not a verified grid).
        dict(name="advec_small_records", kind="advec", instances=1, side_lo=61, side_hi=61, ppc_lo=37, ppc_hi=37,
             grid=False, dh=0.0, steps=1, graph=False, layout=5),
        # The benchmark's ensemble of 64 uneven instances, ten steps replayed from a graph.
        dict(name="advec_ensemble", kind="advec", instances=64, side_lo=64, side_hi=512, ppc_lo=10, ppc_hi=200,
             grid=True, dh=0.0, steps=10, graph=True, layout=5),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> int:
    return max(int(lo), min(int(hi), round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["fempic", "fempic", "fempic", "field", "cabana", "advec"])
    if kind == "fempic":
        nx, ny = _log(rng, 4, 48), _log(rng, 4, 48)
        nz = _log(rng, 8, 192)
        inject = max(2 * nx * ny, _log(rng, 1000, 200000))
        fill = rng.choice(["HoleFill_All", "Sort_Periodic", "Sort_Periodic", "Sort_All", "Shuffle_Periodic"])
        period = rng.choice([5, 10])
        api = rng.choice(["step", "graph", "host", "loops"])
        precision = "f64" if api == "loops" else rng.choice(["f64", "mixed"])
        dh = round(rng.uniform(0.015, 0.05), 3) if api in ("step", "host") and rng.random() < 0.3 else 0.0
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, inject=inject, precision=precision, fill=fill, period=period,
                    dh=dh, api=api, steps=period)
    if kind == "field":
        return dict(kind=kind, nx=_log(rng, 4, 48), ny=_log(rng, 4, 48), nz=_log(rng, 8, 192))
    if kind == "cabana":
        nx, ny, nz = _log(rng, 4, 32), _log(rng, 4, 32), _log(rng, 8, 256)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nppc=2 * _log(rng, 8, 200), precision=rng.choice(["f64", "mixed"]),
                    steps=rng.choice([1, 5, 10]))
    n = _log(rng, 1, 48)
    lo = _log(rng, 16, 300)
    grid = rng.random() < 0.6
    dh = round(rng.uniform(0.4, 2.0), 2) if rng.random() < 0.25 else 0.0
    return dict(kind=kind, instances=n, side_lo=lo, side_hi=lo + _log(rng, 1, 150), ppc_lo=5, ppc_hi=_log(rng, 6, 150),
                grid=grid, dh=dh, steps=rng.choice([1, 10]), graph=rng.random() < 0.5, layout=rng.randrange(1000))


# ------------------------------------------------------------------------------ set-up

@functools.lru_cache(maxsize=2)
def _host_mesh(nx: int, ny: int, nz: int) -> HostMesh:
    return HostMesh(nx, ny, nz, 1.0, 1.0, 4.0)


def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _injection_table(g: torch.Generator, count: int) -> torch.Tensor:
    t = torch.empty((5, count), dtype=torch.float64, device=DEV)
    t[:2].uniform_(0.0, 1.0, generator=g)
    t[2:].normal_(0.0, SIGMA, generator=g)
    return t


def _capacity(case: dict) -> int:
    """Room for the steady state, ten steps' injection and the graph capture's 2 % slack."""
    return case["inject"] * 248 + 1000


def _prepare_fempic(case: dict, seed: int) -> dict:
    hm = _host_mesh(case["nx"], case["ny"], case["nz"])
    n = case["inject"]
    sim = FemPIC(hm, DEV, inject_per_step=n, precision=case["precision"], fill=case["fill"],
                 fill_period=case["period"], capacity=_capacity(case), fused_deposit=case["api"] != "loops",
                 direct_hop=case["dh"] or None)
    g = _gen(seed)
    for _ in range(FILL_STEPS):
        sim.step(_injection_table(g, n))
    tables = [_injection_table(g, n) for _ in range(case["steps"])]
    state = dict(case=case, sim=sim, tables=tables)
    if case["api"] == "host":
        state["host"] = [t.cpu().pin_memory() for t in tables]
        state["charges"] = [torch.empty(hm.n_nodes, dtype=torch.float64).pin_memory() for _ in tables]
    return state


def _prepare_field(case: dict, seed: int) -> dict:
    hm = _host_mesh(case["nx"], case["ny"], case["nz"])
    fd = FieldDevice(hm, DEV, boundary_potential(hm.n_type, 1.0, 0.0))
    # Node charges of a steady state: about 20 particles a cell, deposited with their weights.
    count = 20.0 * hm.n_cells
    vol = torch.from_numpy(np.ascontiguousarray(hm.n_vol)).to(DEV)
    mean = vol * (count / float(vol.sum()))
    g = _gen(seed)
    noise = torch.empty(hm.n_nodes, dtype=torch.float64, device=DEV).normal_(0.0, 1.0, generator=g)
    charge = (mean + noise * (0.5 * mean).sqrt()).clamp_min_(0.0)
    return dict(case=case, fd=fd, charge=charge, den=torch.empty_like(charge), vol=vol, spwt=4.0 / count,
                consts=FieldConstants(**FIELD), ef=torch.zeros(hm.n_cells, 4, dtype=torch.float64, device=DEV))


def _deck(case: dict) -> Deck:
    return Deck(case["nx"], case["ny"], case["nz"], case["nx"] / 32.0, case["ny"] / 32.0, case["nz"] / 32.0,
                nppc=case["nppc"], courant_frac=0.5)


_CABANA_DATS = ("pos", "vel", "vel32", "p2c", "streak")


def _prepare_cabana(case: dict, seed: int) -> dict:
    mesh, deck = HexMesh(case["nx"], case["ny"], case["nz"]), _deck(case)
    cd = CabanaDevice(mesh, DEV, len(mesh.interior) * case["nppc"], precision=case["precision"])
    interp = synthetic_interp(mesh, seed)
    cd.set_interp(interp)
    cd.fill_two_stream(mesh, deck, 0.2, 0.01, seed)
    for _ in range(20):  # a run in progress: the streams have left their initial cells
        cd.move_deposit(deck)
    start = {k: getattr(cd, k).clone() for k in _CABANA_DATS if getattr(cd, k) is not None}
    return dict(case=case, cd=cd, deck=deck, start=start, mesh=mesh, interp=interp)


@functools.lru_cache(maxsize=256)
def _advec_mesh(side: int) -> AdvecMesh:
    return AdvecMesh(side, side, 1.0)


def _advec_layout(case: dict) -> tuple[list[int], list[int]]:
    rng = np.random.default_rng(case["layout"])
    sides = rng.integers(case["side_lo"], case["side_hi"] + 1, case["instances"])
    ppcs = rng.integers(case["ppc_lo"], case["ppc_hi"] + 1, case["instances"])
    return [int(s) for s in sides], [int(p) for p in ppcs]


def _prepare_advec(case: dict, seed: int) -> dict:
    sides, ppcs = _advec_layout(case)
    meshes = [_advec_mesh(s) for s in sides]
    bd = AdvecBatchDevice(meshes, [m.n_cells * p for m, p in zip(meshes, ppcs)], [0.5] * len(meshes), DEV,
                          grid=case["grid"])
    for k, p in enumerate(ppcs):
        bd.fill_instance(k, p, 0.5, 1.0, seed * 1000 + k)
    if case["dh"]:
        bd.enable_direct_hop(case["dh"])
    for _ in range(5):
        bd.step()
    state = dict(case=case, bd=bd)
    if case["graph"]:
        state["graph"] = bd.capture(case["steps"])
    return state


def prepare(case: dict, seed: int) -> dict:
    return {"fempic": _prepare_fempic, "field": _prepare_field, "cabana": _prepare_cabana,
            "advec": _prepare_advec}[case["kind"]](case, seed)


# -------------------------------------------------------------------------------- pass

def _run_fempic(s: dict) -> dict:
    sim, api = s["sim"], s["case"]["api"]
    if api == "graph":
        sim.run_graph(s["tables"])
    elif api == "host":
        sim.run_steps(s["host"], s["charges"])
    else:
        for t in s["tables"]:
            sim.step(t)
    p = sim.parts
    n = p.size
    out = {"size": n, "charge": sim.node_charge}
    for k in ("pos", "vel", "lc", "p2c"):  # the set's whole buffers, the free slots cleared
        out[k] = getattr(p, k)
        out[k][:, n:].zero_()
    if api == "host":
        out["charges"] = s["charges"]
    return out


def _run_field(s: dict) -> dict:
    fd = s["fd"]
    s["den"].copy_(s["charge"])
    fd.d.zero_()   # the Newton step of a run's first field phase
    fd.f1.zero_()
    fd.launch(s["den"], s["vol"], s["spwt"], s["consts"], s["ef"], 4)
    return {"density": s["den"], "potential": fd.potential, "d": fd.d, "f1": fd.f1, "ef": s["ef"]}


def _run_cabana(s: dict) -> dict:
    cd = s["cd"]
    for k, t in s["start"].items():  # restart from the saved state: every pass advances the same steps
        getattr(cd, k).copy_(t)
    for _ in range(s["case"]["steps"]):
        cd.move_deposit(s["deck"])
    return {"pos": cd.pos, "vel": cd.vel if cd.vel32 is None else cd.vel32, "p2c": cd.p2c, "acc": cd.acc}


def _run_advec(s: dict) -> dict:
    bd = s["bd"]
    if "graph" in s:
        s["graph"].replay()
    else:
        for _ in range(s["case"]["steps"]):
            bd.step()
    return {"pos": bd.pos, "mdir": bd.mdir, "p2c": bd.p2c}


def run(state: dict) -> dict:
    return {"fempic": _run_fempic, "field": _run_field, "cabana": _run_cabana,
            "advec": _run_advec}[state["case"]["kind"]](state)


# ------------------------------------------------------------------------ work, tolerance

def work(case: dict) -> dict:
    if case["kind"] == "fempic":
        n = case["inject"] * RESIDENCE
        cells, nodes = 6 * case["nx"] * case["ny"] * case["nz"], (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        # pos, vel, p2c read and written and the weights written; the cell's geometry, neighbours,
        # nodes and field read; the node charges written.
        step = n * 136 + cells * ((160 if case["precision"] == "f64" else 80) + 16 + 32) + nodes * 8
        sorts = case["steps"] if case["fill"].endswith("_All") and case["fill"] != "HoleFill_All" else \
            case["steps"] // case["period"] if case["fill"].endswith("Periodic") else 0
        return {"bytes": float(case["steps"] * step + sorts * n * 168), "flops": float(case["steps"] * n * 2.4 * 40)}
    if case["kind"] == "field":
        cells = 6 * case["nx"] * case["ny"] * case["nz"]
        neq = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] - 1)
        it = 3.3 * max(case["nx"], case["ny"], case["nz"])  # CG iterations to 1e-10 grow with the box's edge
        return {"bytes": float(neq * (15 * 12 + 6 * 8) + cells * (16 + 8 + 96 + 32)),
                "flops": float(it * neq * (2 * 15 + 12))}
    if case["kind"] == "cabana":
        cells = (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
        n = case["nx"] * case["ny"] * case["nz"] * case["nppc"]
        per = 108 if case["precision"] == "f64" else 84
        return {"bytes": float(case["steps"] * (n * per + cells * 384)), "flops": float(case["steps"] * n * 300)}
    sides, ppcs = _advec_layout(case)
    n = sum(s * s * p for s, p in zip(sides, ppcs))
    # pos, vel and p2c read; pos, direction and p2c written.
    return {"bytes": float(case["steps"] * (n * 64 + sum(s * s for s in sides) * 32)),
            "flops": float(case["steps"] * n * 40)}


def tolerance(case: dict):
    """About four times what the same pass in another order of sums, or in plain torch, differs by."""
    if case["kind"] == "fempic":  # charges 5e-15 from the torch sums; FP32 weights 1e-7
        return {"rel": 3e-14} if case["precision"] == "f64" else {"rel": 5e-7}
    if case["kind"] == "field":   # the CG stops at 1e-10 of ||B||: the cell field is 2e-9 from the exact one
        return {"rel": 1e-8}
    if case["kind"] == "cabana":  # FP64 accumulator sums; FP32 momentum 4e-7
        return {"rel": 1e-13} if case["precision"] == "f64" else {"rel": 2e-6}
    return "exact"


# ------------------------------------------------------------------- the pass in plain torch

def _walk(mesh: dict, x: torch.Tensor, cell: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
    """Final cells (REMOVED for particles that leave) and weights of positions x [3, n]."""
    n = x.shape[1]
    out_cell, lc = cell.long().clone(), torch.zeros((4, n), dtype=torch.float64, device=DEV)
    todo = torch.arange(n, device=DEV)
    while todo.numel():
        c = out_cell[todo]
        xx, y, z = x[0, todo], x[1, todo], x[2, todo]
        d, coef = mesh["det"][c], mesh["coef"][c]
        lam = torch.stack([coef * (((d[:, 4 * i] - d[:, 4 * i + 1] * xx) + d[:, 4 * i + 2] * y) - d[:, 4 * i + 3] * z)
                           for i in range(4)])
        lc[:, todo] = lam
        inside = ((lam > -1e-10) & (lam - 1.0 < 1e-10)).all(0)
        nxt = mesh["c2c"][c, lam.argmin(0)]
        nxt = torch.where(nxt < 0, REMOVED, nxt)
        go = ~inside
        out_cell[todo[go]] = nxt[go]
        todo = todo[go & (nxt != REMOVED)]
    return out_cell, lc


def _exact_fempic(case: dict, seed: int):
    if case["inject"] * RESIDENCE * case["steps"] > 2e8:
        return None
    s = _prepare_fempic(case, seed)
    sim, hm = s["sim"], s["sim"].hm
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    mesh = {"det": t(hm.c_det), "coef": (1.0 / 6.0) / t(hm.c_vol), "c2c": t(hm.c2c).long()}
    c2n, ef = t(hm.c2n).long(), t(hm.c_ef)
    n = sim.parts.size
    x, v, cell = sim.parts.pos[:, :n].clone(), sim.parts.vel[:, :n].clone(), sim.parts.p2c[0, :n].long()
    lc = sim.parts.lc[:, :n].clone()
    dist, if2c = t(sim.dist_host), t(hm.if2c).long()
    u, w, norm, node0 = t(hm.if_u), t(hm.if_v), t(hm.if_norm), t(hm.if_n_pos)[:, :3]
    qm, dt, charges = sim.qm, sim.dt, []
    for k, tab in enumerate(s["tables"]):
        m = tab.shape[1]
        face = torch.searchsorted(dist, torch.arange(m, dtype=dist.dtype, device=DEV), right=True)
        face = face.clamp_max(len(if2c) - 1)
        fc = if2c[face]
        a, b = tab[0], tab[1]
        fold = a + b > 1
        a, b = torch.where(fold, 1 - a, a), torch.where(fold, 1 - b, b)
        xi = a * u[face].T + b * w[face].T + node0[face].T
        vi = norm[face].T * sim.ion_velocity - qm * ef[fc].T * (0.5 * dt) + tab[2:]
        x, v, cell = torch.cat([x, xi], 1), torch.cat([v, vi], 1), torch.cat([cell, fc])
        for d in range(3):
            v[d] += (qm * dt) * ef[cell, d]
            x[d] += v[d] * dt
        cell, lc = _walk(mesh, x, cell)
        live = cell != REMOVED
        charge = torch.zeros(hm.n_nodes, dtype=torch.float64, device=DEV)
        charge.index_add_(0, c2n[cell[live]].reshape(-1), lc[:, live].T.reshape(-1))
        charges.append(charge)
        it = FILL_STEPS + k
        removed = int((~live).sum())
        keep = cell.numel() - removed
        order = torch.arange(cell.numel(), device=DEV)
        periodic = case["fill"].endswith("Periodic")
        if removed and (case["fill"] == "HoleFill_All" or (periodic and it % case["period"])):
            holes, back = (~live).nonzero()[:, 0], live.nonzero()[:, 0].flip(0)
            r = min(removed, back.numel())
            holes, back = holes[:r], back[:r]
            ok = back > holes
            order[holes[ok]] = back[ok]
        elif removed and case["fill"].startswith("Sort"):
            order = torch.sort(cell, stable=True).indices
        elif removed:
            order = live.nonzero()[:, 0]  # a shuffle: its order is the framework's own
        order = order[:keep]
        x, v, lc, cell = x[:, order], v[:, order], lc[:, order], cell[order]
    # FP32 increments and weights move particles across faces now and then, and a shuffle has an
    # order of its own: only sums over particles have an exact value there.
    whole = case["precision"] == "f64" and not case["fill"].startswith("Shuffle")
    out = {"size": None, "p2c": None, "charge": charges[-1]}
    for name, a in (("pos", x), ("vel", v), ("lc", lc)):
        out[name] = torch.nn.functional.pad(a, (0, _capacity(case) - a.shape[1])) if whole else None
    if case["api"] == "host":
        out["charges"] = charges
    return out


def _exact_field(case: dict, seed: int):
    s = _prepare_field(case, seed)
    fd, k = s["fd"], FIELD
    n2e, c2n, dj = fd.d_node_to_eq.long(), fd.d_c2n.long().reshape(-1, 4), fd.d_det_j
    neq = fd.neq
    ion = s["charge"] * (s["spwt"] / s["vol"])
    e_all = k["n0"] * math.exp((0.0 - k["phi0"]) / k["kte"])
    free = n2e >= 0
    t1 = torch.zeros(neq, dtype=torch.float64, device=DEV)
    t1[n2e[free]] = (k["qe"] / k["eps0"]) * (ion[free] + e_all)
    t3 = -k["qe"] / k["eps0"] * e_all / k["kte"]
    f1, t2 = torch.zeros_like(t1), torch.zeros_like(t1)
    for v in range(4):
        e = n2e[c2n[:, v]]
        ok = e >= 0
        avg = 0.5 if v < 3 else -0.5
        f1.index_add_(0, e[ok], t1[e[ok]] * dj[ok] * avg)
        t2.index_add_(0, e[ok], t3 * dj[ok] * avg)
    row = torch.repeat_interleave(torch.arange(neq, device=DEV), fd.d_rowptr[1:] - fd.d_rowptr[:-1])
    col, val = fd.d_col.long(), fd.d_val.clone()
    on = row == col
    val[on] -= t2[row[on]]
    diag = val[on]
    jac = torch.sparse_csr_tensor(fd.d_rowptr, col, val, (neq, neq))
    b = -fd.d_f0[:neq] - f1
    y, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, stop = z.clone(), torch.dot(r, z), 1e-14 * float(b.norm())
    for it in range(20000):
        q = jac @ p
        alpha = rz / torch.dot(p, q)
        y += alpha * p
        r -= alpha * q
        if it % 20 == 19 and float(r.norm()) <= stop:
            break
        z = r / diag
        rz, old = torch.dot(r, z), rz
        p = z + (rz / old) * p
    d = -y
    pot = fd.d_bnd.clone()
    pot[free] += d[n2e[free]]
    sd = fd.d_c_sd.reshape(-1, 4, 3)
    ef = torch.zeros_like(s["ef"])
    ef[:, :3] = -(sd * pot[c2n][:, :, None]).sum(1)
    return {"density": ion, "potential": pot, "d": d, "f1": f1, "ef": ef}


def _cabana_current(q, u, mid):
    """The 12 accumulator values of a straight segment: half displacement u about midpoint mid."""
    v5 = q * u[0] * u[1] * u[2] * (1.0 / 3.0)
    out = []
    for a in range(3):
        s, dy, dz = q * u[a], mid[(a + 1) % 3], mid[(a + 2) % 3]
        out += [s * (1 - dy) * (1 - dz) + v5, s * (1 + dy) * (1 - dz) - v5,
                s * (1 - dy) * (1 + dz) - v5, s * (1 + dy) * (1 + dz) + v5]
    return torch.stack(out)


def _exact_cabana(case: dict, seed: int):
    if case["nx"] * case["ny"] * case["nz"] * case["nppc"] * case["steps"] > 1e8:
        return None
    s = _prepare_cabana(case, seed)
    cd, deck, mesh = s["cd"], s["deck"], s["mesh"]
    n, nc = cd.size, mesh.n_cells
    x, cell = s["start"]["pos"][:, :n].clone(), s["start"]["p2c"][:n].long()
    u = s["start"]["vel" if case["precision"] == "f64" else "vel32"][:, :n].to(torch.float64)
    f = torch.from_numpy(s["interp"]).to(DEV)
    c2f = torch.from_numpy(mesh.c2ngc).to(DEV).long()
    q = cd.weight[:n] * deck.qsp
    cdt = torch.tensor(deck.cdt_d, dtype=torch.float64, device=DEV)[:, None]
    k = deck.qdt_2mc
    for _ in range(case["steps"]):
        acc = torch.zeros((12, nc), dtype=torch.float64, device=DEV)
        r = f[cell].T
        e = k * torch.stack([r[0] + x[1] * r[1] + x[2] * (r[2] + x[1] * r[3]),
                             r[4] + x[2] * r[5] + x[0] * (r[6] + x[2] * r[7]),
                             r[8] + x[0] * r[9] + x[1] * (r[10] + x[0] * r[11])])
        b = torch.stack([r[12] + x[0] * r[13], r[14] + x[1] * r[15], r[16] + x[2] * r[17]])
        u = u + e
        v0 = k / torch.sqrt(1.0 + (u * u).sum(0))
        v1 = (b * b).sum(0)
        v2 = v0 * v0 * v1
        v3 = v0 * (1.0 + v2 * (1.0 / 3.0 + v2 * (2.0 / 15.0)))
        v4 = 2.0 * v3 / (1.0 + v1 * v3 * v3)
        w = u + v3 * torch.linalg.cross(u, b, dim=0)
        u = u + v4 * torch.linalg.cross(w, b, dim=0) + e
        s_all = u * cdt / torch.sqrt(1.0 + (u * u).sum(0))  # half displacement in cell units
        todo, disp, first = torch.arange(n, device=DEV), s_all.clone(), True
        while todo.numel():
            xs, ds, c = x[:, todo], disp[:, todo], cell[todo]
            sgn = torch.where(ds > 0, 1.0, -1.0).to(torch.float64)
            frac = torch.where(ds == 0, 3.4e38, (sgn - xs) / ds)
            if first:  # a particle that stays in its cell takes the whole displacement at once
                stay = ((xs + ds + ds).abs() <= 1.0).all(0)
                frac = torch.where(stay, 3.0, frac)
                first = False
            lim, axis = frac.min(0)
            ends = lim >= 2.0
            half = 0.5 * torch.clamp_max(lim, 2.0)
            d = ds * half
            mid = xs + d
            acc.index_add_(1, c, _cabana_current(q[todo], d, mid))
            x[:, todo] = mid + d
            disp[:, todo] = ds - d
            on = ~ends
            ax, dir_ = axis[on], sgn[:, on].gather(0, axis[on][None])[0]
            x[ax, todo[on]] = -dir_
            cell[todo[on]] = c2f[c[on], ax + torch.where(dir_ > 0, 3, 0)]
            todo = todo[on]
    return {"pos": x, "vel": u, "p2c": None, "acc": acc}


def _exact_advec(case: dict, seed: int):
    sides, ppcs = _advec_layout(case)
    if sum(s * s * p for s, p in zip(sides, ppcs)) > 1e8:
        return None
    s = _prepare_advec(case, seed)
    bd = s["bd"]
    pos = bd.pos.clone()
    for k, side in enumerate(sides):
        a, n = bd.part_offsets[k], bd.counts[k]
        for _ in range(case["steps"]):
            for d in range(2):
                x = pos[d, a:a + n] + bd.vel[d, a:a + n] * 0.5
                t = x + torch.trunc(x.abs() + 2.0) * float(side)
                pos[d, a:a + n] = t - float(side) * torch.trunc(t / float(side))
    return {"pos": pos, "mdir": None, "p2c": None}


def exact(case: dict, seed: int):
    return {"fempic": _exact_fempic, "field": _exact_field, "cabana": _exact_cabana,
            "advec": _exact_advec}[case["kind"]](case, seed)
