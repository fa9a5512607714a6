"""Timed cases of the library's compute paths, each through the call a user's program makes.

listed() names the ordinary work: one tendency of a small mesh, runs of RK4 steps of one model
(device and host states), batched ensembles in FP64 and FP32 with and without the learned
closure, the ICON triangle model, the horizontal operators of the 3-D MPAS dycore, and the
closure network's inference and training. draw(rng) gives further cases of the same ranges.
prepare() makes what a program holds before the call, run() is one pass and returns what it
computes, work() counts the bytes and operations a pass cannot do without, and exact() gives the
outputs in plain 64-bit torch.

States are smooth random height fields of the Earth's atmosphere (10 km depth, 100 m rms) with
the geostrophic wind of that field (40 m/s at most), on the unit sphere as the models take them.
The time step is a tenth of the gravity wave's Courant limit, so that a state can be stepped on
through thousands of passes.
"""
import functools
import math
import os

import numpy as np
import torch

import dmplex_b200 as d
from dmplex_b200 import closure as closure_net
from dmplex_b200 import icon, mpas
from dmplex_b200 import workloads as w
from dmplex_b200.coarsen import edge_geometry

DEV = "cuda"
CLOSURE = os.path.join(os.path.dirname(d.__file__), "data", "closure_hexagon6.npz")
PV = ("trisk", "gassmann", "gassmann_mean")
KE = ("cell", "vertex", "mixed")


def listed():
    return [
        # one right-hand side of a coarse mesh, as an outer time stepper calls it: latency
        {"name": "tendency-hex3", "kind": "tendency", "level": 3, "centroidal": True, "pv": "gassmann_mean",
         "ke": "mixed"},
        # the reference's small run: hexagon 5, the classic TRiSK scheme, 100 RK4 steps in one call
        {"name": "rk4-hex5", "kind": "rk4", "level": 5, "centroidal": True, "pv": "trisk", "ke": "cell",
         "steps": 100},
        # the drop-in run on hexagon 7 with the Gassmann flux and the vertex kinetic energy
        {"name": "rk4-hex7", "kind": "rk4", "level": 7, "centroidal": True, "pv": "gassmann", "ke": "vertex",
         "steps": 20},
        # a host program that keeps its state in its own memory and calls once per step
        {"name": "rk4-host-hex6", "kind": "host", "level": 6, "centroidal": True, "pv": "gassmann", "ke": "vertex",
         "steps": 1},
        # the largest single run: the mesh of the Galewsky jet example, half a million cells and more
        {"name": "rk4-hex8", "kind": "rk4", "level": 8, "centroidal": False, "pv": "trisk", "ke": "cell",
         "steps": 10},
        # uneven meshes in one ensemble: 64, 32 and 8 members on hexagons 5, 6 and 7
        {"name": "ensemble-3-levels", "kind": "ensemble", "groups": "5x64,6x32,7x8", "centroidal": True,
         "pv": "gassmann", "ke": "vertex", "bits": 64, "every": 0, "steps": 16},
        # the learned closure's ensemble: FP32 state, its network on every fourth step
        {"name": "ensemble-closure", "kind": "ensemble", "groups": "6x128", "centroidal": True, "pv": "trisk",
         "ke": "cell", "bits": 32, "every": 4, "steps": 16},
        # small groups of odd member counts
        {"name": "ensemble-odd", "kind": "ensemble", "groups": "5x13,6x5", "centroidal": True, "pv": "trisk",
         "ke": "mixed", "bits": 64, "every": 0, "steps": 32},
        # ICON triangles, the size of the R02B07 grid
        {"name": "icon-8", "kind": "icon", "level": 8, "damping": False, "gradient": "icon", "steps": 10},
        # the horizontal operators of a 30-layer baroclinic wave on hexagon 7
        {"name": "mpas-hex7x30", "kind": "mpas", "level": 7, "nlev": 30, "pv": "iap", "vertical": "iap",
         "ke": "cell", "solver": "five_band"},
        # the network on the (edge, member) rows of a 32-member hexagon-6 ensemble
        {"name": "mlp-forward", "kind": "forward", "rows": 3932160},
        # eight training batches of the closure's own size
        {"name": "mlp-train", "kind": "train", "rows": 65536, "batches": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("tendency", "rk4", "rk4", "host", "ensemble", "ensemble", "closure", "icon", "mpas", "forward",
                       "train"))
    scheme = {"pv": rng.choice(PV), "ke": rng.choice(KE), "centroidal": rng.random() < 0.5}
    if kind in ("tendency", "rk4", "host"):
        level = rng.randint(2, 7)
        steps = {"tendency": 1, "rk4": _log(rng, 1, 100 if level < 6 else 30), "host": _log(rng, 1, 8)}[kind]
        return {"kind": kind, "level": level, **scheme, "steps": steps}
    if kind == "ensemble":
        most = {3: 96, 4: 96, 5: 48, 6: 24, 7: 4}
        levels = rng.sample(sorted(most), rng.randint(1, 3))
        groups = ",".join(f"{n}x{_log(rng, 1, most[n])}" for n in sorted(levels))
        return {"kind": "ensemble", "groups": groups, **scheme, "bits": rng.choice((64, 64, 32)), "every": 0,
                "steps": _log(rng, 4, 32)}
    if kind == "closure":
        return {"kind": "ensemble", "groups": f"6x{_log(rng, 2, 96)}", "centroidal": True, "pv": "trisk",
                "ke": "cell", "bits": rng.choice((32, 32, 64)), "every": rng.choice((1, 2, 4)), "steps": 12}
    if kind == "icon":
        return {"kind": "icon", "level": rng.randint(3, 7), "damping": rng.random() < 0.5,
                "gradient": rng.choice(("icon", "centered")), "steps": _log(rng, 1, 40)}
    if kind == "mpas":
        vertical = rng.choice(("iap", "iap", "vector_invariant", "advective"))
        return {"kind": "mpas", "level": rng.randint(4, 6), "nlev": rng.randint(8, 60), "pv": rng.choice(("iap", "trisk")),
                "vertical": vertical, "ke": rng.choice(("cell", "vertex", "mixed")),
                "solver": "tridiagonal" if vertical == "advective" else rng.choice(("five_band", "tridiagonal"))}
    if kind == "forward":
        return {"kind": "forward", "rows": _log(rng, 200, 4_000_000)}
    return {"kind": "train", "rows": _log(rng, 1000, 131072), "batches": rng.randint(1, 8)}


# ---- meshes, models and states -------------------------------------------------------------


@functools.lru_cache(maxsize=4)
def _grid(level, centroidal):
    return d.TRiSKGrid(d.create_hexagon_mesh(level, centroidal=centroidal))


@functools.lru_cache(maxsize=4)
def _model(level, centroidal, pv, ke):
    return d.TRiSKShallowWater(_grid(level, centroidal), pv_flux=pv, kinetic_energy=ke, **w.si_parameters())


@functools.lru_cache(maxsize=2)
def _icon_model(level, damping, gradient):
    g = d.TRiSKGrid(d.hilbert_order(d.create_triangle_mesh(level)))
    nu = 0.0
    if damping:
        area = g.cell_areas[g.edge_cells - 1].mean(axis=1)
        nu = 0.0025 * area ** 2 / _icon_dt(g)
    return icon.ICONShallowWater(g, divergence_damping=nu, kinetic_gradient=gradient)


def _icon_dt(g):
    return 0.1 * float(g.dual_lengths.min())


@functools.lru_cache(maxsize=1)
def _mpas_tables(level, nlev, pv, vertical, ke, solver):
    g = d.TRiSKGrid(d.hilbert_order(d.create_hexagon_mesh(level)))
    v = mpas.vertical_grid(nlev, 30000.0)
    return v, mpas.mpas_tables(g, v, kinetic_energy=ke, pv_flux=pv, vertical_advection=vertical,
                               vertical_solver=solver)


@functools.lru_cache(maxsize=1)
def _mpas_operators(*key):
    return mpas.MPASOperators(_mpas_tables(*key)[1])


@functools.lru_cache(maxsize=6)
def _points(g):
    """The grid's geometry on the GPU, for the initial states."""
    t = {k: torch.from_numpy(getattr(g, k)).to(DEV) for k in ("centers", "vertices", "cell_areas", "primal_lengths")}
    t["ev"] = torch.from_numpy(g.edge_vertices - 1).to(DEV)
    return t


def _state(g, seed, rms=100.0):
    """[u; h] in SI units on the unit sphere: 24 random waves and their geostrophic wind."""
    p = _points(g)
    gen = torch.Generator().manual_seed(seed)
    k = torch.randn(24, 3, generator=gen, dtype=torch.float64) * 4
    phase = torch.rand(24, generator=gen, dtype=torch.float64) * 2 * math.pi
    amp = torch.randn(24, generator=gen, dtype=torch.float64)
    k, phase, amp = k.to(DEV), phase.to(DEV), amp.to(DEV)

    def field(x):
        return torch.cos(x @ k.T + phase) @ amp

    hc, area = field(p["centers"]), p["cell_areas"]
    mean = (area * hc).sum() / area.sum()
    scale = rms / torch.sqrt((area * (hc - mean) ** 2).sum() / area.sum())
    psi = field(p["vertices"]) * scale
    u = -(psi[p["ev"][:, 1]] - psi[p["ev"][:, 0]]) / p["primal_lengths"]
    u = u * (40.0 / u.abs().max() / w.EARTH_RADIUS)
    return torch.cat([u, w.MEAN_DEPTH + (hc - mean) * scale])


def _dt(g):
    return w.courant_dt(g, 0.1)


def _icon_state(g, seed):
    """The steady zonal flow of Williamson's second case with a random part, on the unit sphere."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    x, n, c = (torch.from_numpy(a).to(DEV) for a in (g.edge_points, g.edge_normals, g.centers))
    u = 0.2 * (-x[:, 1] * n[:, 0] + x[:, 0] * n[:, 1])
    h = 1 - (0.2 + 0.02) * c[:, 2] ** 2
    u = u + 1e-3 * torch.randn(len(u), generator=gen, device=DEV, dtype=torch.float64)
    h = h + 1e-3 * torch.randn(len(h), generator=gen, device=DEV, dtype=torch.float64)
    return torch.cat([u, h])


def _mpas_state(t, v, seed):
    """A stratified column on every cell with a perturbed wind and density."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    nlev, nc, ne = t["nlev"], t["nc"], t["ne"]

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float64)

    z = torch.from_numpy(v["z_full"]).to(DEV)[:, None]
    rho = 1.2 * torch.exp(-z / 8000.0) * (1 + 1e-3 * randn(nlev, nc))
    wind = torch.zeros(nlev + 1, nc, device=DEV, dtype=torch.float64)
    wind[1:nlev] = 0.1 * randn(nlev - 1, nc)
    return 10 * randn(nlev, ne), wind, rho, rho * (290.0 * torch.exp(z / 30000.0))


def _groups(case):
    return [tuple(int(x) for x in g.split("x")) for g in case["groups"].split(",")]


def _member_seed(seed, group, member):
    return (seed * 8 + group) * 1000 + member


@functools.lru_cache(maxsize=1)
def _saved_closure():
    z = np.load(CLOSURE)
    return z["params"], z["norm"]


def _batches(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n = case["rows"] * case.get("batches", 1)
    X = torch.randn(n, closure_net.NIN, generator=gen, device=DEV).to(torch.bfloat16)
    T = torch.randn(n, closure_net.NOUT, generator=gen, device=DEV) if case["kind"] == "train" else None
    return X, T


# ---- the cases -----------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("tendency", "rk4", "host"):
        m = _model(case["level"], case["centroidal"], case["pv"], case["ke"])
        y0 = _state(m.grid, seed)
        s.update(model=m, y0=y0, dt=_dt(m.grid), cache=d.RK4Cache(y0))
        if kind == "host":
            s["y"] = y0.cpu().numpy()
        else:
            s["y"] = torch.empty_like(y0)
    elif kind == "ensemble":
        groups = [(_model(n, case["centroidal"], case["pv"], case["ke"]), k) for n, k in _groups(case)]
        ens = d.Ensemble([(m, k, _dt(m.grid), 1 << 30) for m, k in groups], state_bits=case["bits"])
        for g, (m, members) in enumerate(groups):
            for k in range(members):
                ens.set_member(g, k, _state(m.grid, _member_seed(seed, g, k)))
        if case["every"]:
            params, norm = _saved_closure()
            s["net"] = closure_net.ClosureMLP(params)
            for g, (m, _) in enumerate(groups):
                ens.set_closure(g, s["net"], edge_geometry(m.grid), norm, every=case["every"])
        s.update(ensemble=ens, out=[torch.empty(k, m.state_size, device=DEV, dtype=torch.float64) for m, k in groups])
    elif kind == "icon":
        m = _icon_model(case["level"], case["damping"], case["gradient"])
        y0 = _icon_state(m.grid, seed)
        s.update(model=m, y0=y0, y=torch.empty_like(y0), dt=_icon_dt(m.grid))
    elif kind == "mpas":
        key = (case["level"], case["nlev"], case["pv"], case["vertical"], case["ke"], case["solver"])
        v, t = _mpas_tables(*key)
        ops = _mpas_operators(*key)
        s.update(ops=ops, fields=_mpas_state(t, v, seed), out=ops.work())
    else:
        X, T = _batches(case, seed)
        s.update(net=closure_net.ClosureMLP(seed=seed), X=X, T=T)
        if kind == "forward":
            s["Y"] = torch.empty(case["rows"], closure_net.NOUT, device=DEV)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "tendency":
        return d.tendency(state["y"], state["y0"], state["model"])
    if kind == "rk4":  # from the kept initial state
        state["y"].copy_(state["y0"])
    if kind in ("rk4", "host"):
        return d.rk4_step(state["y"], state["dt"], d.tendency, state["cache"], state["model"], nsteps=case["steps"])
    if kind == "ensemble":  # steps, then every member read out
        ens = state["ensemble"]
        ens.run(case["steps"])
        for g, y in enumerate(state["out"]):
            for k in range(len(y)):
                ens.get_member(g, k, y[k])
        return state["out"]
    if kind == "icon":
        state["y"].copy_(state["y0"])
        return state["model"].rk4_step(state["y"], state["dt"], case["steps"])
    if kind == "mpas":
        return state["ops"].slow_tendencies(*state["fields"], state["out"])
    if kind == "forward":
        return state["net"].forward(state["X"], state["Y"])
    n = case["rows"]
    losses = [state["net"].train_step(state["X"][b * n:(b + 1) * n], state["T"][b * n:(b + 1) * n], 1e-3)
              for b in range(case["batches"])]
    return losses, state["net"].params()


# ---- what a pass cannot do without ---------------------------------------------------------


def _counts(level):
    nc = 10 * 4 ** level + 2
    return nc, 3 * (nc - 2), 2 * (nc - 2)


def _scheme_work(level, pv, ke):
    """Bytes of the tables one tendency reads once (int32 indices, FP64 weights) and its
    floating-point operations."""
    nc, ne, nv = _counts(level)
    cell, vertex = ke != "vertex", ke != "cell"
    table = nv * (3 * 24 + (24 if vertex else 0) + (8 if pv == "trisk" else 0))
    table += ne * (8 + (24 if cell else 0) + (16 if vertex else 0) + (0 if pv == "trisk" else 24))
    table += nc * 6 * 12 * (2 + (1 if cell and vertex else 0))
    table += ne * ((120 if pv == "trisk" else 192 if pv == "gassmann" else 144) + 16)
    flops = nv * (11 + (9 if vertex else 0) + 2) + ne * (12 + (42 if pv == "trisk" else 39)) + nc * (30 + 12)
    return table, 8 * (nc + ne), flops


def work(case):
    kind = case["kind"]
    if kind == "tendency":
        table, state, flops = _scheme_work(case["level"], case["pv"], case["ke"])
        return {"bytes": table + 2 * state, "flops": flops}
    if kind in ("rk4", "host"):  # four tendencies a step, each of the whole previous stage state
        table, state, flops = _scheme_work(case["level"], case["pv"], case["ke"])
        return {"bytes": case["steps"] * 4 * (table + 2 * state),
                "flops": case["steps"] * (4 * flops + 13 * state / 8)}
    if kind == "ensemble":
        total = {"bytes": 0.0, "flops": 0.0}
        for level, members in _groups(case):
            table, state, flops = _scheme_work(level, case["pv"], case["ke"])
            state = state * members * case["bits"] // 64
            total["bytes"] += case["steps"] * 4 * (table + 2 * state)
            total["flops"] += case["steps"] * members * 4 * flops
            if case["every"]:  # the network's rows
                rows = _counts(level)[1] * members * -(-case["steps"] // case["every"])
                total["flops"] += rows * 2 * (24 * 64 + 64 * 64 + 64 * 2)
        return total
    if kind == "icon":
        nc, ne, nv = 20 * 4 ** case["level"], 30 * 4 ** case["level"], 10 * 4 ** case["level"] + 2
        table = ne * (112 + (8 if case["damping"] else 0)) + nc * 60 + nv * 72
        flops = ne * (8 + 4 + 4 + 13) + nc * 12 + nv * 12 + (ne * 12 + nc * 12 if case["damping"] else 0)
        return {"bytes": case["steps"] * 4 * (table + 16 * (nc + ne)),
                "flops": case["steps"] * (4 * flops + 13 * (nc + ne))}
    if kind == "mpas":
        nc, ne, nv = _counts(case["level"])
        nlev, vi, vk = case["nlev"], case["vertical"] != "advective", case["ke"] != "cell"
        fields = ne + 3 * nc + 3 * nc + (4 if vk else 3) * nv + (5 if vi else 4) * ne + nc
        metrics = 3 * nc + 2 * ne
        table = ne * (10 * 20 + 64) + nc * 6 * (28 + (12 if vk else 0)) + nv * 3 * (24 + (8 if vk else 0))
        flops = nlev * (nv * 14 + nc * (18 + 40 + 6 * 12) + ne * (20 + 40 + 40))
        return {"bytes": 8 * nlev * (fields + metrics) + table, "flops": flops}
    params = 4 * (24 * 64 + 64 + 64 * 64 + 64 + 128 + 2)
    mac = 24 * 64 + 64 * 64 + 64 * 2
    if kind == "forward":
        return {"bytes": case["rows"] * (48 + 8) + params, "flops": case["rows"] * 2 * mac}
    rows = case["rows"] * case["batches"]
    return {"bytes": rows * (48 + 8) + case["batches"] * 6 * params, "flops": rows * 6 * mac}


# ---- the outputs in 64 bits ----------------------------------------------------------------


def _tables(grid, pv, ke):
    t = d.model_tables(grid, pv_flux=pv, kinetic_energy=ke, **w.si_parameters())
    return _on_gpu(t)


def _on_gpu(t):
    """Index tables 0-based, everything on the GPU."""
    out = {}
    for k, v in t.items():
        if isinstance(v, np.ndarray):
            x = torch.from_numpy(np.ascontiguousarray(v)).to(DEV)
            out[k] = x.long() - 1 if v.dtype.kind == "i" else x
        else:
            out[k] = v
    return out


def _rows(weights, idx, x):
    """sum_k weights[:, k] x[idx[:, k]] for x (entities, members)."""
    s = torch.zeros(len(idx), x.shape[1], device=DEV, dtype=torch.float64)
    for k in range(idx.shape[1]):
        s += weights[:, k:k + 1] * x[idx[:, k]]
    return s


def _shallow_water(t, y, pv, ke, closure=None):
    """The tendency of y (ne + nc, members); closure: (dF, dq), added to the mass flux of the
    continuity equation and to the momentum tendency. Also the parts the closure's inputs use."""
    ne, nc = t["ne"], t["nc"]
    u, h = y[:ne], y[ne:]
    l, r = t["edge_cells"][:, 0], t["edge_cells"][:, 1]
    v0, v1 = t["edge_vertices"][:, 0], t["edge_vertices"][:, 1]
    zv = _rows(t["curl"], t["vertex_edges"], u)
    hv = _rows(t["vertex_height"], t["vertex_cells"], h)
    qv = (zv + t["coriolis"][:, None]) / hv
    K = torch.zeros(nc, y.shape[1], device=DEV, dtype=torch.float64)
    he = torch.zeros(ne, y.shape[1], device=DEV, dtype=torch.float64)
    if ke != "vertex":
        K = K + _rows(t["kinetic"], t["cell_edges"], u * u)
        he = he + t["edge_height"][:, :1] * h[l] + t["edge_height"][:, 1:] * h[r]
    if ke != "cell":
        K = K + _rows(t["vk_kites"], t["vk_cell_vertices"], _rows(t["vk_weights"], t["vertex_edges"], u * u))
        he = he + t["vk_height"][:, :1] * hv[v0] + t["vk_height"][:, 1:] * hv[v1]
    F = he * u
    B = K + t["gravity"] * h
    if pv == "trisk":
        q = (qv[v0] + qv[v1]) / 2
        du = torch.zeros_like(u)
        for k in range(t["trisk_edges"].shape[1]):
            e = t["trisk_edges"][:, k]
            du += t["trisk"][:, k:k + 1] * F[e] * (q + q[e])
        du = du / 2
    else:
        rh = t["rhombus"]
        q = (rh[:, :1] * zv[v0] + rh[:, 1:] * zv[v1] + t["g_coriolis"][:, None]) / (
            rh[:, :1] * hv[v0] + rh[:, 1:] * hv[v1])
        du = torch.zeros_like(u)
        for k in range(12):
            e = t["g_edges"][:, k]
            qk = (q + q[e]) / 2 if pv == "gassmann_mean" else q[t["g_pv_edges"][:, k]]
            du += t["g_weights"][:, k:k + 1] * F[e] * qk
    du = du - (B[r] - B[l]) * t["inverse_dual"][:, None]
    if closure is not None:
        F, du = F + closure[0], du + closure[1]
    return torch.cat([du, -_rows(t["divergence"], t["cell_edges"], F)]), qv, K


def _rk4(f, y, dt, first=None):
    k1 = f(y) if first is None else first
    k2 = f(y + dt / 2 * k1)
    k3 = f(y + dt / 2 * k2)
    k4 = f(y + dt * k3)
    return y + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _unpack(params):
    p = torch.as_tensor(np.asarray(params, dtype=np.float64), device=DEV)
    out, k = [], 0
    for _, shape in closure_net.SHAPES:
        n = int(np.prod(shape))
        out.append(p[k:k + n].reshape(shape))
        k += n
    return out


def _network(p, X):
    W1, b1, W2, b2, W3, b3 = p
    return _gelu(_gelu(X @ W1.T + b1) @ W2.T + b2) @ W3.T + b3


def _corrections(t, geometry, p, norm, y, qv, K):
    """The closure's mass-flux and momentum corrections of the state y, members one by one."""
    ne = t["ne"]
    u, h = y[:ne], y[ne:]
    l, r = t["edge_cells"][:, 0], t["edge_cells"][:, 1]
    v0, v1 = t["edge_vertices"][:, 0], t["edge_vertices"][:, 1]
    mean, scale, out = norm[:24], norm[24:48], norm[48:]
    dF, dq = torch.empty_like(u), torch.empty_like(u)
    for m in range(y.shape[1]):
        um, hm, qm, Km = u[:, m], h[:, m], qv[:, m], K[:, m]
        near = torch.where(t["trisk"] != 0, um[t["trisk_edges"]] - um[:, None], 0.0)
        pairs = [(x[a] + x[b]) / 2 if k == 0 else x[b] - x[a]
                 for x, a, b in ((hm, l, r), (qm, v0, v1), (Km, l, r)) for k in (0, 1)]
        X = torch.cat([um[:, None], near, torch.stack(pairs, 1), geometry], 1)
        Y = _network(p, (X - mean) * scale)
        dF[:, m], dq[:, m] = out[0] * Y[:, 0], out[1] * Y[:, 1]
    return dF, dq


def _exact_ensemble(case, seed):
    outs = []
    for g, (level, members) in enumerate(_groups(case)):
        grid = _grid(level, case["centroidal"])
        t = _tables(grid, case["pv"], case["ke"])
        y = torch.stack([_state(grid, _member_seed(seed, g, k)) for k in range(members)], 1)
        dt, corr = _dt(grid), None
        if case["every"]:
            params, norm = _saved_closure()
            p, norm = _unpack(params), torch.from_numpy(np.asarray(norm, dtype=np.float64)).to(DEV)
            geometry = torch.from_numpy(edge_geometry(grid).astype(np.float64)).to(DEV)
        for step in range(case["steps"]):
            if case["every"] and step % case["every"] == 0:
                _, qv, K = _shallow_water(t, y, case["pv"], case["ke"])
                corr = _corrections(t, geometry, p, norm, y, qv, K)
            y = _rk4(lambda x: _shallow_water(t, x, case["pv"], case["ke"], corr)[0], y, dt)
        outs.append(y.T.contiguous())
    return outs


def _exact_icon(case, seed):
    m = _icon_model(case["level"], case["damping"], case["gradient"])
    t, ne = _on_gpu(m.tables), m.ne
    l, r = t["edge_cells"][:, 0], t["edge_cells"][:, 1]
    g0, g1, invd = t["gradient"][:, 0], t["gradient"][:, 1], t["inverse_dual"]

    def rows(name, idx, x):
        return (t[name] * x[t[idx]]).sum(1)

    def tendency(y):
        u, h = y[:ne], y[ne:]
        v = rows("rbf", "rbf_edges", u)
        Ke = (u * u + v * v) / 2
        F = (t["edge_height"][:, 0] * h[l] + t["edge_height"][:, 1] * h[r]) * u
        K = rows("bilinear", "cell_edges", Ke)
        zv = rows("curl", "vertex_edges", u)
        zeta = zv[t["edge_vertices"]].mean(1)
        du = (t["edge_coriolis"] + zeta) * v - (Ke * (g0 - g1) + g1 * K[r] - g0 * K[l])
        du = du - t["gravity"] * (h[r] - h[l]) * invd
        if case["damping"]:
            D = -rows("divergence", "cell_edges", u)
            D = -rows("divergence", "cell_edges", (D[r] - D[l]) * invd)
            du = du - t["divergence_damping"] * (D[r] - D[l]) * invd
        return torch.cat([du, -rows("divergence", "cell_edges", F)])

    y, dt = _icon_state(m.grid, seed), _icon_dt(m.grid)
    for _ in range(case["steps"]):
        y = _rk4(tendency, y, dt)
    return y


def _exact_mpas(case, seed):
    v, host = _mpas_tables(case["level"], case["nlev"], case["pv"], case["vertical"], case["ke"], case["solver"])
    vn, wind, rho, rt = _mpas_state(host, v, seed)
    t = _on_gpu({k: x for k, x in host.items() if k != "trisk_index"})
    ti = torch.from_numpy(host["trisk_index"]).to(DEV).long() - 1
    n = host["nlev"]
    l, r = t["edge_cells"][:, 0], t["edge_cells"][:, 1]
    v0, v1 = t["edge_vertices"][:, 0], t["edge_vertices"][:, 1]
    ew, rh, invd = t["edge_weight"], t["rhombus"], t["inverse_dual"]

    def rows(weights, idx, x):  # x (levels, entities)
        s = torch.zeros(x.shape[0], len(idx), device=DEV, dtype=torch.float64)
        for k in range(idx.shape[1]):
            s += weights[:, k] * x[:, idx[:, k]]
        return s

    out = {"theta": rt / rho, "exner": (287.0 * rt / 1.0e5) ** (287.0 / (1004.0 - 287.0))}
    K = rows(t["kinetic"], t["cell_edges"], vn * vn)
    if host["vk_weights"] is not None:
        out["Kv"] = rows(t["vk_weights"], t["vertex_edges"], vn * vn)
        K = K + rows(t["vk_kites"], t["vk_cell_vertices"], out["Kv"])
    else:
        out["Kv"] = torch.zeros(n, host["nv"], device=DEV, dtype=torch.float64)
    z, h = rows(t["curl"], t["vertex_edges"], vn), rows(t["vertex_weight"], t["vertex_cells"], rho)
    out.update(zetav=z, rhov=h, qv=(z + t["coriolis"]) / h)
    if host["iap_pv"]:
        q = (rh[:, 0] * z[:, v0] + rh[:, 1] * z[:, v1] + t["edge_coriolis"]) / (
            rh[:, 0] * h[:, v0] + rh[:, 1] * h[:, v1])
    else:
        q = (out["qv"][:, v0] + out["qv"][:, v1]) / 2
    re = ew[:, 0] * rho[:, l] + ew[:, 1] * rho[:, r]
    F = re * vn
    out.update(qe=q, rhoe=re, Fs=F, eta=torch.zeros(n + 1, host["ne"], device=DEV, dtype=torch.float64))
    tw = torch.zeros(n + 1, host["nc"], device=DEV, dtype=torch.float64)
    wi, inner = wind[1:n], torch.zeros(n - 1, host["nc"], device=DEV, dtype=torch.float64)
    massweighted = host["vertical"] == 2
    if host["vertical"] > 0:
        dzh = t["dzh_cells"]
        Kw = K + (dzh[:-1] * wind[:-1] ** 2 + dzh[1:] * wind[1:] ** 2) / (4 * t["dz_cells"])
        eta = (vn[1:] - vn[:-1]) / t["dzh_edges"][1:n] - (wi[:, r] - wi[:, l]) * invd
        out["eta"][1:n] = eta
        wl = t["wlow"][1:n]
        for k in range(t["cell_edges"].shape[1]):
            e = t["cell_edges"][:, k]
            a, b = (re[:-1][:, e], re[1:][:, e]) if massweighted else (1.0, 1.0)
            inner += t["inner"][:, k] * eta[:, e] * (a * vn[:-1][:, e] + b * vn[1:][:, e]) / (2 * (wl * a + (1 - wl) * b))
        below = K if host["five_band"] else Kw
        tw[1:n] = inner - (below[1:] - below[:-1]) / dzh[1:n]
        K = Kw
    else:
        for k in range(t["cell_edges"].shape[1]):
            e = t["cell_edges"][:, k]
            inner += t["kinetic"][:, k] * (vn[:-1][:, e] + vn[1:][:, e]) * (wi[:, r[e]] - wi[:, l[e]]) * invd[e]
        dz = t["dz_cells"]
        tw[1:n] = -inner - wi * (wind[2:] - wind[:-2]) / (dz[:-1] + dz[1:])
    s = torch.zeros_like(vn)
    for k in range(ti.shape[1]):
        s += t["trisk"][:, k] * F[:, ti[:, k, 0]] * (q[:, ti[:, k, 1]] + q[:, ti[:, k, 2]])
    th, pe = out["theta"], out["exner"]
    s = s - invd * (K[:, r] - K[:, l])
    s = s - 1004.0 * (ew[:, 0] * th[:, l] + ew[:, 1] * th[:, r]) * (pe[:, r] - pe[:, l]) * invd
    if host["vertical"] > 0:
        ml, mr = torch.ones_like(wi[:, l]), torch.ones_like(wi[:, l])
        if massweighted:
            at = t["wlow"][1:n] * rho[:-1] + (1 - t["wlow"][1:n]) * rho[1:]
            ml, mr = at[:, l], at[:, r]
        W = torch.zeros(n + 1, host["ne"], device=DEV, dtype=torch.float64)
        W[1:n] = (ew[:, 0] * ml * wi[:, l] + ew[:, 1] * mr * wi[:, r]) / (ew[:, 0] * ml + ew[:, 1] * mr)
        X = t["dzh_edges"] * out["eta"] * W
        s = s - (X[:-1] + X[1:]) / (2 * t["dz_edges"])
    else:
        we = (wind[:-1][:, l] + wind[:-1][:, r] + wind[1:][:, l] + wind[1:][:, r]) / 4
        half = torch.cat([vn[:1], (vn[:-1] + vn[1:]) / 2, vn[-1:]])
        s = s - we * (half[1:] - half[:-1]) / t["dz_edges"]
    out.update(K=K, tw=tw, tvn=s)
    return out


def _exact_train(case, seed):
    X, T = _batches(case, seed)
    X, T = X.double(), T.double()
    p = _unpack(closure_net.he_init(seed))
    first, second = [torch.zeros_like(x) for x in p], [torch.zeros_like(x) for x in p]
    losses, n = [], case["rows"]
    for b in range(case["batches"]):
        q = [x.clone().requires_grad_() for x in p]
        with torch.enable_grad():
            loss = ((_network(q, X[b * n:(b + 1) * n]) - T[b * n:(b + 1) * n]) ** 2).sum() / n
            grads = torch.autograd.grad(loss, q)
        losses.append(float(loss))
        for x, g, a, v in zip(p, grads, first, second):
            a.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).add_(g * g, alpha=0.001)
            x.sub_(1e-3 * (a / (1 - 0.9 ** (b + 1))) / (torch.sqrt(v / (1 - 0.999 ** (b + 1))) + 1e-8))
    return losses, torch.cat([x.reshape(-1) for x in p])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("tendency", "rk4", "host"):
        grid = _grid(case["level"], case["centroidal"])
        t = _tables(grid, case["pv"], case["ke"])
        y = _state(grid, seed)[:, None]

        def f(x):
            return _shallow_water(t, x, case["pv"], case["ke"])[0]

        if kind == "tendency":
            return f(y)[:, 0]
        for _ in range(case["steps"]):
            y = _rk4(f, y, _dt(grid))
        return y[:, 0]
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    if kind == "icon":
        return _exact_icon(case, seed)
    if kind == "mpas":
        return _exact_mpas(case, seed)
    if kind == "forward":
        X, _ = _batches(case, seed)
        p = _unpack(closure_net.he_init(seed))
        return torch.cat([_network(p, x.double()) for x in X.split(1 << 18)])
    return _exact_train(case, seed)
