"""The work a user of the solver has it do, as cases that can be timed: RK4 marching of single grids with
snapshots to the host, a step-by-step loop, batched ensembles, x-slab groups, the discrete adjoint (forward
and backward) and the end-of-step metrics of caller-owned fields.

listed(): the cases; draw(rng): one more of the same ranges; prepare(case, seed): what a program has in hand
before the call; run(state): one pass through the public entry points; work(case): the bytes and operations of
one pass; exact(case, seed): what run returns, from plain torch in 64 bits.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "3d-ns-fsi_b200"))

import nsfsi  # noqa: E402

CONSERVED = 0x1F  # rho, rho_u, rho_v, rho_w, rho_E
SAVED = 0x3E1     # the fields the case files save: rho, u, v, w, p, T


def listed():
    return [
        # Simulation::run as the reference's main has it: one step, read t / dt, next step; the smallest grid
        {"name": "loop_sphere_32", "kind": "loop", "flow": "sphere", "ni": 32, "nj": 32, "nk": 32, "steps": 10},
        # the default ConfigFile and its hard-coded cylinder case (inlet / outlet x, symmetry y, one layer in z)
        {"name": "march_cylinder_161x83x3", "kind": "march", "flow": "shipped", "ni": 161, "nj": 83, "nk": 3,
         "steps": 100, "mask": SAVED},
        # one sphere in a channel, 100 steps between snapshots of the saved fields
        {"name": "march_sphere_48", "kind": "march", "flow": "sphere", "ni": 48, "nj": 48, "nk": 48, "steps": 100,
         "mask": SAVED},
        # odd node counts, symmetry walls in y, two spheres
        {"name": "march_walls_75x53x61", "kind": "march", "flow": "walls", "ni": 75, "nj": 53, "nk": 61, "steps": 50,
         "mask": CONSERVED},
        # Taylor-Green vortex at the size below the benchmark's
        {"name": "march_tgv_128", "kind": "march", "flow": "tgv", "ni": 128, "nj": 128, "nk": 128, "steps": 20,
         "mask": CONSERVED},
        # sixteen spheres in a long channel
        {"name": "march_spheres16_256x128", "kind": "march", "flow": "spheres16", "ni": 256, "nj": 128, "nk": 128,
         "steps": 20, "mask": CONSERVED},
        # the benchmark workload, a snapshot of the saved fields every 20 steps
        {"name": "march_tgv_256", "kind": "march", "flow": "tgv", "ni": 256, "nj": 256, "nk": 256, "steps": 20,
         "mask": SAVED},
        # the batched-ensemble workload: 64 sphere flows of five grid shapes
        {"name": "ensemble_64", "kind": "ensemble", "members": 64, "steps": 20},
        # gradient with every step on the tape (the default), the gradient workload's grid
        {"name": "adjoint_64_tape", "kind": "adjoint", "ni": 64, "nj": 64, "nk": 64, "steps": 100, "avg": 25,
         "tape": True},
        # gradient from 20 checkpoints (what a grid too large for a tape runs), uneven grid
        {"name": "adjoint_45x37x50_checkpoints", "kind": "adjoint", "ni": 45, "nj": 37, "nk": 50, "steps": 60,
         "avg": 15, "tape": False},
        # one grid in two x-slabs on one device
        {"name": "slabs2_tgv_96", "kind": "slab", "flow": "tgv", "ni": 96, "nj": 96, "nk": 96, "steps": 20, "slabs": 2},
        # end-of-step metrics of fields a host framework owns
        {"name": "metrics_192", "kind": "metrics", "flow": "tgv", "ni": 192, "nj": 192, "nk": 192},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["march", "march", "march", "loop", "ensemble", "adjoint", "slab", "metrics"])
    if kind == "ensemble":
        return {"kind": kind, "members": _log(rng, 4, 64), "steps": rng.randint(5, 20)}
    if kind == "adjoint":
        return {"kind": kind, "ni": _log(rng, 28, 64), "nj": _log(rng, 28, 64), "nk": _log(rng, 28, 64),
                "steps": rng.randint(20, 80), "avg": rng.randint(1, 20), "tape": rng.random() < 0.5}
    if kind == "metrics":
        return {"kind": kind, "flow": "tgv", "ni": _log(rng, 24, 250), "nj": _log(rng, 24, 250),
                "nk": _log(rng, 24, 250)}
    flow = "tgv" if kind == "slab" else rng.choice(["tgv", "sphere", "walls", "shipped"])
    c = {"kind": kind, "flow": flow}
    if flow == "shipped":
        c.update(ni=_log(rng, 81, 400), nj=_log(rng, 41, 200), nk=_log(rng, 3, 12))
    else:
        top = 72 if kind == "loop" else 250
        c.update(ni=_log(rng, 28, top), nj=_log(rng, 28, top), nk=_log(rng, 28, top))
    nodes = c["ni"] * c["nj"] * c["nk"]
    # no more node-steps than the largest listed grid's, and no more small steps than its time
    c["steps"] = 10 if kind == "loop" else max(5, min(100, int(2.5e8 / nodes)))
    if kind == "march":
        c["mask"] = rng.choice([CONSERVED, SAVED])
    if kind == "slab":
        c["slabs"] = rng.randint(2, 4)
    return c


def _nodes(case):
    return case["ni"] * case["nj"] * case["nk"]


def _config(case, seed):
    """The case's configuration; the seed moves the Mach and Reynolds numbers and the initial noise."""
    r = random.Random(seed)
    flow = case["flow"]
    n = [case["ni"], case["nj"], case["nk"]]
    if flow == "shipped":
        c = nsfsi.config_defaults()
        c.stop_criterion = 0
        c.lz = 0.05 * (n[2] - 2)
    else:
        c = nsfsi.config_load(nsfsi.case_path({"tgv": "tgv256", "spheres16": "spheres16"}.get(flow, "sphere48")))
    c.NI, c.NJ, c.NK = n
    if flow in ("sphere", "walls", "spheres16"):  # a frequent density filter, as coarse flows past bodies are run
        c.n_filter_intervals, c.n_filter_change_times = 1, 0
        c.filter_intervals[0] = 4 if flow == "walls" else 5
    if flow in ("sphere", "walls", "gradient"):
        walls = flow == "walls"
        cells = [n[0] - 1, n[1] - (3 if walls else 2), n[2] - 2]
        h = 1.0 / min(cells[1:])
        c.lx, c.ly, c.lz = (h * m for m in cells)
        rad = max(3.0 * h, 0.1 * min(c.lx, c.ly, c.lz))
        c.spheres[0] = nsfsi.Sphere(0.4 * c.lx, 0.5 * c.ly, 0.5 * c.lz, rad)
        if walls:
            for side in range(2):
                c.bc[1][side] = nsfsi.BC["symmetry"]
            if n[0] >= 64:
                c.n_spheres = 2
                c.spheres[0] = nsfsi.Sphere(0.3 * c.lx, 0.5 * c.ly, 0.5 * c.lz, 3.0 * h)
                c.spheres[1] = nsfsi.Sphere(0.7 * c.lx, 0.5 * c.ly, 0.5 * c.lz, 3.5 * h)
    c.stop_time_level = case.get("steps", 1)
    c.machine_precision_buffer = float(np.finfo(np.float64).eps) * (c.lx + c.ly + c.lz)
    c.m0 *= 1 + 0.1 * (r.random() - 0.5)
    c.re *= 1 + 0.1 * (r.random() - 0.5)
    c.seed = seed
    return c


def _pinned(rows, n):
    return torch.zeros((rows, n), dtype=torch.float64, pin_memory=True)


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "metrics":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = _nodes(case)
        new = 0.05 * torch.randn((5, n), dtype=torch.float64, device="cuda", generator=g)
        new[0] *= 0.1
        new[4] = 0.02 * new[4] + new[1:4].square().sum(0) / 2
        old = new + 1e-3 * torch.randn((5, n), dtype=torch.float64, device="cuda", generator=g)
        return {"case": case, "cfg": _config(case, seed), "old": old, "new": new,
                "out": torch.zeros(6, dtype=torch.float64, device="cuda")}
    if kind == "ensemble":
        cfgs = nsfsi.ensemble_configs(n=case["members"], steps=case["steps"])
        r = random.Random(seed)
        for c in cfgs:
            c.seed += seed
            c.n_filter_intervals, c.n_filter_change_times = 1, 0
            c.filter_intervals[0] = 5
            c.m0 *= 1 + 0.05 * (r.random() - 0.5)
        e = nsfsi.Ensemble(cfgs)
        return {"case": case, "ensemble": e, "host": [_pinned(5, int(c.NI * c.NJ * c.NK)) for c in cfgs]}
    if kind == "adjoint":
        c = _config(dict(case, flow="gradient"), seed)
        s = nsfsi.Solver(c)
        s.adj_configure(case["avg"], 20)
        if not case["tape"]:
            s.adj_tape_limit(0)
        g = np.random.default_rng(seed)
        v = 1e-4 * g.standard_normal((3, s.N))
        v[0] += c.m0
        u0 = np.zeros((5, s.N))
        u0[1:4] = v
        u0[4] = 0.5 * (v * v).sum(0)
        return {"case": case, "solver": s, "u0": u0,
                "inflow": 1 + 0.01 * g.standard_normal((case["nj"], case["nk"]))}
    c = _config(case, seed)
    if kind == "slab":
        return {"case": case, "group": nsfsi.SlabGroup(c, case["slabs"]), "host": _pinned(5, _nodes(case))}
    mask = case.get("mask", CONSERVED)
    return {"case": case, "solver": nsfsi.Solver(c), "mask": mask, "host": _pinned(bin(mask).count("1"), _nodes(case)),
            "ticket": ctypes.c_uint64()}


def run(state):
    kind = state["case"]["kind"]
    L = nsfsi.lib()
    if kind == "march":  # the steps, a snapshot that travels while the next steps march, and the time reached
        s = state["solver"]
        s.march(state["case"]["steps"])
        s._check(L.nsf_download_async(s.h, state["mask"], _ptr(state["host"]), ctypes.byref(state["ticket"])))
        t, level, dt = s.time()
        return {"fields": state["host"], "t": t, "dt": dt}
    if kind == "loop":
        s = state["solver"]
        for _ in range(state["case"]["steps"]):
            s.march(1)
            t, level, dt = s.time()
        s._check(L.nsf_download(s.h, state["mask"], _ptr(state["host"])))
        return {"fields": state["host"], "t": t, "dt": dt}
    if kind == "ensemble":
        e = state["ensemble"]
        e.march(state["case"]["steps"])
        for m, host in enumerate(state["host"]):
            s = e.member(m)
            s._check(L.nsf_download(s.h, CONSERVED, _ptr(host)))
        return state["host"]
    if kind == "adjoint":
        s = state["solver"]
        J = s.adj_forward(state["u0"], state["inflow"])
        g_inflow, g_u0 = s.adj_backward()
        return {"J": J, "g_inflow": g_inflow, "g_u0": g_u0}
    if kind == "slab":
        g = state["group"]
        g.march(state["case"]["steps"])
        g._check(L.nsf_slab_group_download(g.h, CONSERVED, _ptr(state["host"])))
        return state["host"]
    st = L.nsf_step_metrics_noalloc(ctypes.byref(state["cfg"]), state["old"].data_ptr(), state["new"].data_ptr(), None,
                                    state["out"].data_ptr(), torch.cuda.current_stream().cuda_stream)
    if st:
        raise nsfsi.NsfError(st, "nsf_step_metrics_noalloc")
    return state["out"]


# Per node and RK4 step, stages as separate passes over fields that do not fit on the chip: stage 1 reads U0 and
# writes U1 (k1 = 2 (U1 - U0) / dt), stage 2 reads U0, U1 and writes U2 and the weighted sum of slopes, stage 3
# reads U0, U2 and writes U3, stage 4 reads U0, U3 and the sum and writes the new state: 13 passes over five
# doubles. Operations: about 400 a stage.
STEP_BYTES = 13 * 40
STEP_FLOPS = 1600


def work(case):
    kind = case["kind"]
    if kind == "metrics":
        return {"bytes": 80 * _nodes(case), "flops": 70 * _nodes(case)}
    if kind == "ensemble":
        n = sum(int(c.NI * c.NJ * c.NK) for c in nsfsi.ensemble_configs(n=case["members"], steps=case["steps"]))
    else:
        n = _nodes(case)
    steps = case["steps"]
    if kind == "adjoint":
        # the forward run, then per stage of the backward run: the stage input and the adjoint state read, the
        # adjoint state written; about three times a stage's operations
        return {"bytes": n * steps * (STEP_BYTES + 4 * 120), "flops": n * steps * 4 * STEP_FLOPS}
    fields = bin(case.get("mask", CONSERVED)).count("1")
    return {"bytes": n * (steps * STEP_BYTES + 16 * fields), "flops": n * steps * STEP_FLOPS}


# ---------------------------------------------------------------------------------------------------------
# The scheme in plain torch, 64 bits, for fully periodic boxes without bodies.
def _prims(c, U):
    r = 1 + U[0]
    v = [U[1] / r, U[2] / r, U[3] / r]
    p = (c.gamma - 1) * (U[4] - 0.5 * r * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2))
    T = (c.gamma * p - U[0]) / r
    sc = 1 + c.sutherlands_c2 / c.t0
    mu = (1 + T) ** 1.5 * sc / (c.re * (T + sc))
    return v, p, T, mu


def _time_step(c, d, U, P):
    v, p, _, mu = P
    r = 1 + U[0]
    a = torch.sqrt((1 + c.gamma * p) / r)
    conv = abs(c.conv_stability_limit) / sum(float((a + v[b].abs()).max()) / d[b] for b in range(3))
    nu = float((mu / r).max()) * max(4 / 3, c.gamma / c.pr)
    return min(conv, abs(c.visc_stability_limit) / (nu * sum(1 / h ** 2 for h in d)))


def _rhs(c, d, U, P):
    """Central differences D_a and face terms F_a of the five equations (second order, conservative)."""
    v, p, T, mu = P
    kappa = mu / ((c.gamma - 1) * c.pr)

    def D(a, f):
        return torch.roll(f, -1, a) - torch.roll(f, 1, a)

    def F(a, w, f):  # (w_P + w_E)(f_E - f_P) - (w_W + w_P)(f_P - f_W)
        e = (w + torch.roll(w, -1, a)) * (torch.roll(f, -1, a) - f)
        return e - torch.roll(e, 1, a)

    grad = [[D(a, v[b]) for b in range(3)] for a in range(3)]
    H = 1 / (c.gamma - 1) + U[4] + p
    out = [-sum(D(a, U[1 + a]) / (2 * d[a]) for a in range(3))]
    for m in range(3):
        k = -D(m, p) / (2 * d[m])
        for a in range(3):
            k = k - D(a, U[1 + m] * v[a]) / (2 * d[a]) + F(a, mu, v[m]) * ((2 / 3 if a == m else 1 / 2) / d[a] ** 2)
            if a != m:
                k = k - D(m, mu * grad[a][a]) / (6 * d[a] * d[m]) + D(a, mu * grad[m][a]) / (4 * d[a] * d[m])
        out.append(k)
    k = 0
    for a in range(3):
        k = k - D(a, H * v[a]) / (2 * d[a]) + F(a, kappa, T) / (2 * d[a] ** 2)
        for b in range(3):
            w = mu * v[b]
            k = k + F(a, w, v[b]) * ((2 / 3 if a == b else 1 / 2) / d[a] ** 2)
            if a != b:
                k = k - D(a, v[a] * mu * grad[b][b]) / (6 * d[a] * d[b]) + D(a, w * grad[b][a]) / (4 * d[a] * d[b])
    out.append(k)
    return out


def exact(case, seed):
    """run's result for Taylor-Green boxes and metrics; None where bodies or open faces take part."""
    if case["kind"] == "metrics":
        s = prepare(case, seed)
        c, old, new = s["cfg"], s["old"], s["new"]
        n = [case["ni"], case["nj"], case["nk"]]
        d = [L / (m - 2) for L, m in zip((c.lx, c.ly, c.lz), n)]
        diff = (old - new).reshape(5, *n)[:, 1:-1, 1:-1, 1:-1]
        norms = [math.sqrt(d[0] * d[1] * d[2] * float(f.square().sum())) for f in diff]
        return torch.tensor(norms + [_time_step(c, d, new, _prims(c, new))], dtype=torch.float64)
    if case.get("flow") != "tgv":
        return None
    c = _config(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = [case["ni"] - 2, case["nj"] - 2, case["nk"] - 2]
    if dev == "cpu" and n[0] * n[1] * n[2] * case["steps"] > 1e7:
        return None
    d = [L / m for L, m in zip((c.lx, c.ly, c.lz), n)]
    X = [(torch.arange(m, dtype=torch.float64, device=dev) * h).reshape([-1 if b == a else 1 for b in range(3)])
         for a, (m, h) in enumerate(zip(n, d))]
    M = c.m0
    u = M * torch.sin(X[0]) * torch.cos(X[1]) * torch.cos(X[2])
    v = -M * torch.cos(X[0]) * torch.sin(X[1]) * torch.cos(X[2])
    p = M * M / 16 * (torch.cos(2 * X[0]) + torch.cos(2 * X[1])) * (torch.cos(2 * X[2]) + 2)
    rho = c.gamma * p
    U = [rho, (1 + rho) * u, (1 + rho) * v, torch.zeros_like(u), p / (c.gamma - 1) + (1 + rho) / 2 * (u * u + v * v)]
    t, dt = 0.0, _time_step(c, d, U, _prims(c, U))
    for level in range(case["steps"]):
        P = _prims(c, U)  # of the unfiltered density
        used = sum(t > c.filter_change_times[q] for q in range(c.n_filter_change_times))
        if used < c.n_filter_intervals and (level + 1) % c.filter_intervals[used] == 0:
            U = [(6 * U[0] + sum(torch.roll(U[0], q, a) for a in range(3) for q in (1, -1))) / 12] + U[1:]
        k1 = _rhs(c, d, U, P)
        V = [a + dt / 2 * b for a, b in zip(U, k1)]
        k2 = _rhs(c, d, V, _prims(c, V))
        V = [a + dt / 2 * b for a, b in zip(U, k2)]
        k3 = _rhs(c, d, V, _prims(c, V))
        V = [a + dt * b for a, b in zip(U, k3)]
        k4 = _rhs(c, d, V, _prims(c, V))
        U = [a + dt / 6 * (w + 2 * x + 2 * y + z) for a, w, x, y, z in zip(U, k1, k2, k3, k4)]
        t, dt = t + dt, _time_step(c, d, U, _prims(c, U))
    w, p, T, mu = _prims(c, U)
    every = U + w + [p, T, mu, mu / ((c.gamma - 1) * c.pr)]
    mask = case.get("mask", CONSERVED)
    rows = [torch.nn.functional.pad(f[None, None], (1,) * 6, mode="circular").reshape(-1).cpu()
            for q, f in enumerate(every) if mask >> q & 1]
    fields = torch.stack(rows)
    return fields if case["kind"] == "slab" else {"fields": fields, "t": t, "dt": dt}
