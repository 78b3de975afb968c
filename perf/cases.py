"""Performance cases: what a user's program has this library do, through its public entry points.

A stepping case holds one resident ``mpm2d.Simulation`` (or ``Batch``).  One pass advances it to its next
output frame and reads that frame (the driver's thirteen particle fields) into pinned host buffers the
program keeps, so consecutive passes continue one run, as a driver's loop does.  The FP64 form's frame is
FP64; a mixed form's is handed on in FP32, the type of the particle state it holds.  The adjoint case is
one forward-and-backward evaluation of a gradient, the sort case one call of the allocation-free cell sort
on device arrays.

Starts are states out of the middle of a run: a lattice fill whose particles have drifted off it, a
lithostatic stress around the yield ratio (elastic and flowing regions both occur), a smooth velocity field
with small scatter, and the full body force.  ``exact`` is the same step in plain FP64 torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpm-2d_gb300"))
import mpm2d  # noqa: E402
import scenes  # noqa: E402

# the driver's output frame (write_frame, src/writer.c:169-201)
FRAME = ("m", "v", "x", "y", "vx", "vy", "sxx", "sxy", "syy", "ux", "uy", "state9", "state10")
ADJOINT_STATE = ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy", "Tzz")
RHO, GRAVITY = 2450.0, -9.8
# material constants where a scene sets none: the scenes' E and nu, the plugins' mu(I) constants
CONSTANTS = {"E": 1e6, "nu": 0.3, "mu_s": 0.3819, "mu_2": 0.6435, "I0": 0.278, "grains_rho": 2450.0,
             "grains_d": 5.3e-4, "rho_critical": 1485.0, "A": 0.48}
THETA = ("mu_s", "mu_2", "I0", "E")


def listed():
    return [
        # the smallest call: the plain isolin block (4096 particles, 65^2 nodes), latency-bound
        {"name": "block_4k_fp64", "kind": "step", "shape": "block", "cells": 64, "material": "isolin",
         "precision": "fp64", "scheme": "usl", "dt": 1e-5, "drift": 0.13, "steps": 100, "calls": 1},
        # a small granular column in the reference's other scheme (MUSL)
        {"name": "column_2k_musl", "kind": "step", "shape": "column", "cells": 64, "material": "g_local_mu2",
         "precision": "fp64", "scheme": "musl", "dt": 1e-5, "drift": 0.6, "steps": 50, "calls": 1},
        # the 512 x 128 column collapse driven as the reference's driver does it, one step per call
        {"name": "collapse_31k_single", "kind": "step", "shape": "collapse", "cells": 512,
         "material": "g_local_mu2", "precision": "fp64", "scheme": "usl", "dt": 2e-6, "drift": 0.6, "steps": 50,
         "calls": 50},
        # the fine 1024 x 256 column collapse
        {"name": "collapse_125k_fp64", "kind": "step", "shape": "collapse", "cells": 1024,
         "material": "g_local_mu2", "precision": "fp64", "scheme": "usl", "dt": 2e-6, "drift": 0.6, "steps": 40,
         "calls": 1},
        # the headline workload (1 048 576 particles, 513^2 nodes), plain FP64 form
        {"name": "box_1m_fp64", "kind": "step", "shape": "box", "cells": 512, "material": "g_local_mu2",
         "precision": "fp64", "scheme": "usl", "dt": 2e-6, "drift": 0.1, "steps": 20, "calls": 1},
        # the same workload in the mixed form
        {"name": "box_1m_mixed", "kind": "step", "shape": "box", "cells": 512, "material": "g_local_mu2",
         "precision": "mixed", "scheme": "usl", "dt": 2e-6, "drift": 0.1, "steps": 200, "calls": 1},
        # a silo discharge on an odd grid (387^2 elements, 474 k particles), mixed form with FP64 nodal sums
        {"name": "silo_474k_f64node", "kind": "step", "shape": "silo", "cells": 387, "material": "g_local_mu2",
         "precision": "mixed_f64node", "scheme": "usl", "dt": 2e-6, "drift": 0.6, "steps": 100, "calls": 1},
        # the nonlocal silo (835 996 particles): an implicit fluidity solve every step
        {"name": "nonlocal_836k_fp64", "kind": "step", "shape": "silo", "cells": 512,
         "material": "g_nonlocal_mu2", "precision": "fp64", "scheme": "usl", "dt": 1e-6, "drift": 0.1, "steps": 10,
         "calls": 1},
        # a smaller, odd nonlocal silo in the mixed form
        {"name": "nonlocal_53k_mixed", "kind": "step", "shape": "silo", "cells": 129,
         "material": "g_nonlocal_mu2", "precision": "mixed", "scheme": "usl", "dt": 5e-6, "drift": 0.1, "steps": 20,
         "calls": 1},
        # a parameter study: uneven silo and heap runs stepped together (mixed form)
        {"name": "ensemble_32", "kind": "batch", "members": 32, "fleet": 1, "dt": 5e-6, "drift": 0.6, "steps": 50},
        # calibration: gradient of a loss on the final positions (65 536 particles)
        {"name": "adjoint_65k", "kind": "adjoint", "cells": 256, "ppc": 4, "dt": 2e-6, "drift": 0.1, "steps": 16,
         "every": 8},
        # the cell sort called from a host program that owns its device memory
        {"name": "cell_sort_125k", "kind": "sort", "n": 125563, "elements": 262144, "outside": 0.01},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["batch", "adjoint", "sort"])
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(3, 32), "fleet": rng.randint(2, 10**6), "dt": 5e-6,
                "drift": 0.6, "steps": rng.randint(10, 50)}
    if kind == "adjoint":
        return {"kind": kind, "cells": _log(rng, 64, 256), "ppc": rng.choice([2, 3, 4]), "dt": 2e-6, "drift": 0.1,
                "steps": rng.randint(5, 16), "every": rng.choice([3, 5, 8])}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 500, 1 << 20), "elements": _log(rng, 500, 1 << 19),
                "outside": round(rng.uniform(0.0, 0.2), 3)}
    shape = rng.choice(["block", "column", "collapse", "box", "silo"])
    precision = rng.choice(["fp64", "fp64", "mixed", "mixed_f64node"])
    cells = _log(rng, 32, 1024 if shape == "collapse" else 512)
    nonlocal_ = shape == "silo" and rng.random() < 0.6
    material = "g_nonlocal_mu2" if nonlocal_ else "isolin" if shape == "block" else "g_local_mu2"
    scheme = "musl" if precision == "fp64" and not nonlocal_ and rng.random() < 0.2 else "usl"
    most = 10 if nonlocal_ else 20 if precision == "fp64" else 150
    if cells < 200 and not nonlocal_:
        most *= 4 if precision == "fp64" else 1
    steps = rng.randint(max(5, most // 3), most)
    return {"kind": kind, "shape": shape, "cells": cells, "material": material, "precision": precision,
            "scheme": scheme, "dt": 1e-6 if nonlocal_ else 2e-6, "drift": 0.1 if nonlocal_ else rng.choice([0.1, 0.6]),
            "steps": steps, "calls": steps if rng.random() < 0.2 else 1}


# ---------------------------------------------------------------------------------------------------------
# inputs


def _mid_run(scene, drift, seed):
    """The lattice fill of a scene turned into a state out of the middle of a run (see the module's text)."""
    rng = np.random.default_rng(seed)
    p = {k: np.array(a, copy=True) for k, a in scene["particles"].items()}
    n, s = p["x"].size, math.sqrt(p["v"][0])
    lo = {k: p[k].min() - 0.45 * s for k in "xy"}
    hi = {k: p[k].max() + 0.45 * s for k in "xy"}
    for k in "xy":
        p[k] = np.clip(p[k] + rng.uniform(-drift, drift, n) * s, lo[k], hi[k])
    a = rng.uniform(-1.0, 1.0, (2, 6))
    wave = [sum(c[i] * np.sin((i + 1) * 3.0 * p["x"] + c[i + 3] * 5.0 + (2 - i) * 4.0 * p["y"]) for i in range(3))
            for c in a]
    p["vx"] = 0.03 * wave[0] + 1e-4 * rng.standard_normal(n)
    p["vy"] = 0.03 * wave[1] + 1e-4 * rng.standard_normal(n)
    p["syy"] = -RHO * 9.8 * (hi["y"] - p["y"]) - 500.0
    p["sxx"] = (0.5 + 0.15 * rng.uniform(0.5, 1.0) * wave[0]) * p["syy"]
    p["sxy"] = 0.05 * wave[1] * p["syy"]
    return dict(scene, particles=p, gravity=GRAVITY)


def _scene(case):
    cells, mat, dt = case["cells"], case["material"], case["dt"]
    h = 1.0 / cells
    mp = None if mat == "isolin" else {"grains_d": 5.3e-4}
    if mat == "g_nonlocal_mu2":
        mp["A"] = 0.48
    if case["shape"] == "box":
        sc = scenes.box_fill(cells=cells, material=mat, dt=dt, mp=mp)
    elif case["shape"] == "silo":
        sc = scenes.silo(cells=cells, material=mat, open_time=0.0, dt=dt, mp=mp)
    elif case["shape"] == "collapse":       # a 0.4 x 0.3 m column in a 2 x 0.5 m box
        h = 2.0 / cells
        sc = scenes.column(Nx=cells + 1, Ny=cells // 4 + 1, h=h, width=0.4, height=0.3, material=mat, rho=RHO, dt=dt,
                           mp=mp)
    else:                                   # a block of half the width, or a column of a quarter of it
        sc = scenes.column(Nx=cells + 1, Ny=cells + 1, h=h, width=0.5 if case["shape"] == "block" else 0.25,
                           height=0.5, material=mat, rho=RHO, dt=dt, mp=mp)
    return dict(sc, scheme=case["scheme"])


def _step_scene(case, seed):
    return _mid_run(_scene(case), case["drift"], seed)


def _batch_scenes(case, seed):
    fleet = scenes.ensemble(case["members"], seed=case["fleet"], dt=case["dt"])
    return [_mid_run(sc, case["drift"], seed * 1000 + k) for k, sc in enumerate(fleet)]


def _adjoint_scene(case, seed):
    c = case["cells"]
    sc = scenes.column(Nx=c + 1, Ny=c // 2 + 1, h=1.0 / c, width=0.25, height=0.25, ppc_1d=case["ppc"],
                       material="g_local_mu2", rho=RHO, dt=case["dt"], mp={"grains_d": 5.3e-4})
    return _mid_run(sc, case["drift"], seed)


def _loss_seeds(n, seed):
    rng = np.random.default_rng(seed + 7)
    return rng.standard_normal(n), rng.standard_normal(n)


def _fields(case):
    return FRAME + (("state3",) if case.get("material") == "g_nonlocal_mu2" else ())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, ne = case["n"], case["elements"]
        # cells in storage order with some scatter, as a running simulation's keys are
        key = torch.arange(n, device="cuda") * ne // n + torch.randint(-3, 4, (n,), generator=g, device="cuda")
        key = torch.where(torch.rand(n, generator=g, device="cuda") < case["outside"], -1, key.clamp(0, ne - 1))
        fn = mpm2d.lib().mpmg_sort_cells_noalloc
        vp = mpm2d.C.c_void_p
        fn.argtypes, fn.restype = [vp, mpm2d.C.c_int, mpm2d.C.c_int, vp, vp, vp, vp], mpm2d.C.c_int
        return {"kind": kind, "n": n, "ne": ne, "fn": fn, "keys": key.to(torch.int32),
                "sorted": torch.empty(n, dtype=torch.int32, device="cuda"),
                "perm": torch.empty(n, dtype=torch.int32, device="cuda"),
                "start": torch.empty(ne + 1, dtype=torch.int32, device="cuda")}
    if kind == "adjoint":
        sim = mpm2d.Simulation(_adjoint_scene(case, seed))
        return {"kind": kind, "sim": sim, "steps": case["steps"], "every": case["every"],
                "loss": _loss_seeds(sim.n, seed)}
    if kind == "batch":
        sim = mpm2d.Batch(_batch_scenes(case, seed), precision="mixed")
        precision = "mixed"
    else:
        precision = case["precision"]
        sim = mpm2d.Simulation(_step_scene(case, seed), precision=precision)
    names = _fields(case)
    pinned = {k: torch.empty(sim.n, dtype=torch.float64, pin_memory=True) for k in names}
    state = {"kind": kind, "sim": sim, "names": names, "calls": case.get("calls", 1),
             "each": case["steps"] // case.get("calls", 1), "pinned": pinned,
             "host": {k: a.numpy() for k, a in pinned.items()}, "single": None}
    if precision != "fp64":
        state["single"] = {k: torch.empty(sim.n, dtype=torch.float32) for k in names}
    return state


def run(state):
    if state["kind"] == "sort":
        s = state
        rc = s["fn"](s["keys"].data_ptr(), s["n"], s["ne"], s["sorted"].data_ptr(), s["perm"].data_ptr(),
                     s["start"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError(mpm2d.lib().mpmg_last_error().decode())
        return {"sorted": s["sorted"], "perm": s["perm"], "start": s["start"]}
    sim = state["sim"]
    if state["kind"] == "adjoint":
        sim.adj_forward_tape(state["steps"], state["every"])
        dtheta = sim.adj_backward(*state["loss"])
        out = {"d" + k: sim.adj_state(k) for k in ADJOINT_STATE}
        out["dtheta"] = dtheta
        return out
    for _ in range(state["calls"]):
        sim.step(state["each"])
    frame = sim.get_frame(state["names"], out=state["host"])
    if state["single"] is None:
        return frame
    for k in state["names"]:
        state["single"][k].copy_(state["pinned"][k])
    return state["single"]


def _sizes(case):
    """(particles, elements, nodes) of a stepping case."""
    if case["kind"] == "batch":
        fleet = scenes.ensemble(case["members"], seed=case["fleet"])
    elif case["kind"] == "adjoint":
        fleet = [_adjoint_scene(case, 0)]
    else:
        fleet = [_scene(case)]
    return (sum(sc["particles"]["x"].size for sc in fleet), sum((sc["Nx"] - 1) * (sc["Ny"] - 1) for sc in fleet),
            sum(sc["Nx"] * sc["Ny"] for sc in fleet))


def work(case):
    """Every step reads and writes the particle state once (mass is read only) and the frame leaves once."""
    if case["kind"] == "sort":
        return {"bytes": 4.0 * (3 * case["n"] + case["elements"] + 1), "flops": 0.0}
    n, ne, nn = _sizes(case)
    steps = case["steps"]
    if case["kind"] == "adjoint":
        # forward, the taped forward again and the reverse sweep over state and adjoint
        return {"bytes": float(steps) * n * 208 * 4, "flops": 700.0 * n * steps}
    if case["kind"] == "batch" or case["precision"] != "fp64":
        per = {"isolin": 92, "g_nonlocal_mu2": 108}.get(case.get("material"), 108)
        return {"bytes": float(steps) * n * per + 4.0 * len(_fields(case)) * n, "flops": 250.0 * n * steps}
    per = {"isolin": 168, "g_nonlocal_mu2": 200}.get(case["material"], 208)
    # a nonlocal step also solves for the nodal fluidity: the matrix rows and vectors once
    extra = nn * 88.0 if case["material"] == "g_nonlocal_mu2" else 0.0
    return {"bytes": steps * (float(n) * per + extra) + 8.0 * len(_fields(case)) * n, "flops": 250.0 * n * steps}


# ---------------------------------------------------------------------------------------------------------
# the step in plain FP64 torch


def _law_isolin(P, S, D, e):
    exx, exy, eyy, wxy = e
    tr, w2s = exx + eyy, 2.0 * wxy * S["sxy"]
    sxx = S["sxx"] + P["dt"] * (P["lam"] * tr + 2 * P["G"] * exx + w2s)
    sxy = S["sxy"] + P["dt"] * (2 * P["G"] * exy - wxy * (S["sxx"] - S["syy"]))
    syy = S["syy"] + P["dt"] * (P["lam"] * tr + 2 * P["G"] * eyy - w2s)
    return dict(S, sxx=sxx, sxy=sxy, syy=syy)


def _flow_root(P, p, tau):
    """tau on the flow curve mu(I) below a trial (p, tau) above yield (p > 0): the smaller root."""
    S0, S2 = P["mu_s"] * p, P["mu_2"] * p
    alpha = P["G"] * P["I0"] * P["dt"] * torch.sqrt(p / P["rho"]) / P["d"]
    B, H = S2 + tau + alpha, S2 * tau + S0 * alpha
    return 2 * H / (B + torch.sqrt(B * B - 4 * H))


def _law_mu2(P, S, D, e):
    exx, exy, eyy, wxy = e
    dt, tr = P["dt"], exx + eyy
    j = 2.0 * wxy * S["sxy"]
    txx = S["sxx"] + dt * (2 * P["G"] * exx + P["lam"] * tr + j)
    txy = S["sxy"] + dt * (2 * P["G"] * exy + wxy * (S["syy"] - S["sxx"]))
    tyy = S["syy"] + dt * (2 * P["G"] * eyy + P["lam"] * tr - j)
    tzz = S["Tzz"] + dt * P["lam"] * tr
    p = -(txx + tyy + tzz) / 3.0
    axx, ayy, azz = txx + p, tyy + p, tzz + p
    q = 0.5 * (axx * axx + 2 * txy * txy + ayy * ayy + azz * azz)
    tau = torch.sqrt(torch.where(q > 0, q, torch.ones_like(q))) * (q > 0)
    dense = (D["m"] / S["v"] >= P["rho_c"]) & (p > 0)
    flow = dense & (tau > P["mu_s"] * p)
    one = torch.ones_like(p)
    ps, ts = torch.where(flow, p, one), torch.where(flow, tau, one)
    tt = torch.where(flow, _flow_root(P, ps, ts), tau)
    f = torch.where(flow, tt / ts, one)
    z = torch.zeros_like(p)
    nup = torch.where(flow, (tau - tt) / P["G"] / dt, z)
    return dict(S, sxx=torch.where(dense, axx * f - p, z), sxy=torch.where(dense, txy * f, z),
                syy=torch.where(dense, ayy * f - p, z), Tzz=torch.where(dense, azz * f - p, z),
                state9=S["state9"] + nup * dt, state10=nup)


def _solve_fluidity(Nx, Ny, nd, Ke, fe, tol=1e-14):
    """The assembled symmetric system's solution by Jacobi-preconditioned CG; zero where no row is."""
    dev = fe[0].device
    nn = Nx * Ny
    C = torch.zeros(9, nn, dtype=torch.float64, device=dev)
    b = torch.zeros(nn, dtype=torch.float64, device=dev)
    pos = [(0, 0), (1, 0), (1, 1), (0, 1)]
    for r in range(4):
        b.index_add_(0, nd[r], fe[r])
        for c in range(4):
            k = (pos[c][1] - pos[r][1] + 1) * 3 + pos[c][0] - pos[r][0] + 1
            C[k].index_add_(0, nd[r], Ke[r][c])
    C = C.view(9, Ny, Nx)
    diag = C[4]
    inv = torch.where(diag > 0, 1.0 / torch.where(diag > 0, diag, torch.ones_like(diag)), torch.zeros_like(diag))

    def mul(u):
        w = torch.nn.functional.pad(u, (1, 1, 1, 1))
        return sum(C[k] * w[k // 3:k // 3 + Ny, k % 3:k % 3 + Nx] for k in range(9))

    r = torch.where(diag > 0, b.view(Ny, Nx), torch.zeros_like(diag))
    x = torch.zeros_like(r)
    r0 = float(r.norm())
    if r0 == 0.0:
        return x.view(-1)
    z = inv * r
    d, rz = z.clone(), (r * z).sum()
    for it in range(4000):
        q = mul(d)
        a = rz / (d * q).sum()
        x, r = x + a * d, r - a * q
        if it % 16 == 15 and float(r.norm()) <= tol * r0:
            break
        z = inv * r
        rz2 = (r * z).sum()
        d, rz = z + (rz2 / rz) * d, rz2
    return x.view(-1)


def _law_nonlocal(P, S, D, e, N, gx, gy, nd, Nx, Ny, on):
    exx, exy, eyy, wxy = e
    dt = P["dt"]
    t = _law_isolin(P, S, D, e)
    p = -0.5 * (t["sxx"] + t["syy"])
    axx, axy, ayy = t["sxx"] + p, t["sxy"], t["syy"] + p
    tau = torch.sqrt(0.5 * (axx * axx + 2 * axy * axy + ayy * ayy))
    z, one = torch.zeros_like(p), torch.ones_like(p)
    dense = on & (D["m"] / S["v"] >= P["rho_c"]) & (p >= 0)
    act = dense & (p > 0)
    flow = act & (tau > P["mu_s"] * p)
    ps, ts = torch.where(act, p, one), torch.where(flow, tau, one)
    tt = torch.where(flow, _flow_root(P, torch.where(flow, p, one), ts), tau)
    gfl = torch.where(flow, ps * (tau - tt) / (P["G"] * dt * torch.where(flow, tt, one)), z)
    xi = torch.where(act, (tt / ps - P["mu_s"]).abs() / (P["A"] * P["A"] * P["d"] * P["d"]), z)
    w = torch.where(dense, S["v"], z)
    Ke = [[w * (xi * N[r] * N[c] + gx[r] * gx[c] + gy[r] * gy[c]) for c in range(4)] for r in range(4)]
    fe = [w * gfl * xi * N[r] for r in range(4)]
    g = _solve_fluidity(Nx, Ny, nd, Ke, fe)
    gf = sum(N[r] * g[nd[r]] for r in range(4))
    pd = torch.where(dense, p, z)
    live = pd > 0
    s = torch.where(live, pd / torch.where(live, P["G"] * dt * gf + pd, one), z)
    nup = torch.where(live, (tau - tau * s) / (P["G"] * dt), z)
    return dict(S, sxx=torch.where(live, s * axx - pd, z), sxy=torch.where(live, s * axy, z),
                syy=torch.where(live, s * ayy - pd, z), state9=S["state9"] + nup * dt, state10=nup, state3=gf)


def _exact_run(scene, steps, theta=None, S=None):
    """(fixed data, state) after `steps` steps of the scene; differentiable in theta and the start state S."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = dict(dtype=torch.float64, device=dev)
    pt = {k: torch.as_tensor(np.asarray(a), **f64) for k, a in scene["particles"].items()}
    mat, Nx, Ny, h, dt = scene["material"], scene["Nx"], scene["Ny"], scene["h"], scene["dt"]
    mp = dict(CONSTANTS, **scene.get("mp", {}))
    th = theta if theta is not None else [mp[k] for k in THETA]
    G, K = th[3] / (2 * (1 + mp["nu"])), th[3] / (3 * (1 - 2 * mp["nu"]))
    P = {"G": G, "K": K, "lam": K - 2 * G / 3, "dt": dt, "mu_s": th[0], "mu_2": th[1], "I0": th[2],
         "rho": mp["grains_rho"], "d": mp["grains_d"], "rho_c": mp["rho_critical"], "A": mp["A"]}
    D = {"m": pt["m"]}
    z = torch.zeros_like(pt["x"])
    if S is None:
        S = {k: pt[k] for k in ("x", "y", "vx", "vy", "v", "sxx", "sxy", "syy")}
        S.update({k: z for k in ("ux", "uy", "Tzz", "state9", "state10", "state3")})
    xmax, ymax = scene.get("xmax", 1.0), scene.get("ymax", 1.0)
    i, j = torch.arange(Nx, device=dev), torch.arange(Ny, device=dev)
    mx, my = torch.zeros(Ny, Nx, dtype=torch.bool, device=dev), torch.zeros(Ny, Nx, dtype=torch.bool, device=dev)
    if scene["bc"] == "box":                # the walls are the grid's edges in every scene here
        for k, sl in enumerate([(slice(None), 0), (0, slice(None)), (slice(None), Nx - 1), (Ny - 1, slice(None))]):
            mx[sl] |= bool(scene["bci"][k] & 1)
            my[sl] |= bool(scene["bci"][k] & 2)
    else:
        floor = ~(i * h <= scene["bcf"][0])
        mx[0] |= floor
        my[0] |= floor
        mx[:, 0] = True
        mx[:, int((Nx - 1) * scene["bcf"][2])] = True
    mx, my = mx.view(-1), my.view(-1)
    nn, ne_x, ne_y = Nx * Ny, Nx - 1, Ny - 1
    on = torch.ones_like(z, dtype=torch.bool)
    for _ in range(steps):
        with torch.no_grad():
            x, y = S["x"].detach(), S["y"].detach()
            ci, cj = torch.floor(x / h), torch.floor(y / h)
            on = on & (x >= 0) & (x < xmax) & (y >= 0) & (y < ymax) & (ci < ne_x) & (cj < ne_y)
            n0 = torch.where(on, cj * Nx + ci, torch.zeros_like(ci)).long()
            nd = [n0, n0 + 1, n0 + Nx + 1, n0 + Nx]
            gate = on.to(torch.float64)
        a, b = S["x"] / h - ci, S["y"] / h - cj
        N = [(1 - a) * (1 - b), a * (1 - b), a * b, (1 - a) * b]
        gx = [-(1 - b) / h, (1 - b) / h, b / h, -b / h]
        gy = [-(1 - a) / h, -a / h, a / h, (1 - a) / h]

        def nodes(parts):
            acc = torch.zeros(nn, **f64)
            for r in range(4):
                acc = acc.index_add(0, nd[r], torch.where(on, parts(r), z))
            return acc

        m, v = D["m"], S["v"]
        M = nodes(lambda r: N[r] * m)
        PX, PY = nodes(lambda r: N[r] * m * S["vx"]), nodes(lambda r: N[r] * m * S["vy"])
        FX = nodes(lambda r: -v * (gx[r] * S["sxx"] + gy[r] * S["sxy"]))
        FY = nodes(lambda r: N[r] * m * scene["gravity"] - v * (gx[r] * S["sxy"] + gy[r] * S["syy"]))
        o = torch.zeros(nn, **f64)
        PX, FX, PY, FY = torch.where(mx, o, PX), torch.where(mx, o, FX), torch.where(my, o, PY), torch.where(my, o, FY)
        has = M > 1e-10
        Ms = torch.where(has, M, torch.ones_like(M))
        AX, AY = torch.where(has, FX / Ms, o), torch.where(has, FY / Ms, o)
        VX, VY = torch.where(has, (PX + dt * FX) / Ms, o), torch.where(has, (PY + dt * FY) / Ms, o)

        def at(q, w):
            return sum(w[r] * q[nd[r]] for r in range(4))

        dx, dy = dt * at(VX, N), dt * at(VY, N)
        T = dict(S, vx=S["vx"] + dt * at(AX, N), vy=S["vy"] + dt * at(AY, N), x=S["x"] + dx, y=S["y"] + dy,
                 ux=S["ux"] + dx, uy=S["uy"] + dy)
        if scene.get("scheme") == "musl":
            VX, VY = nodes(lambda r: N[r] * m * T["vx"]), nodes(lambda r: N[r] * m * T["vy"])
            VX, VY = torch.where(has, VX / Ms, o), torch.where(has, VY / Ms, o)
        exx, eyy = at(VX, gx), at(VY, gy)
        xy, yx = at(VX, gy), at(VY, gx)
        e = (exx, 0.5 * (xy + yx), eyy, 0.5 * (xy - yx))
        T["v"] = v * torch.exp(dt * (exx + eyy))
        if mat == "isolin":
            T = _law_isolin(P, T, D, e)
        elif mat == "g_local_mu2":
            T = _law_mu2(P, T, D, e)
        else:
            T = _law_nonlocal(P, T, D, e, N, gx, gy, nd, Nx, Ny, on)
        S = {k: torch.where(on, T[k], S[k]) for k in T}
    return D, S


def exact(case, seed):
    if case["kind"] == "sort":
        return None
    if case["kind"] == "adjoint":
        sc = _adjoint_scene(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        theta = [torch.tensor(CONSTANTS[k], dtype=torch.float64, device=dev, requires_grad=True) for k in THETA]
        S = {k: torch.as_tensor(a, dtype=torch.float64, device=dev) for k, a in sc["particles"].items() if k != "m"}
        z = torch.zeros_like(S["x"])
        S.update({k: z.clone() for k in ("ux", "uy", "Tzz", "state9", "state10", "state3")})
        lead = {k: S[k].clone().requires_grad_(True) for k in ADJOINT_STATE}
        _, T = _exact_run(sc, case["steps"], theta, dict(S, **lead))
        lx, ly = (torch.as_tensor(a, device=dev) for a in _loss_seeds(z.numel(), seed))
        (T["x"] * lx + T["y"] * ly).sum().backward()
        out = {"d" + k: lead[k].grad.cpu().numpy() for k in ADJOINT_STATE}
        out["dtheta"] = np.array([float(t.grad) for t in theta] + [0.0])
        return out
    scs = _batch_scenes(case, seed) if case["kind"] == "batch" else [_step_scene(case, seed)]
    names = _fields(case)
    got = [dict(S, **D) for D, S in (_exact_run(sc, case["steps"]) for sc in scs)]
    return {k: torch.cat([g[k] for g in got]).cpu().numpy() for k in names}
