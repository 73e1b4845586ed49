"""The measured workloads of the engine: what its users run, end to end
through the ctypes binding of the C ABI (host arrays in, host arrays out).

Every case is a whole call of a solver: the context with its mode table and
geometry loaded is what a program keeps, the run and its output arrays are
what it asks for.  Sizes follow the repository's benchmark configurations,
its tests and the ranges between and around them.

Outputs are sums over random trajectories that the engine draws from its own
counter-based streams, so no closed formula gives them (`exact` is None); one
seed repeats one result to the order of the FP64 additions."""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "bte-barna_gb300"))

import btegpu  # noqa: E402
import synth  # noqa: E402

T0 = 300.0


def listed():
    return [
        # the smallest call: a parity-sized ribbon, where the chain of one
        # particle's flights and the launches around it set the time
        {"name": "ribbon_smallest", "kind": "ribbon", "n": 8, "opt": 3, "length": 200.0, "width": 50.0, "cells": 5,
         "dt": 10.0, "bins": 20, "p": 0.0, "N": 2000},
        # the plain ribbon between two reservoirs at the benchmark's size
        {"name": "ribbon_plain", "kind": "ribbon", "n": 32, "opt": 3, "length": 1000.0, "width": 100.0, "cells": 50,
         "dt": 10.0, "bins": 100, "p": 0.0, "N": 1000000},
        # the transient at scale: large table, porous rectangle, hot spot, partly specular walls
        {"name": "pore_transient", "kind": "pore", "n": 64, "opt": 6, "lx": 2000.0, "ly": 500.0, "nx": 100, "ny": 25,
         "pore": 200.0, "dt": 50.0, "bins": 200, "p": 0.3, "N": 2000000},
        # one round of the batched sweep: 64 ribbons at four temperatures in
        # one launch, eight replica groups for the error bars
        {"name": "sweep_64", "kind": "sweep", "n": 32, "opt": 3, "widths": 16, "cells": 50, "dt": 10.0, "bins": 100,
         "groups": 8, "N": 4000000},
        # boxes off a grid: the periodic bar on the convex-polygon kernel
        {"name": "bar_periodic", "kind": "bar", "n": 32, "opt": 3, "length": 40.0, "width": 20.0, "strips": 10,
         "dt": 10.0, "bins": 100, "N": 2000000},
        # two crystals joined by a diffuse mismatch interface
        {"name": "two_crystals", "kind": "crystals", "n": 16, "opt": 3, "length": 200.0, "width": 50.0, "cells": 10,
         "dt": 10.0, "bins": 30, "N": 300000},
        # the steady state of a nanoribbon under a gradient (periodic along it, diffuse walls)
        {"name": "steady_ribbon", "kind": "steady", "n": 16, "opt": 3, "length": 40.0, "width": 100.0, "nx": 2, "ny": 2,
         "N": 200000},
        # forward and adjoint pass: gradient of kappa_eff with respect to
        # every lifetime and the specularity
        {"name": "adjoint_ribbon", "kind": "adjoint", "n": 32, "opt": 3, "length": 1000.0, "width": 100.0, "cells": 50,
         "dt": 10.0, "bins": 100, "p": 0.2, "N": 1000000},
        # spectral decomposition at three boxes, with its four outputs
        {"name": "spectral_ribbon", "kind": "spectral", "n": 16, "opt": 3, "length": 1000.0, "width": 100.0,
         "cells": 25, "dt": 10.0, "bins": 40, "ticks": 200, "N": 200000},
        # replay mode: the run a user checks the engine with, draw for draw
        {"name": "replay_ribbon", "kind": "replay", "n": 16, "opt": 3, "length": 400.0, "width": 100.0, "cells": 20,
         "dt": 10.0, "bins": 50, "N": 100000},
        # beyond-RTA steps with a propagator of the benchmark's size
        {"name": "berta_propagator", "kind": "berta", "n": 32, "opt": 3, "length": 100.0, "width": 100.0, "cells": 5,
         "dt": 1.0, "steps": 30, "alive": 4000000, "rta": False},
        # the same loop with its RTA scattering
        {"name": "berta_rta", "kind": "berta", "n": 16, "opt": 3, "length": 100.0, "width": 50.0, "cells": 4,
         "dt": 1.0, "steps": 40, "alive": 2000000, "rta": True},
    ]


def _log(rng, lo, hi):
    return float(np.exp(rng.uniform(np.log(lo), np.log(hi))))


def draw(rng):
    kind = rng.choice(["ribbon", "ribbon", "pore", "pore", "sweep", "bar", "crystals", "steady", "adjoint", "spectral",
                       "replay", "berta"])
    c = {"kind": kind, "opt": rng.randint(1, 4)}
    cells = rng.randint(3, 60)  # cell widths in quarters of a nm: lengths are exact multiples of them
    ribbon = {"length": 0.25 * round(4 * _log(rng, 100.0, 1500.0) / cells) * cells,
              "width": round(_log(rng, 20.0, 400.0), 1), "cells": cells, "dt": round(_log(rng, 5.0, 20.0), 2), "bins": rng.randint(15, 100)}
    if kind == "ribbon":
        c.update(ribbon, n=rng.randint(8, 32), p=rng.choice([0.0, 0.2, round(rng.random(), 3)]),
                 N=int(_log(rng, 1e3, 1e6)))
    elif kind == "pore":
        nx, ny = rng.randint(15, 100), rng.randint(8, 25)
        c.update(n=2 * rng.randint(6, 24), lx=20.0 * nx, ly=20.0 * ny, nx=nx, ny=ny,
                 pore=round(20.0 * ny * rng.uniform(0.1, 0.6), 1), dt=round(rng.uniform(20.0, 50.0), 2),
                 bins=rng.randint(20, 150), p=round(rng.uniform(0.0, 0.6), 3), N=int(_log(rng, 1e4, 1e6)))
    elif kind == "sweep":
        c.update(n=rng.randint(8, 32), widths=rng.randint(3, 16), cells=rng.randint(10, 50), dt=10.0,
                 bins=rng.randint(50, 100), groups=rng.randint(2, 8), N=int(_log(rng, 2e5, 4e6)))
    elif kind == "bar":
        c.update(n=rng.randint(8, 32), length=round(_log(rng, 20.0, 200.0), 1), width=round(_log(rng, 10.0, 100.0), 1),
                 strips=rng.randint(4, 16), dt=10.0, bins=rng.randint(20, 100), N=int(_log(rng, 1e4, 1e6)))
    elif kind == "crystals":
        cells = rng.randint(4, 20)
        c.update(n=2 * rng.randint(4, 9), length=0.25 * round(4 * _log(rng, 100.0, 400.0) / cells) * cells,
                 width=round(_log(rng, 20.0, 200.0), 1), cells=cells, dt=10.0, bins=rng.randint(15, 40),
                 N=int(_log(rng, 1e4, 3e5)))
    elif kind == "steady":
        c.update(n=2 * rng.randint(4, 10) + 1, length=round(_log(rng, 20.0, 200.0), 1),
                 width=round(_log(rng, 50.0, 400.0), 1), nx=rng.randint(2, 3), ny=rng.randint(2, 4),
                 N=int(_log(rng, 2e4, 2e5)))
    elif kind == "adjoint":
        c.update(ribbon, n=rng.randint(8, 32), p=round(rng.uniform(0.05, 0.9), 3), N=int(_log(rng, 1e4, 1e6)))
    elif kind == "spectral":
        c.update(ribbon, n=rng.randint(8, 16), bins=rng.randint(10, 40), ticks=rng.randint(50, 200),
                 N=int(_log(rng, 1e4, 2e5)))
    elif kind == "replay":
        c.update(ribbon, n=rng.randint(8, 16), bins=rng.randint(15, 50),
                 N=int(_log(rng, 2e3, 1e5)))
    else:
        cells = rng.randint(3, 5)
        c.update(n=rng.randint(12, 20), length=0.25 * round(4 * _log(rng, 60.0, 120.0) / cells) * cells,
                 width=round(_log(rng, 50.0, 100.0), 1), cells=cells, dt=1.0, steps=rng.randint(15, 40), alive=int(rng.uniform(2e6, 4e6)),
                 rta=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ inputs
def _modes(case, seed, T=T0, k=0):
    """A synthetic mode table of the case's size; the seed gives its branches and lifetimes."""
    return synth.mode_table(case["n"], 3, case["opt"], T, config=1000 + 2 * seed + k)


def _ribbon(case):
    return synth.ribbon_geometry(case["length"], case["width"], case["cells"])


def _propagator(m, dt, seed):
    """exp(B dt) of a relaxation operator with a sparse sign-changing coupling
    (the form of synth.propagator), by its power series on the GPU: what a
    propagator file holds, made quickly."""
    import torch
    w = np.asarray(m["w"])[3:]
    c = np.sqrt(synth.be_kernel(np.asarray(m["omega"])[3:], T0))
    n, rng = w.size, np.random.default_rng(np.random.SeedSequence((seed, 77)))
    rows, cols = np.repeat(np.arange(n), 32), rng.integers(0, n, size=32 * n)
    g = rng.lognormal(0.0, 1.0, rows.size)
    s = 0.1 * g * np.minimum(w[rows], w[cols]) * (rows != cols)
    s[(g < 0.5) & (rng.random(rows.size) < 0.25)] *= -1.0  # weak couplings only: the operator stays positive
    d = dict(device="cuda", dtype=torch.float64)
    W, C = torch.tensor(w, **d), torch.tensor(c, **d)
    S = torch.zeros((n, n), **d)
    # entry by entry in a fixed order (no atomics), so that one seed gives one matrix
    key = rows * n + cols
    uniq, inv = np.unique(key, return_inverse=True)
    S.view(-1)[torch.tensor(uniq, device="cuda")] = torch.tensor(np.bincount(inv, weights=s), **d)
    S = S + S.T
    A = torch.diag(W + (S @ C) / C) - torch.outer(W * C, W * C) / (C @ (W * C)) - S
    # exp(-A dt) = (exp(-A dt / 2^k))^(2^k), FP32 products (an input: its rounding is part of it)
    X = (-A * dt).float()
    norm = float(X.abs().sum(dim=0).max())
    k = max(0, int(np.ceil(np.log2(max(norm, 1e-9)))))
    X = X / 2.0 ** k
    E = torch.eye(n, device="cuda") + X
    term = X
    for i in range(2, 9):
        term = (term @ X) / i
        E = E + term
    for _ in range(k):
        E = E @ E
    E = E.double() * C[:, None] / C[None, :]
    return np.asfortranarray(E.T.contiguous().cpu().numpy().T)


def prepare(case, seed):
    kind = case["kind"]
    eng = btegpu.Engine(0)
    s = {"eng": eng, "kind": kind, "seed": 11 + 7 * seed, "case": case}
    if kind in ("ribbon", "adjoint", "spectral", "replay"):
        m = _modes(case, seed)
        eng.load_modes(m)
        eng.load_geometry(_ribbon(case))
        if kind == "adjoint":
            s["W"] = _kappa_weights(case)
        if kind == "spectral":
            nc = case["cells"]
            s["boxes"] = sorted({0, nc // 2, nc - 1})
            eng.set_spectral(s["boxes"], case["ticks"])
    elif kind == "pore":
        eng.load_modes(_modes(case, seed))
        eng.load_geometry(synth.grid_geometry(
            case["lx"], case["ly"], case["nx"], case["ny"], T0, pore_center=(0.5 * case["lx"], 0.5 * case["ly"]),
            pore_diameter=case["pore"], hot_center=(0.25 * case["lx"], 0.5 * case["ly"]), hot_sigma=50.0, hot_dT=1.0))
    elif kind == "sweep":
        cases = synth.sweep_cases(n_widths=case["widths"])
        temps = sorted({c["T"] for c in cases})
        tabs = {T: _modes(case, seed, T) for T in temps}
        eng.load_modes(tabs[temps[0]])
        eng.load_geometry(synth.sweep_union_geometry(cases, length=20.0 * case["cells"], ncells=case["cells"]))
        b = np.array([c["budget"] for c in cases], dtype=float)
        eng.load_materials([tabs[c["T"]]["w"] for c in cases], [c["T"] for c in cases], b / b.sum())
        eng.set_groups(case["groups"])
    elif kind == "bar":
        eng.load_modes(_modes(case, seed))
        eng.load_geometry(synth.periodic_bar_geometry(case["width"], case["length"], case["strips"]))
    elif kind == "crystals":
        eng.load_mode_tables([_modes(case, seed), _modes(case, seed, k=1)])
        g, nc = _ribbon(case), case["cells"]
        g["material"] = np.array([0] * (nc // 2) + [1] * (nc - nc // 2) + [0, 1], dtype=np.int32)
        eng.load_geometry(g)
    elif kind == "steady":
        eng.load_modes(_modes(case, seed))
        eng.load_geometry(synth.periodic_ribbon_geometry(case["length"], case["width"], case["nx"], case["ny"]))
    else:
        m = _modes(case, seed)
        eng.load_modes(m)
        eng.load_geometry(_ribbon(case))
        s["Eeff"] = _berta_eeff(m, case)
        if not case["rta"]:
            eng.load_propagator(_propagator(m, case["dt"], seed), T0)
    return s


def _kappa_weights(case):
    """kappa_eff as a linear functional of the raw tallies: the flux of the
    interior cells over the last bins, per unit particle energy."""
    nb, nc = case["bins"], case["cells"]
    last = min(10, nb)
    cnt = np.array([(nb - b) if b >= nb - last else last for b in range(nb)], float) / last
    W = np.zeros((nc + 2, nb, 3))
    W[:nc, :, 1] = cnt / (nc * case["width"] * case["length"] / nc)
    return W


def _berta_eeff(m, case):
    """Particle energy for about `alive` particles at the end: the energy that
    the two reservoirs inject over the run, shared out (a program finds it
    with a short run)."""
    v = np.asarray(m["vg"]).reshape(-1, 3)[:, 0]
    cap = 1.3806488e-23 * synth.be_kernel(np.asarray(m["omega"]), T0) * (np.asarray(m["omega"]) > 0)
    flux = float((cap * v)[v > 0].sum()) / (m["nq"] * m["V"])  # J nm^-2 ps^-1 per kelvin
    return 2.0 * flux * case["width"] * synth.C_LAT * case["dt"] * case["steps"] / case["alive"]


# ------------------------------------------------------------------ one call
_RTA = ("temperature", "jx", "jy", "gz", "gz_jx", "gz_jy", "Eeff", "energy_rate", "events", "wall_hits", "crossings",
        "absorbed", "specular_hits", "tally_updates", "translations", "interface_hits", "interface_transmissions")
_STEADY = ("temperature", "jx", "jy", "gz", "gz_jx", "gz_jy", "Eeff", "energy_rate", "generations", "events",
           "wall_hits", "crossings", "absorbed", "translations", "scattered", "births", "lost")


def run(s):
    eng, c, kind = s["eng"], s["case"], s["kind"]
    if kind == "berta":
        r = eng.berta_run(c["dt"], (c["steps"] - 0.5) * c["dt"], s["Eeff"], T0=T0, seed=s["seed"], rta=c["rta"])
        return {"ed": r["ed"], "flux": r["flux"]}
    if kind == "steady":
        r = eng.steady_run(T0, (-0.01, 0.0), c["N"], seed=s["seed"], max_generations=60, log_cap=60)
        log = np.zeros((60, 4))  # the convergence table has a row per generation
        log[:len(r["log"])] = r["log"]
        return {**{k: r[k] for k in _STEADY}, "log": log}
    maxtime = c["dt"] * c["bins"]
    if kind == "adjoint":
        r = eng.rta_adjoint(s["W"], T0, c["dt"], maxtime, c["N"], seed=s["seed"], specularity=c["p"])
        return {k: r[k] for k in ("phi", "dphi_dtau", "dphi_dp", "events")}
    kw = {"seed": s["seed"], "specularity": c.get("p", 0.0)}
    if kind == "pore":
        kw["source"] = btegpu.SOURCE_INITIAL
    if kind == "replay":
        kw.update(mode=btegpu.MODE_REPLAY, exact=True)
    r = eng.rta_run(T0, c["dt"], maxtime, c["N"], **kw)
    out = {k: r[k] for k in _RTA + (("exact",) if kind == "replay" else ())}
    if kind == "sweep":
        for g in range(c["groups"]):
            out["jx_group%d" % g] = eng.group_result(g, r["jx"].shape, keys=("jx",))["jx"]
    if kind == "spectral":
        q = eng.get_spectral(c["bins"])
        out.update({"spec_" + k: q[k] for k in ("omega", "dT_omega", "jx_omega", "jy_omega", "fd_q", "q1bz", "raw")})
    return out


# ------------------------------------------------------------------ work
def work(case):
    """Each table the path reads and each output it writes once, and the FP64
    arithmetic of the flights: per flight an exit time in x and y, the
    advance, the time left and three tally differences (12 operations), and
    as many flights per particle as its scattering rate gives."""
    kind = case["kind"]
    modes = case["n"] ** 2 * (3 + case["opt"])
    if kind == "berta":
        nm = modes - 3
        psteps = 0.5 * case["alive"] * case["steps"]
        # per particle-step its state read and written, one table entry; the tables once
        return {"bytes": 64.0 * psteps + (0 if case["rta"] else 8.0 * nm * nm) + 40.0 * modes, "flops": 12.0 * psteps}
    bins = 1 if kind == "steady" else case["bins"]
    boxes = {"pore": lambda: case["nx"] * case["ny"], "sweep": lambda: 4 * case["widths"] * (case["cells"] + 2),
             "bar": lambda: case["strips"] + 4, "steady": lambda: case["nx"] * case["ny"] + 2}.get(
                 kind, lambda: case["cells"] + 2)()
    nbytes = 40.0 * modes + 6 * 8.0 * boxes * bins
    if kind == "sweep":
        nbytes += 8.0 * boxes * bins * case["groups"]
    if kind == "spectral":
        nbytes += 3 * bins * 8.0 * (modes + 3 * case["ticks"])
    passes = 2.0 if kind == "adjoint" else 1.0
    # a particle from a reservoir mostly goes back soon; one of an initial
    # deviation or a closed structure scatters until the end
    flights = {"pore": 1.0, "steady": 20.0}.get(kind, 0.2)
    if kind != "steady":
        flights *= case["dt"] * case["bins"] * 0.2
    return {"bytes": nbytes, "flops": 12.0 * passes * case["N"] * flights}


def exact(case, seed):
    return None
