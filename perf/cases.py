"""Timed cases of the force-and-step path, each through the calls a program makes.

A case is a dict of plain values.  ``listed()`` names the standing ones, ``draw(rng)`` gives further
cases of the same ranges, ``prepare(case, seed)`` makes what a program has in hand before the call,
``run(state)`` is one pass, ``work(case)`` what a pass cannot do without, and ``exact(case, seed)``
the same outputs in 64-bit torch or numpy.

Kinds of case:

* ``force``     accelerations of device-resident bodies (gtd_direct_accelerations_noalloc)
* ``direct``    System.evolve by direct summation, optionally followed by System.energy
* ``bh_step``   System.evolve with Barnes-Hut forces
* ``bh_force``  System.bh_accelerations: tree build, walk, interaction counts
* ``ensemble``  Ensemble.evolve of many small systems, then their state
* ``adjoint``   leapfrog_final_state and its gradients
* ``comet``     an evolve driven by device callbacks, with overlap collisions

Results whose terms are FP32 by the caller's choice (mixed precision, the FP32 tree, the ensemble's
pair forces) are kept in single precision, as such a program stores them; positions and velocities
are FP64 state throughout.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import gregpackagescpp_b200 as gtd
from gregpackagescpp_b200 import _lib
from gregpackagescpp_b200.adjoint import leapfrog_final_state
from gregpackagescpp_b200.ensemble import Ensemble
from gregpackagescpp_b200.ics import AU, G_DEFAULT, UNITS_G6674, comet_stage, ensemble, plummer, two_plummer

HOUR = 3600.0
METHODS = {"euler": 2, "modified_euler": 4, "midpoint": 8, "kdk": 16, "dkd": 32}
BARNES_HUT = 65536

# One unordered pair: 3 differences, 5 for the squared distance, 4 for its -3/2 power, 2 mass factors
# and 6 multiply-adds.
PAIR_FLOPS = 26
# Per unordered pair of a VJP: the pair above plus both bodies' J^T w and mass terms.
VJP_PAIR_FLOPS = 60


def listed():
    return [
        # the smallest call: one force evaluation of a small system inside somebody else's loop
        {"name": "force_f64_1000", "kind": "force", "n": 1000, "precision": "f64"},
        # the same call near its size limit, FP32 pair terms, an odd count
        {"name": "force_mixed_60001", "kind": "force", "n": 60001, "precision": "mixed"},
        # a small cluster followed for many steps, as the reference library is run
        {"name": "kdk_f64_1024", "kind": "direct", "n": 1024, "precision": "f64", "method": "kdk", "steps": 500,
         "energy": False},
        # an ordinary FP64 run with a two-stage method: two force evaluations a step
        {"name": "meuler_f64_16384", "kind": "direct", "n": 16384, "precision": "f64", "method": "modified_euler",
         "steps": 8, "energy": False},
        # an ordinary mixed run between two looks at the energy
        {"name": "kdk_mixed_40000_energy", "kind": "direct", "n": 40000, "precision": "mixed", "method": "kdk",
         "steps": 5, "energy": True},
        # the headline size: mixed leapfrog on a Plummer sphere
        {"name": "kdk_mixed_262144", "kind": "direct", "n": 262144, "precision": "mixed", "method": "kdk", "steps": 2,
         "energy": False},
        # two approaching clusters with the FP32 tree
        {"name": "bh_float_1048576", "kind": "bh_step", "n": 1048576, "tree": "float", "steps": 24, "theta": 0.5},
        # tree forces and interaction counts once, FP64 tree, softened, an odd count
        {"name": "bh_double_131071", "kind": "bh_force", "n": 131071, "tree": "double", "theta": 0.5, "eps": 1e7},
        # a batch of few-body systems of uneven size
        {"name": "ensemble_512", "kind": "ensemble", "systems": 512, "n_max": 2048, "steps": 100, "density": 1500.0},
        # a fit on a small system: launches and allocations count
        {"name": "adjoint_1000", "kind": "adjoint", "n": 1000, "steps": 60},
        # a fit on the adjoint's ordinary size
        {"name": "adjoint_16384", "kind": "adjoint", "n": 16384, "steps": 30},
        # a collapsing cloud of touching bodies, callbacks and collisions every step
        {"name": "comet_727", "kind": "comet", "n": 727, "steps": 512},
    ]


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["force", "direct", "direct", "bh_step", "bh_force", "ensemble", "adjoint", "comet"])
    if kind == "force":
        return {"kind": kind, "n": _spread(rng, 100, 65536), "precision": rng.choice(["f64", "mixed"])}
    if kind == "direct":
        precision = rng.choice(["f64", "mixed"])
        n = _spread(rng, 100, 65536 if precision == "f64" else 262144)
        steps = max(2, min(500, int(2e10 / n ** 2), int(2e6 / n)))
        # few steps at FP32 pair terms, so that their rounding stays far below the state's
        return {"kind": kind, "n": n, "precision": precision, "method": rng.choice(sorted(METHODS)),
                "steps": steps if precision == "f64" else min(steps, 5), "energy": rng.random() < 0.3}
    if kind == "bh_step":
        tree = rng.choice(["float", "float", "double"])
        return {"kind": kind, "n": _spread(rng, 1000, 1048576 if tree == "float" else 262144), "tree": tree,
                "steps": rng.randint(2, 8), "theta": round(rng.uniform(0.4, 0.9), 3)}
    if kind == "bh_force":
        return {"kind": kind, "n": _spread(rng, 1000, 524288), "tree": rng.choice(["float", "double"]),
                "theta": round(rng.uniform(0.4, 0.9), 3), "eps": rng.choice([0.0, 1e7])}
    if kind == "ensemble":
        return {"kind": kind, "systems": _spread(rng, 16, 512), "n_max": _spread(rng, 16, 2048),
                "steps": rng.randint(20, 100), "density": rng.choice([1500.0, 1500.0, 1.5])}
    if kind == "adjoint":
        n = _spread(rng, 100, 16384)
        return {"kind": kind, "n": n, "steps": max(5, min(60, int(8e9 / n ** 2)))}
    return {"kind": kind, "n": _spread(rng, 64, 727), "steps": rng.randint(128, 512)}


# ---- inputs ---------------------------------------------------------------------------------------

def _bodies(case, seed):
    """(m, x, v) of a case's bodies."""
    kind, n = case["kind"], case["n"]
    if kind == "force":  # unequal masses
        m, x, v = plummer(n, seed)
        return m * np.random.default_rng(seed).uniform(0.2, 1.8, n), x, v
    if kind in ("bh_step", "bh_force"):
        m, x, v = two_plummer((n + 1) // 2, seed)
        return m[:n], np.ascontiguousarray(x[:n]), np.ascontiguousarray(v[:n])
    m, x, v = plummer(n, seed)
    if kind == "direct":  # a cluster that moves through its frame, so that momentum and centre are not zero
        x, v = x + np.array([3.0, -2.0, 1.0]) * AU, v + np.array([2e4, 1e4, -1.5e4])
    return m, x, v


def _comet(case, seed):
    """A cloud with the shape and constants of random_comet's evolve stage once it has contracted, its
    bodies moving at about the cloud's own escape speed."""
    c = comet_stage(case["n"], 1200.0 * (case["n"] / 727) ** (1 / 3), 75.0, 4197481476.49696707306, 3.0, 1200.0, 0.5,
                    0.95, 0.0, seed)
    c["v"] = np.random.default_rng(seed).normal(0.0, 0.5, (case["n"], 3))
    return c


COMET_DT, COMET_PROBING = 1 / 128, 50000


def _ensemble(case, seed):
    """(offsets, m, r, x, v) of systems whose sizes, uniform on 3 .. n_max, belong to the case."""
    sizes = np.random.default_rng(case["systems"]).integers(3, case["n_max"] + 1, case["systems"])
    parts = [ensemble(1, seed * 1009 + k, n_min=n, n_max=n, density=case["density"])[1:]
             for k, n in enumerate(sizes.tolist())]
    return (np.concatenate([[0], np.cumsum(sizes)]), *(np.concatenate(a) for a in zip(*parts)))


ENSEMBLE_DT = 60.0
BH_DT = 600.0


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "force":
        m, x, _ = _bodies(case, seed)
        lib = _lib.load()
        lib.gtd_direct_accelerations_noalloc.argtypes = [C.c_int64, C.c_void_p, C.c_double, C.c_int, C.c_void_p,
                                                         C.c_void_p]
        st["lib"] = lib
        st["pm4"] = torch.tensor(np.concatenate([x, m[:, None]], 1), device="cuda")
        st["acc"] = torch.empty((case["n"], 3), dtype=torch.float64, device="cuda")
    elif kind in ("direct", "bh_step", "bh_force"):
        m, x, v = _bodies(case, seed)
        s = gtd.System(m, x, v, timestep=HOUR if kind == "direct" else BH_DT, num_iterations=case.get("steps", 1),
                       units_format=UNITS_G6674, precision=case.get("precision", "f64"))
        if kind != "direct":
            s.set_bh_opening_angle(case["theta"])
            s.bh_tree_float(case["tree"] == "float")
            if case.get("eps"):
                s.set_softening(case["eps"])
        st.update(system=s, x=x, v=v)
    elif kind == "ensemble":
        off, m, r, x, v = _ensemble(case, seed)
        st["ensemble"] = Ensemble(off, m, x, v, r=r, dt=ENSEMBLE_DT)
    elif kind == "adjoint":
        m, x, v = _bodies(case, seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        for k, a in (("m", m), ("x0", x), ("v0", v)):
            st[k] = torch.tensor(a, device="cuda").requires_grad_()
        st["gx"], st["gv"] = _upstream(case, g)
    else:
        c = _comet(case, seed)
        st["stage"] = c
        st["system"] = gtd.System(c["m"], c["x"], c["v"], r=c["r"], rest=c["rest"], timestep=COMET_DT,
                                  num_iterations=100, units_format="M1:1,D1:1,T1:1", collisions=3)
    return st


def _upstream(case, g):
    """Gradients of a loss with respect to the final positions and velocities, each of unit order in
    its own scale."""
    gx = torch.randn((case["n"], 3), dtype=torch.float64, device="cuda", generator=g) / AU
    gv = torch.randn((case["n"], 3), dtype=torch.float64, device="cuda", generator=g) / 2e4
    return gx, gv


# ---- passes ---------------------------------------------------------------------------------------

def _run_force(st):
    case = st["case"]
    mixed = case["precision"] == "mixed"
    _lib.check(st["lib"].gtd_direct_accelerations_noalloc(
        case["n"], st["pm4"].data_ptr(), G_DEFAULT, _lib.PREC_MIXED if mixed else _lib.PREC_F64,
        st["acc"].data_ptr(), torch.cuda.current_stream().cuda_stream))
    return st["acc"].float() if mixed else st["acc"]


def _run_direct(st):
    s, case = st["system"], st["case"]
    s.x, s.v = st["x"], st["v"]
    s.evolve(METHODS[case["method"]])
    out = {"x": s.x, "v": s.v, "a": s.a.astype(np.float32) if case["precision"] == "mixed" else s.a}
    if case["energy"]:
        out["energy"] = s.energy()
    return out


def _run_bh_step(st):
    s = st["system"]
    s.x, s.v = st["x"], st["v"]
    s.evolve(METHODS["kdk"] | BARNES_HUT)
    return {"x": s.x, "v": s.v, "a": s.a.astype(np.float32) if st["case"]["tree"] == "float" else s.a}


def _run_bh_force(st):
    single = st["case"]["tree"] == "float"
    a, count = st["system"].bh_accelerations(single)
    return {"a": a.astype(np.float32) if single else a, "count": count}


def _run_ensemble(st):
    e = st["ensemble"]
    e.evolve(st["case"]["steps"])
    systems = e.state()
    count, merges, _ = e.counts()
    total = len(e.m)
    out = {"m": np.zeros(total), "r": np.zeros(total), "x": np.zeros((total, 3)), "v": np.zeros((total, 3)),
           "a": np.zeros((total, 3), np.float32)}
    for first, system in zip(e.offsets, systems):  # survivors first, in each system's own range
        for k, a in out.items():
            a[first:first + len(system[k])] = system[k]
    return {**out, "count": count, "merges": merges}


def _run_adjoint(st):
    x0, v0, m = st["x0"], st["v0"], st["m"]
    xT, vT = leapfrog_final_state(x0, v0, m, G_DEFAULT, HOUR, st["case"]["steps"])
    gx, gv, gm = torch.autograd.grad((xT, vT), (x0, v0, m), (st["gx"], st["gv"]))
    return {"x": xT.detach(), "v": vT.detach(), "gx": gx, "gv": gv, "gm": gm}


def _run_comet(st):
    s, c = st["system"], st["stage"]
    s.x, s.v, s.rest = c["x"], c["v"], c["rest"]
    centre = gtd.RestFromCom(c["min_cor"], c["max_cor"], c["scale_factor"], c["n_exp"], c["com"])
    s.evolve(METHODS["kdk"], gtd.WhileRestBelow(c["min_max_cor"], COMET_PROBING), None, centre,
             max_steps=st["case"]["steps"])
    return {"x": s.x, "v": s.v, "rest": s.rest, "com": centre.com, "steps": s.steps_taken}


_RUN = {"force": _run_force, "direct": _run_direct, "bh_step": _run_bh_step, "bh_force": _run_bh_force,
        "ensemble": _run_ensemble, "adjoint": _run_adjoint, "comet": _run_comet}


def run(state):
    return _RUN[state["kind"]](state)


# ---- work -----------------------------------------------------------------------------------------

def work(case):
    kind, n = case["kind"], case.get("n", 0)
    pairs = n * (n - 1) / 2
    if kind == "force":
        return {"bytes": 56 * n, "flops": PAIR_FLOPS * pairs}
    if kind == "direct":
        evals = case["steps"] * (2 if case["method"] in ("modified_euler", "midpoint") else 1)
        evals += (1 if case["method"] == "kdk" else 0) + (0.5 if case["energy"] else 0)
        return {"bytes": (72 + 88) * n, "flops": PAIR_FLOPS * pairs * evals}
    if kind in ("bh_step", "bh_force"):
        # accepted cells per octree level around a body, (4 pi / 3) (2^3 - 1) / theta^3, over log8(n) levels
        inter = min(n - 1, 29.3 / case["theta"] ** 3 * math.log(n, 8))
        walks = case["steps"] + 1 if kind == "bh_step" else 1
        return {"bytes": (72 + 88) * n, "flops": 20 * n * inter * walks}
    if kind == "ensemble":
        # sizes are uniform on 3 .. n_max
        k = np.arange(3, case["n_max"] + 1, dtype=np.float64)
        total = case["systems"] * float((k * (k - 1) / 2).mean())
        return {"bytes": case["systems"] * float(k.mean()) * 200, "flops": PAIR_FLOPS * total * case["steps"]}
    if kind == "adjoint":
        return {"bytes": 200 * n, "flops": (PAIR_FLOPS + VJP_PAIR_FLOPS) * pairs * (case["steps"] + 1)}
    # comet: the force, and a squared distance against a squared reach for every pair
    return {"bytes": 200 * n, "flops": (PAIR_FLOPS + 10) * pairs * (case["steps"] + 1)}


# ---- the same outputs in 64 bits --------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _chunks(n, width):
    rows = max(1, (1 << 26) // max(width, 1))
    return ((b, min(n, b + rows)) for b in range(0, n, rows))


def _pair(x, rows):
    """Separations (3 matrices) and r^-1 (0 for the pair of a body with itself) of rows of bodies."""
    d = [x[None, :, k] - x[rows, None, k] for k in range(3)]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    return d, torch.where(r2 > 0, r2.rsqrt(), torch.zeros_like(r2))


def _force(x, m, G):
    out = torch.empty_like(x)
    for b, e in _chunks(len(x), len(x)):
        d, inv = _pair(x, slice(b, e))
        s = inv * inv * inv * m
        for k in range(3):
            out[b:e, k] = G * (s * d[k]).sum(1)
    return out


def _evolve(x, v, m, G, h, steps, method, force=_force):
    """(x, v, a) after `steps`, a being the last acceleration the method evaluates for its state."""
    a = force(x, m, G) if method == "kdk" else None
    for _ in range(steps):
        if method == "kdk":
            v = v + 0.5 * h * a
            x = x + h * v
            a = force(x, m, G)
            v = v + 0.5 * h * a
        elif method == "dkd":
            x = x + 0.5 * h * v
            a = force(x, m, G)
            v = v + h * a
            x = x + 0.5 * h * v
        elif method == "euler":
            a = force(x, m, G)
            x, v = x + h * v, v + h * a
        else:
            a = force(x, m, G)
            hp = h if method == "modified_euler" else 0.5 * h
            vp = v + hp * a
            ap = force(x + hp * v, m, G)
            if method == "modified_euler":
                x, v = x + 0.5 * h * (v + vp), v + 0.5 * h * (a + ap)
            else:
                x, v = x + h * vp, v + h * ap
    return x, v, a


def _energy(x, v, m, G):
    pe = 0.0
    for b, e in _chunks(len(x), len(x)):
        _, inv = _pair(x, slice(b, e))
        pe -= 0.5 * G * float((m[b:e] * (inv * m).sum(1)).sum())
    ke = 0.5 * float((m * (v * v).sum(1)).sum())
    return ke, pe, (m[:, None] * v).sum(0), (m[:, None] * x).sum(0) / m.sum()


def _tree_force(x, m, G, theta, eps):
    """Accelerations by the octree walk: cells of the padded root cube split at their middles, a cell
    taken when width / distance < theta, a body never meeting its own leaf."""
    lo, hi = x.min(0).values, x.max(0).values
    edge = (hi - lo).max()
    origin, edge = lo - edge / 20, edge + edge / 10
    low = origin.repeat(len(x), 1)
    high = (origin + edge).repeat(len(x), 1)
    code = torch.zeros(len(x), dtype=torch.int64, device=x.device)
    for _ in range(21):
        mid = (low + high) * 0.5
        up = x >= mid
        low, high = torch.where(up, mid, low), torch.where(up, high, mid)
        code = (code << 3) | (up[:, 0].long() | (up[:, 1].long() << 1) | (up[:, 2].long() << 2))
    code, order = code.sort()
    xs, ms = x[order], m[order]
    levels = []  # per depth: prefix, bodies, first body, centre of mass, mass
    for depth in range(22):
        prefix, inverse, count = torch.unique_consecutive(code >> (63 - 3 * depth), return_inverse=True,
                                                          return_counts=True)
        mass = torch.zeros(len(prefix), dtype=x.dtype, device=x.device).index_add_(0, inverse, ms)
        com = torch.zeros((len(prefix), 3), dtype=x.dtype, device=x.device).index_add_(0, inverse, ms[:, None] * xs)
        levels.append((prefix, count, count.cumsum(0) - count, com / mass[:, None], mass))
        if int(count.max()) == 1:
            break
    acc = torch.zeros_like(xs)
    for b, e in _chunks(len(x), 4096):
        body = torch.arange(b, e, device=x.device)
        cell = torch.zeros_like(body)
        for depth in range(1, len(levels)):
            parent = levels[depth - 1][0][cell]
            prefix, count, first, com, mass = levels[depth]
            start = torch.searchsorted(prefix, parent << 3)
            size = torch.searchsorted(prefix, (parent + 1) << 3) - start
            body = body.repeat_interleave(size)
            offset = torch.arange(len(body), device=x.device) - (size.cumsum(0) - size).repeat_interleave(size)
            cell = start.repeat_interleave(size) + offset
            d = com[cell] - xs[body]
            r2 = (d * d).sum(1)
            single = count[cell] == 1
            take = torch.where(single, first[cell] != body, (edge * 0.5 ** depth) ** 2 < theta * theta * r2)
            inv = (r2[take] + eps * eps).rsqrt()
            acc.index_add_(0, body[take], (G * mass[cell[take]] * inv ** 3)[:, None] * d[take])
            down = ~take & ~single
            body, cell = body[down], cell[down]
    out = torch.empty_like(acc)
    out[order] = acc
    return out


def _exact_adjoint(x, v, m, gx, gv, G, h, steps):
    a = _force(x, m, G)
    path = [x]
    for _ in range(steps):
        v = v + 0.5 * h * a
        x = x + h * v
        a = _force(x, m, G)
        v = v + 0.5 * h * a
        path.append(x)
    lx, lv, mu = gx.clone(), gv.clone(), torch.zeros_like(m)
    for k in range(steps, -1, -1):  # kicks and drifts in reverse
        w = (0.5 * h if k in (0, steps) else h) * lv
        xk, mk = path[k].detach().requires_grad_(), m.detach().requires_grad_()
        for b, e in _chunks(len(x), 4 * len(x)):
            d = [xk[None, :, j] - xk[b:e, None, j] for j in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            own = torch.arange(b, e, device=x.device)[:, None] == torch.arange(len(x), device=x.device)[None, :]
            s = torch.where(own, torch.ones_like(r2), r2).pow(-1.5).masked_fill(own, 0.0) * mk
            kick = sum((w[b:e, j] * G * (s * d[j]).sum(1)).sum() for j in range(3))
            dx, dm = torch.autograd.grad(kick, (xk, mk))
            lx, mu = lx + dx, mu + dm
        if k:
            lv = lv + h * lx
    return {"x": x, "v": v, "gx": lx, "gv": lv, "gm": mu}


def _exact_ensemble(case, seed):
    off, m, r, x, v = (torch.tensor(a, device=_device()) for a in _ensemble(case, seed))
    outs = []
    for b, e in zip(off[:-1].tolist(), off[1:].tolist()):
        mk, rk, apart = m[b:e], r[b:e], []

        def force(p, masses, G):
            d = p[None, :, :] - p[:, None, :]
            r2 = (d * d).sum(2).fill_diagonal_(math.inf)
            apart.append((r2.sqrt() - rk[None, :] - rk[:, None]).min())
            return G * ((masses * r2.pow(-1.5))[:, :, None] * d).sum(1)

        outs.append(_evolve(x[b:e], v[b:e], mk, G_DEFAULT, ENSEMBLE_DT, case["steps"], "kdk", force))
        if float(torch.stack(apart).min()) <= 0:
            return None  # bodies merge: the states that follow are not this sum's
    out = {k: torch.cat([o[j] for o in outs]) for j, k in enumerate(("x", "v", "a"))}
    return {**out, "m": m, "r": r, "count": None, "merges": None}


def _bounce(x, v, m, r, rest):
    """The restitution of overlapping bodies: for each body the later ones it overlaps, nearest first,
    their momenta along the separation taken before any of that body's impulses."""
    dist = np.sqrt(((x[:, None] - x[None]) ** 2).sum(2))
    over = np.triu(dist < r[:, None] + r[None], 1)
    for o in np.flatnonzero(over.any(1)):
        hits = sorted(np.flatnonzero(over[o]), key=lambda i: dist[o, i])
        axes = [(x[i] - x[o]) / dist[o, i] for i in hits]
        before = [(v[o] @ u, v[i] @ u) for i, u in zip(hits, axes)]
        for i, u, (vo, vi) in zip(hits, axes, before):
            if not (vo > 0 or vi < 0) or (vo <= 0 and vi < 0 and vo < vi) or (vo > 0 and vi >= 0 and vo < vi):
                continue
            total, mass, e = m[o] * vo + m[i] * vi, m[o] + m[i], 0.5 * (rest[o] + rest[i])
            v[i] += ((total + m[o] * e * (vo - vi)) / mass - vi) * u
            v[o] += ((total - m[i] * e * (vo - vi)) / mass - vo) * u


def _exact_comet(case, seed):
    c = _comet(case, seed)
    G = gtd.parse_units("M1:1,D1:1,T1:1")
    x, v, m, r, rest, com = c["x"].copy(), c["v"].copy(), c["m"], c["r"], c["rest"].copy(), c["com"].copy()

    def force():
        d = x[None] - x[:, None]
        r2 = (d * d).sum(2)
        np.fill_diagonal(r2, np.inf)
        return G * ((m * r2 ** -1.5)[:, :, None] * d).sum(1)

    a = force()
    for _ in range(case["steps"]):
        v += 0.5 * COMET_DT * a
        x += COMET_DT * v
        a = force()
        v += 0.5 * COMET_DT * a
        com = (com + x.sum(0)) / len(m)
        far = np.sqrt(((x - com) ** 2).sum(1)) ** c["n_exp"]
        rest = c["max_cor"] - (c["max_cor"] - c["min_cor"]) * far / (far + c["scale_factor"])
        _bounce(x, v, m, r, rest)
    return {"x": x, "v": v, "rest": rest, "com": com, "steps": None}


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    if kind == "comet":
        return _exact_comet(case, seed)
    m, x, v = (torch.tensor(a, device=_device()) for a in _bodies(case, seed))
    if kind == "force":
        return _force(x, m, G_DEFAULT)
    if kind == "direct":
        x, v, a = _evolve(x, v, m, G_DEFAULT, HOUR, case["steps"], case["method"])
        out = {"x": x, "v": v, "a": a}
        if case["energy"]:
            out["energy"] = _energy(x, v, m, G_DEFAULT)
        return out
    if kind == "adjoint":
        gx, gv = _upstream(case, torch.Generator(device="cuda").manual_seed(seed))
        return _exact_adjoint(x, v, m, gx, gv, G_DEFAULT, HOUR, case["steps"])
    if kind == "bh_force":
        return {"a": _tree_force(x, m, G_DEFAULT, case["theta"], case["eps"]), "count": None}
    if n * (case["steps"] + 1) > 600000:
        return None  # over twenty seconds

    def walk(p, masses, G):
        return _tree_force(p, masses, G, case["theta"], 0.0)

    a = walk(x, m, G_DEFAULT)
    v = v + 0.5 * BH_DT * a
    for _ in range(case["steps"]):
        x = x + BH_DT * v
        a = walk(x, m, G_DEFAULT)
        v = v + BH_DT * a  # the velocities stay half a step ahead
    return {"x": x, "v": v, "a": a}
