"""The work that programs have this framework do, as cases that can be timed.

Every scene is a piece of a settled pile, as simulations hold it nearly all of
the time: spheres of 4 to 6 mm cut out of the committed 200,000-sphere column
(workloads.column_settled) at a place, in an orientation and with small random
velocities that come from the seed, in an open box of their own.  The ball on
the ground of scenes.ball_on_ground is the smallest scene there is.

Kinds of case, each through the public calls of dvide_b200._native:

* "step"    a scene put into a given state, stepped, and its state and contact
            forces read back (System::DoTimeStep in a driver's loop), with the
            APGD, PGJ or PGS solver, in FP64 or in mixed precision;
* "batch"   many independent scenes stepped together;
* "serve"   a burst of requests through the continuous-batching server;
* "inspect" what a program reads of a state: contacts, forces, violation,
            energies.
"""
import math

import numpy as np
import torch

from dvide_b200 import _native as N
from dvide_b200 import scenes, workloads

CONTACTS_PER_SPHERE = 3.7   # in the settled column
TYPICAL_ITERATIONS = 150    # warm-started solves of a pile that still moves
SOLVERS = {"apgd": N.DV_SOLVER_APGD, "pgj": N.DV_SOLVER_PGJ, "pgs": N.DV_SOLVER_PGS}
PRECISIONS = {"fp64": N.DV_PREC_FP64, "mixed": N.DV_PREC_MIXED}


def _step(name, n, steps, precision="fp64", solver="apgd", warm=1, cap=500, refine=0, option=""):
    return dict(name=name, kind="step", n=n, steps=steps, precision=precision, solver=solver,
                warm=warm, cap=cap, refine=refine, option=option)


def _batch(name, count, nmin, nmax, steps, precision="mixed", solver="apgd", cap=500, refine=500,
           graph=True):
    return dict(name=name, kind="batch", count=count, nmin=nmin, nmax=nmax, steps=steps,
                precision=precision, solver=solver, warm=1, cap=cap, refine=refine, graph=graph)


def _serve(name, count, nmin, nmax, steps):
    return dict(name=name, kind="serve", count=count, nmin=nmin, nmax=nmax, steps=steps,
                precision="mixed", solver="apgd", warm=1, cap=500, refine=500)


def listed():
    return [
        # the smallest scene: one ball on the ground, a driver's call per step
        _step("ball", 1, 1, warm=0, cap=100000),
        # the 1,000-sphere box that the parity tests and small studies step, ten steps a frame
        _step("box_1000", 1000, 10),
        # a pile with DOFs pinned by bilateral rows, as drivers hold walls and probes
        _step("pile_5003_rows", 5003, 4, option="rows"),
        # an everyday pile in mixed precision with FP64 refinement
        _step("pile_20011_mixed", 20011, 4, precision="mixed", refine=500),
        # the 200,000-sphere column at rest: every solve runs to the cap
        _step("column", 200000, 1),
        # the same column in mixed precision
        _step("column_mixed", 200000, 1, precision="mixed"),
        # the Jacobi solver, System(5), on a small pile
        _step("pgj_3001", 3001, 2, solver="pgj", warm=0, cap=200),
        # post-processing of a state: collision detection and every contact quantity
        _step_inspect("inspect_30011", 30011),
        # a parameter study of small scenes in FP64, replayed from a graph
        _batch("batch_64_fp64", 64, 50, 1000, 4, precision="fp64", refine=0),
        # scenes of log-uniform sizes 100 to 20,000 in mixed precision with refinement
        _batch("batch_256_mixed", 256, 100, 20000, 3),
        # the Gauss-Seidel solver, System(6): one thread sweeps a scene, so many scenes
        _batch("batch_48_pgs", 48, 20, 120, 1, precision="fp64", solver="pgs", cap=30, refine=0),
        # a burst of requests, of different lengths, through the server
        _serve("serve_40", 40, 100, 5000, 6),
    ]


def _step_inspect(name, n):
    return dict(name=name, kind="inspect", n=n, steps=1, precision="fp64", solver="apgd", warm=1,
                cap=100, refine=0, option="")


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["batch"] * 2 + ["serve", "inspect"])
    if kind == "step":
        solver = rng.choice(["apgd"] * 5 + ["pgj"])
        precision = rng.choice(["fp64", "fp64", "mixed"])
        n = _log_int(rng, 2, 120000 if solver == "apgd" else 20000)
        option = ""
        if solver == "apgd" and precision == "fp64":
            option = rng.choice(["", "", "rows", "anti"])
        warm = 0 if solver == "pgj" else rng.choice([0, 1, 1, 2])
        c = _step("", n, rng.randint(3, max(3, min(8, 40000 // n))) if warm else 1, precision,
                  solver, warm,
                  cap=rng.choice([100, 200]) if solver == "pgj" else rng.choice([200, 500]),
                  refine=rng.choice([0, 500]) if precision == "mixed" and solver == "apgd" else 0,
                  option=option)
    elif kind == "batch":
        count = _log_int(rng, 3, 200)
        nmin = _log_int(rng, 2, 200)
        solver = rng.choice(["apgd"] * 4 + ["pgj", "pgs"])
        precision = "fp64" if solver == "pgs" else rng.choice(["fp64", "mixed"])
        nmax = {"apgd": 200000 // count, "pgj": 40000 // count, "pgs": 150}[solver]
        nmax = max(nmin + 1, min(nmax, 15000))
        c = _batch("", count, nmin, nmax, 3 if solver == "apgd" else 1, precision, solver,
                   cap={"apgd": 500, "pgj": 150, "pgs": 20}[solver],
                   refine=500 if precision == "mixed" and solver == "apgd" else 0,
                   graph=rng.random() < 0.7)
    elif kind == "serve":
        nmin = _log_int(rng, 10, 500)
        c = _serve("", _log_int(rng, 4, 60), nmin, nmin * rng.randint(2, 10), rng.randint(2, 6))
    else:
        c = _step_inspect("", _log_int(rng, 50, 60000))
    del c["name"]
    return c


# ---- scenes ---------------------------------------------------------------------------------

_COLUMN = []


def _column():
    """Positions, radii and velocities of the settled column's spheres."""
    if not _COLUMN:
        s = workloads.column_settled()
        _COLUMN.append((s.pos[5:], s.geom[5:, 0].copy(), s.vel[5:]))
    return _COLUMN[0]


def _cut(rng, place, n, scale):
    """The lowest n spheres inside a square of the settled column's cross-section
    (about as wide as they stand high), in an open box that just holds them;
    scale 10 makes spheres of 4 to 6 cm, as in scenes.settling_box."""
    pos, r, vel = _column()
    side = min(0.4, (n / 1.18e6) ** (1.0 / 3.0) + 0.004)
    while True:
        x0, y0 = place.uniform(-0.2, 0.2 - side, size=2) if side < 0.4 else (-0.2, -0.2)
        at = np.nonzero((pos[:, 0] >= x0) & (pos[:, 0] <= x0 + side) &
                        (pos[:, 1] >= y0) & (pos[:, 1] <= y0 + side))[0]
        if at.size >= n:
            break
        side = min(0.4, side * 1.1)
    if at.size > n:
        at = np.sort(at[np.argpartition(pos[at, 2], n - 1)[:n]])
    p, q, v = pos[at] * scale, r[at] * scale, vel[at].copy()
    for axis in (0, 1):
        if rng.random() < 0.5:
            p[:, axis] *= -1.0
            v[:, axis] *= -1.0
    v += rng.normal(0.0, 1e-3, size=v.shape)
    lo, hi = (p - q[:, None]).min(axis=0), (p + q[:, None]).max(axis=0)
    boxes = scenes.open_box(hi[0] - lo[0], hi[1] - lo[1], hi[2] + 0.1, thick=0.05 * scale,
                            cx=0.5 * (lo[0] + hi[0]), cy=0.5 * (lo[1] + hi[1]))
    p[:, 2] -= min(0.0, lo[2])
    params = scenes.default_params(gravity=(0.0, 0.0, -scenes.G), h=5e-4, mu=0.3, tolerance=1e-4)
    return scenes._assemble(boxes, p, q, 2500.0, params, "cut", spheres_vel=v)


def _scene(case, rng, n, place):
    if n == 1:
        sc = scenes.ball_on_ground()
        sc.vel[1] = rng.normal(0.0, 1e-2, size=3)
    else:
        # the Jacobi and Gauss-Seidel solvers start from unit impulses, which suit heavy spheres
        sc = _cut(rng, place, n, 1.0 if case["solver"] == "apgd" else 10.0)
    sc.params.update(max_iterations=case["cap"], warm_start=case["warm"],
                     solver=SOLVERS[case["solver"]], refine_iterations=case["refine"])
    if case["solver"] != "apgd":
        sc.params["tolerance"] = 1e-8
    option = case.get("option", "")
    if option == "anti":
        sc.params["anti_relaxation"] = 1
    if option == "rows":
        # every hundredth sphere, 40 at most, held in x and y
        first = int(np.argmax(sc.fixed == 0))
        held = first + np.arange(0, n, 100)[:40]
        sc.bilateral = [(3 * int(b) + k, -1, 0.0, 0.0) for b in held for k in (0, 1)]
    return sc


def _scenes(case, seed):
    """The case's scenes.  A pass that starts from a given state with warm-started solves takes
    its first impulses from the pass before, so such a case steps several times a pass: each
    solve then starts from another step's impulses, as in a running simulation."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "inspect":
        # one place for every seed: the number of contacts is the case's
        return [_scene(case, rng, case["n"], np.random.default_rng(case["n"]))]
    if case["kind"] == "step":
        return [_scene(case, rng, case["n"], rng)]
    # sizes at the middles of equal parts of the range's logarithm, in the seed's order
    at = (rng.permutation(case["count"]) + 0.5) / case["count"]
    return [_scene(case, rng, int(case["nmin"] * (case["nmax"] / case["nmin"]) ** x), rng)
            for x in at]


# ---- what is measured -----------------------------------------------------------------------

def _pinned(a):
    """A copy of `a` in page-locked memory, where a driver keeps what it sends and reads often."""
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def prepare(case, seed):
    made = _scenes(case, seed)
    precision = PRECISIONS[case["precision"]]
    state = dict(case=case, scenes=made)
    if case["kind"] in ("step", "batch"):
        nb = sum(sc.nb for sc in made)
        state["out"] = _pinned(np.zeros((nb, 3))), _pinned(np.zeros((nb, 3)))
    if case["kind"] in ("step", "inspect"):
        sc = made[0]
        state["p"], state["v"] = _pinned(sc.pos), _pinned(sc.vel)
        state["scene"] = N.NativeScene.from_scene(sc, precision=precision)
        if case["kind"] == "inspect":
            state["scene"].collide()
            state["scene"].solve()
    elif case["kind"] == "batch":
        state["p"] = _pinned(np.concatenate([sc.pos for sc in made]))
        state["v"] = _pinned(np.concatenate([sc.vel for sc in made]))
        state["batch"] = N.NativeBatch(made, precision=precision)
        if case["graph"]:
            state["batch"].set_graph(True)
    else:
        state["server"] = N.NativeServer(precision=precision, steps_per_round=2)
        state["steps"] = [case["steps"] * (1 + i % 2) for i in range(len(made))]
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        s = state["scene"]
        s.set_state(state["p"], state["v"])
        s.step(case["steps"])
        p, v = state["out"]
        s.state_into(p, v)
        return {"p": p, "v": v, "f": s.fcontact()}
    if case["kind"] == "batch":
        b = state["batch"]
        b.set_state(-1, state["p"], state["v"])
        b.step(case["steps"])
        p, v = state["out"]
        b.state_into(p, v)
        return {"p": p, "v": v, "contacts": np.array([x["num_contacts"] for x in b.scene_stats()])}
    if case["kind"] == "inspect":
        s = state["scene"]
        s.set_state(state["p"], state["v"])
        s.collide()
        a, b, nP, loc = s.contacts()
        normal, friction = s.contact_forces()
        return {"a": a.astype(np.int64), "b": b.astype(np.int64), "nP": nP, "loc": loc,
                "normal": normal, "friction": friction, "violation": s.ccp_violation(),
                "energies": np.array(s.energies())}
    server = state["server"]
    ids = [server.submit(sc, k) for sc, k in zip(state["scenes"], state["steps"])]
    while server.round():
        pass
    done = {x["id"]: x for x in server.poll()}
    got = [server.result_state(i) for i in ids]
    return {"p": np.concatenate([g[0] for g in got]), "v": np.concatenate([g[1] for g in got]),
            "contact_steps": np.array([done[i]["contact_steps"] for i in ids])}


def _bodies_and_steps(case):
    if case["kind"] in ("step", "inspect"):
        return case["n"], case["steps"]
    mean = (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
    return case["count"] * mean, case["steps"] * (1.5 if case["kind"] == "serve" else 1)


def work(case):
    """Collision detection (positions in, contacts out), then per iteration the solver's vectors
    read and written once with one product N x, then the update; contacts and iterations as such
    piles have them."""
    nb, steps = _bodies_and_steps(case)
    if case["kind"] == "step" and nb == 1:
        nc, iterations = 1.0, 10.0
    else:
        nc = CONTACTS_PER_SPHERE * nb
        # the whole column runs to the cap
        iterations = float(case["cap"] if nb > 150000 else min(case["cap"], TYPICAL_ITERATIONS))
    word = 4 if case["precision"] == "mixed" else 8
    detect = 120 * nb + 112 * nc
    if case["kind"] == "inspect":
        # contacts, forces and the violation's items out; no solve
        return {"bytes": detect + 48 * nb + (64 + 48 + 72 + 32) * nc, "flops": 150 * nc + 20 * nb}
    # x, r and n of a contact in, N x, the next iterate and q out; w and q of a body
    vectors = {"apgd": 38 * word * nc + 8 * word * nb, "pgj": 19 * word * nc + 8 * word * nb,
               "pgs": 19 * word * nc + 8 * word * nb}[case["solver"]]
    flops = {"apgd": 210, "pgj": 120, "pgs": 160}[case["solver"]] * nc + 20 * nb
    return {"bytes": steps * (detect + iterations * vectors + 136 * nc + 96 * nb) + 96 * nb,
            "flops": steps * (iterations * flops + 200 * nc)}


# ---- the same in 64 bits, in plain numpy ----------------------------------------------------

def exact(case, seed):
    """FP64 steps of small APGD and PGJ scenes, and inspections.  The mixed solves stop at the
    tolerance on another iterate than 64-bit ones, so they have no such value; the larger scenes,
    the rows and the Gauss-Seidel sweeps (one contact after another) would take too long."""
    if case["precision"] != "fp64" or case["solver"] == "pgs" or case.get("option"):
        return None
    if case["kind"] == "inspect":
        sc = _scenes(case, seed)[0]
        c = _contacts(sc)
        gamma = _apgd(sc, c, _impulse(sc), np.zeros((len(c["a"]), 3)))
        g, h = gamma, sc.params["h"]
        minv, _ = _inverse_mass(sc)
        m = np.where(minv > 0, sc.mass, 0.0)
        vn = c["gap"] / h + np.einsum("ij,ij->i", c["F"][:, 0], sc.vel[c["a"]] - sc.vel[c["b"]])
        cone = np.minimum(sc.params["mu"] * g[:, 0] - np.hypot(g[:, 1], g[:, 2]), 0.0)
        force = m[:, None] * np.array(sc.params["gravity"])
        return {"a": c["a"], "b": c["b"],
                "nP": np.concatenate([c["F"][:, 0], c["gap"][:, None]], axis=1), "loc": c["loc"],
                "normal": g[:, :1] * c["F"][:, 0] / h,
                "friction": (g[:, 1:2] * c["F"][:, 1] + g[:, 2:] * c["F"][:, 2]) / h,
                "violation": np.array([min(g[:, 0].min(), 0.0), min(vn.min(), 0.0),
                                       float((g[:, 0] * vn).sum()), math.sqrt((cone ** 2).sum())]),
                "energies": np.array([0.5 * (m[:, None] * sc.vel ** 2).sum(),
                                      -(force * sc.pos).sum()])}
    if case["kind"] != "step" or case["n"] * case["steps"] > 12000 or case["warm"] == 2:
        return None
    sc = _scenes(case, seed)[0]
    gamma = np.zeros((sc.nb, 3))
    for _ in range(case["steps"]):
        h = sc.params["h"]
        minv, _ = _inverse_mass(sc)
        c, k = _contacts(sc), _impulse(sc)
        f = np.zeros((sc.nb, 3))
        if len(c["a"]):
            start = np.tile([1.0, 0.0, 0.0], (len(c["a"]), 1))
            if case["solver"] == "pgj":
                gamma = _pgj(sc, c, k, start)
            else:
                if case["warm"]:
                    start = np.zeros((len(c["a"]), 3))
                    start[:len(gamma)] = gamma[:len(start)]
                gamma = _apgd(sc, c, k, start)
            f = _transposed(sc, c, gamma)
        sc.vel = minv[:, None] * (k + f)
        sc.pos = sc.pos + h * sc.vel
    return {"p": sc.pos, "v": sc.vel, "f": f / h}


def _unit(v):
    """v over its length, the reciprocal square root taken in single precision as the step
    defines it."""
    d = (v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1] + v[:, 2] * v[:, 2]).astype(np.float32)
    return v * (np.float32(1.0) / np.sqrt(d)).astype(np.float64)[:, None]


def _pairs(pos, radius, reach):
    """Index pairs i < j of spheres nearer than their radii and `reach` allow, by cells."""
    w = 2.0 * radius.max() + reach
    cell = np.floor((pos - pos.min(axis=0)) / w).astype(np.int64) + 1
    dims = cell.max(axis=0) + 2
    key = cell[:, 0] + dims[0] * (cell[:, 1] + dims[1] * cell[:, 2])
    order = np.argsort(key, kind="stable")
    sorted_key = key[order]
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                want = key + dx + dims[0] * (dy + dims[1] * dz)
                lo = np.searchsorted(sorted_key, want, "left")
                n = np.searchsorted(sorted_key, want, "right") - lo
                i = np.repeat(np.arange(len(pos)), n)
                j = order[np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n) + np.repeat(lo, n)]
                d = pos[j] - pos[i]
                near = (i < j) & ((d * d).sum(axis=1) <= (radius[i] + radius[j] + reach) ** 2)
                found.append(np.stack([i[near], j[near]], axis=1))
    return np.concatenate(found)


def _contacts(sc):
    env = sc.params["envelope"]
    ball = np.nonzero(sc.geom[:, 1] == 0)[0]
    box = np.nonzero(sc.geom[:, 1] != 0)[0]
    a, b, gap, normal, loc = [], [], [], [], []
    r = sc.geom[:, 0]
    ij = _pairs(sc.pos[ball], r[ball], 2.0 * env)
    if len(ij):
        i, j = ball[ij[:, 0]], ball[ij[:, 1]]
        d = sc.pos[j] - sc.pos[i]
        length = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]).astype(np.float32))
        pen = (r[i] + r[j]) - length.astype(np.float64)
        k = pen >= -env
        u = _unit(d[k])
        a.append(i[k]), b.append(j[k]), gap.append(-pen[k]), normal.append(-u)
        loc.append(sc.pos[i[k]] + u * r[i[k]][:, None])
    for x in box:  # the boxes come before the spheres
        lo, hi = sc.pos[x] - sc.geom[x], sc.pos[x] + sc.geom[x]
        p = sc.pos[ball]
        d = np.where(p < lo, p - lo, np.where(p > hi, p - hi, 0.0))
        pen = r[ball] - np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
        k = pen >= -env
        u = _unit(d[k])
        a.append(np.full(k.sum(), x)), b.append(ball[k]), gap.append(-pen[k]), normal.append(-u)
        loc.append(p[k] - u * r[ball[k]][:, None])
    a, b = np.concatenate(a), np.concatenate(b)
    order = np.lexsort((b, a))
    n = np.concatenate(normal)[order]
    with np.errstate(divide="ignore", invalid="ignore"):
        zero, one = np.zeros(len(n)), np.ones(len(n))
        u = np.stack([one, zero, -n[:, 0] / n[:, 2]], axis=1)
        flat = n[:, 2] == 0
        u[flat] = np.stack([-n[:, 2] / n[:, 0], zero, one], axis=1)[flat]
        along = flat & (n[:, 0] == 0)
        u[along] = np.stack([one, -n[:, 0] / n[:, 1], zero], axis=1)[along]
    u = _unit(u)
    F = np.stack([n, u, _unit(np.cross(n, u))], axis=1)
    return dict(a=a[order], b=b[order], gap=np.concatenate(gap)[order], F=F,
                loc=np.concatenate(loc)[order])


def _inverse_mass(sc):
    minv = np.where(sc.fixed != 0, 0.0, 1.0 / sc.mass)
    return minv, np.where(minv > 0, 1.0 / np.where(minv > 0, minv, 1.0), 0.0)


def _impulse(sc):
    minv, m = _inverse_mass(sc)
    f = np.where(minv > 0, sc.mass, 0.0)[:, None] * np.array(sc.params["gravity"])
    return sc.params["h"] * f + m[:, None] * sc.vel


def _transposed(sc, c, x):
    q = np.einsum("ckd,ck->cd", c["F"], x)
    return np.stack([np.bincount(c["a"], q[:, d], sc.nb) - np.bincount(c["b"], q[:, d], sc.nb)
                     for d in range(3)], axis=1)


def _times(c, w):
    return np.einsum("ckd,cd->ck", c["F"], w[c["a"]] - w[c["b"]])


def _project(x, mu):
    n, t = x[:, 0], np.sqrt(x[:, 1] ** 2 + x[:, 2] ** 2)
    inside = t < mu * n
    gone = ~inside & ((t < -(1.0 / mu) * n) | (np.abs(n) < 1e-14))
    pn = (t * mu + n) / (mu * mu + 1.0)
    with np.errstate(divide="ignore", invalid="ignore"):
        ratio = pn * mu / t
    y = np.stack([pn, ratio * x[:, 1], ratio * x[:, 2]], axis=1)
    y[inside] = x[inside]
    y[gone] = 0.0
    return y


def _system(sc, c, k):
    minv, _ = _inverse_mass(sc)
    r = _times(c, minv[:, None] * k)
    r[:, 0] += c["gap"] / sc.params["h"]
    return r, lambda x: _times(c, minv[:, None] * _transposed(sc, c, x))


def _apgd(sc, c, k, x):
    r, product = _system(sc, c, k)
    mu, tol = sc.params["mu"], sc.params["tolerance"]
    gd = 1.0 / len(x) ** 2
    lip = np.linalg.norm(product(x - 1.0)) / np.linalg.norm(x - 1.0)
    theta, y, Nx, best, least = 1.0, x, product(x), np.ones_like(x), 10e30
    Ny = Nx
    for _ in range(sc.params["max_iterations"]):
        g = Ny + r
        base = 0.5 * (y * Ny).sum() + (y * r).sum()
        while True:
            new = _project(y - g / lip, mu)
            Nn = product(new)
            step = new - y
            if 0.5 * (new * Nn).sum() + (new * r).sum() < base + (g * step).sum() + 0.5 * lip * (step * step).sum():
                break
            lip *= 2.0
        after = (-theta ** 2 + theta * math.sqrt(theta ** 2 + 4.0)) / 2.0
        beta = theta * (1.0 - theta) / (theta ** 2 + after)
        restart = (g * (new - x)).sum() > 0
        residual = np.abs((new - _project(new - gd * (Nn + r), mu)) / gd).max()
        if residual < least:
            least, best = residual, new
        if least < tol:
            break
        if restart:
            y, Ny, theta = new, Nn, 1.0
        else:
            y, Ny, theta = new + beta * (new - x), Nn + beta * (Nn - Nx), after
        x, Nx = new, Nn
        lip *= 0.9
    return best


def _pgj(sc, c, k, x):
    r, product = _system(sc, c, k)
    minv, _ = _inverse_mass(sc)
    mu, tol = sc.params["mu"], sc.params["tolerance"]
    scale = 3.0 / ((minv[c["a"]] + minv[c["b"]]) * (c["F"] ** 2).sum(axis=(1, 2)))

    def outside(z, s):
        return np.maximum(0.0, -(s * z[:, 0] - np.hypot(z[:, 1], z[:, 2]))).max()

    for i in range(sc.params["max_iterations"]):
        g = product(x) + r
        if i and max(outside(x, mu), outside(g, 1.0 / mu), np.abs((g * x).sum(axis=1)).max()) < tol:
            break
        x = (2.0 / 3.0) * _project(x - 0.3 * scale[:, None] * g, mu) + (1.0 / 3.0) * x
    return x
