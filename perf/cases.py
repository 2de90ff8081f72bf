"""Performance cases: what users of the library have it do, and the exact results to hold it to.

Every case is a whole call as a program makes it: the initial coefficients go from
pinned host memory to the device, the library advances them, and the solution comes
back to the host.  Kinds of case:

  solve      one mesh, matrix-free (HpgemAPISimplified), fixed steps
  adaptive   one mesh, embedded tableau with step rejection (computeOneTimeStepAdaptive)
  linear     one mesh, stored matrices (HpgemAPILinear)
  batch      many small 2D advection problems advanced together (Batch)
  served     a burst of mixed solves through the serving loop (Server)

A case's meshes are periodic unit squares or cubes.  `exact` restates the discontinuous
Galerkin semi-discretisation (basis functions, meshes, upwind and central fluxes,
Runge-Kutta steps) in plain numpy and torch in 64 bits, from the definitions alone.
"""
import math
import random

import numpy as np
import torch
from numpy.polynomial import legendre

import hpgem_b200
from hpgem_b200 import _native

PRECISION = {"fp64": _native.PRECISION_FP64, "fp32": _native.PRECISION_FP32, "bf16x3": _native.PRECISION_BF16X3}


# ---- the cases ------------------------------------------------------------------------
def listed():
    return [
        # the plain method's own configuration: a small 2D run, where latency and launches count
        _one("quad32_p2", "solve", "32x32", False, 2, "advection", "fp64", 100),
        # the headline run: 16.8 M coefficients, 200 steps, and a ragged box in the mixed form
        _one("hex64_p3", "solve", "64x64x64", False, 3, "advection", "fp64", 200),
        _one("hex_ragged_p3_fp32", "solve", "61x43x52", False, 3, "advection", "fp32", 100),
        # an ordinary 2D run on a rectangle whose sides are no powers of two
        _one("quad_ragged_p4", "solve", "150x210", False, 4, "advection", "fp64", 100),
        # 2D advection on triangles
        _one("tri_p3", "solve", "192x160", True, 3, "advection", "fp64", 100),
        # the acoustic wave on tetrahedra: the wave configuration, and a smaller run of higher order
        _one("tet32_wave_p2", "solve", "32x32x32", True, 2, "wave_upwind", "fp64", 60),
        _one("tet_wave_p3_fp32", "solve", "14x18x12", True, 3, "wave", "fp32", 80),
        # adaptive steps with the library's default tableau: a host decision after every try
        _one("tri_adaptive_p2", "adaptive", "48x64", True, 2, "advection", "fp64", 20, tableau="DormandPrince"),
        # applications that bring their own matrices, in full precision and on split-BF16 tiles
        _one("linear_hex_p3", "linear", "24x20x28", False, 3, "advection", "fp64", 60),
        _one("linear_tet_p2_bf16x3", "linear", "16x16x16", True, 2, "wave", "bf16x3", 40),
        # many problems at once: the batched set's shapes, and a burst of served requests
        {"name": "batch_fp32", "kind": "batch", "problems": 96, "mix": 4, "precision": "fp32", "steps": 50},
        {"name": "served_fp64", "kind": "served", "problems": 32, "mix": 5, "precision": "fp64", "steps": 120},
    ]


def _one(name, kind, cells, triangular, order, physics, precision, steps, tableau="RK4_4"):
    return {"name": name, "kind": kind, "cells": cells, "triangular": triangular, "order": order,
            "physics": physics, "precision": precision, "steps": steps, "tableau": tableau}


def draw(rng):
    """One more case: kinds, shapes, orders and forms as users mix them, sizes spread over
    the logarithm of the coefficient count, every side length drawn on its own."""
    kind = rng.choices(["solve", "adaptive", "linear", "batch", "served"], [10, 1, 2, 2, 1])[0]
    if kind in ("batch", "served"):
        return {"kind": kind, "problems": rng.randint(8, 96 if kind == "batch" else 32), "mix": rng.randrange(1 << 20),
                "precision": rng.choice(["fp64", "fp32"]), "steps": rng.randint(20, 60)}
    dim = rng.choice([2, 3])
    triangular = rng.random() < 0.5
    physics = rng.choice(["advection", "advection", "wave", "wave_upwind"])
    if kind == "linear":
        physics = "advection" if not triangular else rng.choice(["advection", "wave"])
    if not triangular and kind != "linear":
        physics = "advection"
    order = rng.randint(1, (5 if dim == 2 else 4) if physics == "advection" else (4 if dim == 2 else 3))
    if kind == "linear":
        order = min(order, 4 if dim == 2 else 3 if not triangular else 2)
    top = {"solve": 4e6, "adaptive": 1e6, "linear": 1e6}[kind]
    target = math.exp(rng.uniform(math.log(3e3), math.log(top)))
    nb = _basis_size(dim, triangular, order) * (dim + 1 if physics != "advection" else 1)
    per_cell = (2 if dim == 2 else 5) if triangular else 1
    side = (target / (nb * per_cell)) ** (1.0 / dim)
    cells = []
    for _ in range(dim):
        n = max(4, int(round(side * math.exp(rng.uniform(-0.3, 0.3)))))
        cells.append(n + n % 2 if triangular else n)  # periodic simplex meshes need even sides
    dof = nb * per_cell * math.prod(cells)
    steps = rng.randint(20, 100)
    if kind == "adaptive":
        steps = rng.randint(8, 20)
    steps = max(4, min(steps, int(3e8 / dof)))
    return {"kind": kind, "cells": "x".join(map(str, cells)), "triangular": triangular, "order": order,
            "physics": physics, "precision": "fp64" if kind == "adaptive" else rng.choice(["fp64", "fp32"]), "steps": steps,
            "tableau": "DormandPrince" if kind == "adaptive" else rng.choice(["RK4_4", "RK4_4", "RK3TVD", "DormandPrince"])}


def _basis_size(dim, triangular, p):
    if triangular:
        return (p + 1) * (p + 2) // 2 if dim == 2 else (p + 1) * (p + 2) * (p + 3) // 6
    return (p + 1) ** dim


def _problems(case):
    """The problems of a case as a list (one entry for a single mesh)."""
    if case["kind"] not in ("batch", "served"):
        cells = [int(v) for v in case["cells"].split("x")]
        rng = random.Random(case["cells"])
        return [_problem(rng, cells, case["triangular"], case["order"], case["physics"], case["steps"])]
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["problems"]):
        if case["kind"] == "batch":  # the batched set: 8^2 to 128^2 cells, quads or triangles, p = 1..5
            n = int(round(math.exp(rng.uniform(math.log(8), math.log(128)))))
            tri = rng.random() < 0.5
            out.append(_problem(rng, [n + n % 2 if tri else n] * 2, tri, rng.randint(1, 5), "advection", case["steps"]))
        else:  # the served stream: 2D and 3D, advection on quads and hexes, the wave on simplices
            wave, dim, p = rng.random() < 0.5, rng.choice([2, 3]), rng.randint(1, 4)
            target = math.exp(rng.uniform(math.log(1e3), math.log(4e5)))
            per = _basis_size(dim, wave, p) * ((dim + 1) * (2 if dim == 2 else 5) if wave else 1)
            n = max(4, int(round((target / per) ** (1.0 / dim))))
            steps = rng.randint(case["steps"] // 2, case["steps"])
            out.append(_problem(rng, [n + n % 2 if wave else n] * dim, wave, p, "wave" if wave else "advection", steps))
    return out


def _problem(rng, cells, triangular, order, physics, steps):
    dim = len(cells)
    a = [rng.gauss(0.0, 1.0) for _ in range(dim)]
    norm = math.sqrt(sum(v * v for v in a))
    dt = (0.1 if physics != "advection" else 0.2) / max(cells) / (2 * order + 1)
    return {"cells": cells, "dim": dim, "triangular": triangular, "order": order, "physics": physics,
            "vars": 1 if physics == "advection" else dim + 1, "a": [v / norm for v in a], "dt": dt, "steps": steps}


def _description(P):
    return hpgem_b200.structured_description(P["cells"], [0] * P["dim"], [1] * P["dim"], P["triangular"], True)


# ---- preparing and running ------------------------------------------------------------------
REL_ERROR = 1e-8  # of the adaptive steps, against the sum of the elements' norms


def prepare(case, seed):
    problems = _problems(case)
    host = [_pinned(_initial(P, seed + 7919 * i).cpu().numpy().reshape(-1)) for i, P in enumerate(problems)]
    state = {"case": case, "problems": problems, "u0": host, "out": [_pinned(np.zeros_like(h)) for h in host]}
    if case["kind"] == "served":
        state["server"] = hpgem_b200.Server(8 << 30, max_chunk=6, setup_threads=4, capacity=256)
        return state
    state["solvers"] = [_solver(case, P) for P in problems]
    if case["kind"] == "batch":
        state["batch"] = hpgem_b200.Batch(len(problems))
    return state


def _solver(case, P):
    kw = {"tableau": case.get("tableau", "RK4_4"), "precision": PRECISION[case["precision"]]}
    if case["kind"] == "linear":
        s = hpgem_b200.HpgemAPILinear(P["dim"], P["order"], P["physics"], advection=P["a"], **kw)
    elif P["physics"] == "advection":
        s = hpgem_b200.Advection(P["dim"], P["order"], P["a"], **kw)
    else:
        s = hpgem_b200.AcousticWave(P["dim"], P["order"], flux="upwind" if P["physics"] == "wave_upwind" else "central",
                                    **kw)
    return s.readMesh(_description(P))


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def run(state):
    case, problems, outs = state["case"], state["problems"], state["out"]
    if case["kind"] == "served":
        server = state["server"]
        ids = [server.submit(_description(P), P["order"], P["physics"], P["a"] if P["physics"] == "advection" else [1.0],
                             P["dt"], P["steps"], u0=u0, precision=PRECISION[case["precision"]], n_vars=P["vars"])
               for P, u0 in zip(problems, state["u0"])]
        outs = [server.poll(i, wait=True)[1] for i in ids]
        for i in ids:
            server.release(i)
        return np.concatenate(outs)
    solvers = state["solvers"]
    for s, u0 in zip(solvers, state["u0"]):
        s.setTimeIntegrationVector(0, u0)
    if case["kind"] == "batch":
        batch = state["batch"]
        slots = [batch.add(s, P["dt"], P["steps"]) for s, P in zip(solvers, problems)]
        batch.step(case["steps"])
        batch.synchronize()
        for slot in slots:
            batch.remove(slot)
        for s, out in zip(solvers, outs):
            s.handle.get_state(0, out)
        return np.concatenate(outs)
    s, P = solvers[0], problems[0]
    if case["kind"] == "adaptive":
        time, s.dtEstimate = 0.0, P["dt"]
        for _ in range(P["steps"]):
            time = s.computeOneTimeStepAdaptive(time, REL_ERROR, 4 * P["dt"])
        return {"u": s.handle.get_state(0, outs[0]), "time": time}
    s.computeTimeSteps(0.0, P["dt"], P["steps"])
    return s.handle.get_state(0, outs[0])


def work(case):
    """The state crosses the host link once each way; a step reads and writes the solution and
    writes every stage vector (they stay readable).  Operations: the element's 1D derivatives
    and lifts on quads and hexes, its dense derivatives and upwind or two-sided face products
    on simplices, its stored matrices in the linear form."""
    total = {"bytes": 0.0, "flops": 0.0}
    for P in _problems(case):
        p, dim, V = P["order"], P["dim"], P["vars"]
        nb = _basis_size(dim, P["triangular"], p)
        elements = math.prod(P["cells"]) * ((2 if dim == 2 else 5) if P["triangular"] else 1)
        stages = len(TABLEAUX[case.get("tableau", "RK4_4")][0])
        faces = dim + 1 if P["triangular"] else 2 * dim
        if case["kind"] == "linear":
            per = 2.0 * (V * nb) ** 2 * (1 + (faces if V > 1 else (faces + 1) // 2))
        elif not P["triangular"]:
            per = 2.0 * nb * dim * (p + 3)
        elif V == 1:
            per = 2.0 * nb * nb * (dim + faces)
        else:
            per = 2.0 * nb * nb * (2 * dim + 4 * faces)
        k_bytes = 8 if case["precision"] == "fp64" else 4
        dof = elements * V * nb
        total["bytes"] += dof * (16.0 + P["steps"] * (16.0 + k_bytes * stages))
        total["flops"] += P["steps"] * stages * elements * per
    return total


# ---- the exact results -------------------------------------------------------------------------
TABLEAUX = {  # stage coefficients, weights, error coefficients, order of the step-size control
    "RK4_4": ([[], [1 / 2], [0, 1 / 2], [0, 0, 1]], [1 / 6, 1 / 3, 1 / 3, 1 / 6], None, 4),
    "RK3TVD": ([[], [1], [1 / 4, 1 / 4]], [1 / 6, 1 / 6, 2 / 3], None, 3),
    "DormandPrince": ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
                       [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
                       [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
                       [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
                      [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0],
                      [35 / 384 - 5179 / 57600, 0, 500 / 1113 - 7571 / 16695, 125 / 192 - 393 / 640,
                       -2187 / 6784 + 92097 / 339200, 11 / 84 - 187 / 2100, -1 / 40], 5),
}


def exact(case, seed):
    tableau = TABLEAUX[case.get("tableau", "RK4_4")]
    outs = []
    for i, P in enumerate(_problems(case)):
        u, rhs = _initial(P, seed + 7919 * i), _Operator(P)
        if case["kind"] == "adaptive":
            u, time = _adaptive(rhs, u, P, tableau)
            return {"u": u.reshape(-1).cpu().numpy(), "time": time}
        for _ in range(P["steps"]):
            u, _ = _step(rhs, u, P["dt"], tableau)
        outs.append(u.reshape(-1).cpu().numpy())
    return np.concatenate(outs)


def _step(rhs, u, dt, tableau):
    ks = []
    for row in tableau[0]:
        w = u
        for a, k in zip(row, ks):
            if a:
                w = w + (dt * a) * k
        ks.append(rhs(w))
    new = u
    for b, k in zip(tableau[1], ks):
        if b:
            new = new + (dt * b) * k
    return new, ks


def _adaptive(rhs, u, P, tableau):
    """Steps whose embedded error is accepted against REL_ERROR times the sum of the elements' norms."""
    time, estimate = 0.0, P["dt"]
    for _ in range(P["steps"]):
        dt = min(estimate, 4 * P["dt"])
        while True:
            new, ks = _step(rhs, u, dt, tableau)
            deviation = sum(dt * e * k for e, k in zip(tableau[2], ks) if e)
            error, norm = float(deviation.norm()), float(new.flatten(1).norm(dim=1).sum())
            ratio = REL_ERROR / error * norm
            if REL_ERROR * norm >= error:
                break
            dt = 0.8 * dt * ratio ** (1 / tableau[3])
        u, time, estimate = new, time + dt, 0.9 * dt * ratio ** (1 / tableau[3])
    return u, time


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tensor(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_device())


def _corners(dim):
    return np.array([[(k >> i) & 1 for i in range(dim)] for k in range(1 << dim)])


def _lattice(P):
    """Lattice coordinates of every element's vertices, [element][vertex][dim], in the mesh's
    order: cells with x fastest; simplex meshes cut a square in 2 triangles or a cube in 5
    tetrahedra by a pattern that turns a quarter with every cell."""
    n, dim = P["cells"], P["dim"]
    cell = np.arange(math.prod(n))
    index = []
    for m in n:
        index.append(cell % m)
        cell = cell // m
    index = np.stack(index, axis=1)
    if not P["triangular"]:
        return index[:, None, :] + _corners(dim)[None]
    pattern = [[0, 1, 2], [1, 3, 2]] if dim == 2 else [[1, 2, 4, 7], [0, 1, 2, 4], [1, 3, 2, 7], [1, 4, 5, 7], [2, 6, 4, 7]]
    turn = np.array([2, 0, 3, 1, 6, 4, 7, 5])
    turned = [np.array(pattern)]
    for _ in range(3):
        turned.append(turn[turned[-1]])
    turns, per = index[:, 0].copy(), n[0]
    for i in range(1, dim):
        per += n[i - 1] % 2 + 1
        turns += index[:, i] * per
        per *= n[i]
    vertices = np.stack(turned)[turns % 4]  # [cell][simplex][vertex]
    return (index[:, None, None, :] + _corners(dim)[vertices]).reshape(-1, dim + 1, dim)


def _lobatto(k, x):
    c = legendre.legder(np.eye(k + 2)[k + 1])
    return -4 * math.sqrt((2 * k + 3) / 2) / ((k + 1) * (k + 2)) * legendre.legval(x, c)


def _line(k, x):
    """The 1D functions: two vertex functions, then (1 - x^2) L_k / 4."""
    return (1 - x) / 2 if k == 0 else (1 + x) / 2 if k == 1 else (1 - x * x) * _lobatto(k - 2, x) / 4


def _hypercube_functions(p, X):
    """The H1 functions of squares and cubes; edge and face functions run from the lower to the
    higher vertex of their edge, so a product of 1D functions is all there is."""
    dim = X.shape[1]
    f = lambda *ks: math.prod(_line(k, X[:, i]) for i, k in enumerate(ks))  # noqa: E731
    out = [f(*[(v >> i) & 1 for i in range(dim)]) for v in range(1 << dim)]
    if dim == 2:
        for i in range(2, p + 1):
            out += [f(i, 0), f(i, 1), f(0, i), f(1, i)] + [f(i, j) for j in range(2, p + 1)]
        return out
    def faces(i, j):  # noqa: E306
        return [f(i, j, 0), f(i, 0, j), f(0, i, j), f(1, i, j), f(i, 1, j), f(i, j, 1)]
    for j in range(2, p + 1):
        out += [f(j, b, c) for c in (0, 1) for b in (0, 1)] + [f(a, j, c) for c in (0, 1) for a in (0, 1)]
        out += [f(a, b, j) for b in (0, 1) for a in (0, 1)]
        out += faces(j, j) + [f(j, j, j)]
        for i in range(2, j):
            out += faces(i, j) + faces(j, i)
            out += [f(i, i, j), f(i, j, i), f(j, i, i), f(j, j, i), f(j, i, j), f(i, j, j)]
            for k in range(2, i):
                out += [f(i, j, k), f(i, k, j), f(j, i, k), f(j, k, i), f(k, i, j), f(k, j, i)]
    return out


TET_EDGES = [(0, 1), (0, 2), (0, 3), (2, 3), (1, 3), (1, 2)]
TET_FACES = [(0, 3, 2), (0, 1, 3), (0, 2, 1), (1, 2, 3)]


def _simplex_functions(p, X):
    dim = X.shape[1]
    l = [1 - X.sum(axis=1)] + [X[:, i] for i in range(dim)]  # noqa: E741
    def f(vs, ks):  # noqa: E306
        return math.prod(l[v] for v in vs) * math.prod(_lobatto(k, l[a] - l[b]) for k, a, b in zip(ks, vs, vs[1:]))
    out = list(l)
    for j in range(p - 1):
        if dim == 2:
            out += [f((a, b), (j,)) for a, b in ((0, 1), (0, 2), (1, 2))]
            if j + 3 <= p:
                out += [f((0, 1, 2), (j - k, k)) for k in range(j + 1)]
        else:
            out += [f(e, (j,)) for e in TET_EDGES]
            out += [f(v, (j - k - 1, k)) for v in TET_FACES for k in range(j)]
            out += [f((0, 1, 2, 3), (i, j - i - k - 2, k)) for i in range(j - 1) for k in range(j - 1 - i)]
    return out


def _basis(P, X, gradients=False):
    """Values [point][function], or gradients [dim][point][function] by complex steps."""
    functions = _simplex_functions if P["triangular"] else _hypercube_functions
    if not gradients:
        return np.stack(functions(P["order"], X), axis=1)
    out = []
    for c in range(X.shape[1]):
        Z = X.astype(complex)
        Z[:, c] += 1e-30j
        out.append(np.stack(functions(P["order"], Z), axis=1).imag / 1e-30)
    return np.stack(out)


def _rule(dim, triangular, m):
    """Points in [0, 1]^dim or the unit simplex and weights that sum to 1."""
    x, w = legendre.leggauss(m)
    x, w = (x + 1) / 2, w / 2
    X = np.stack([g.reshape(-1) for g in np.meshgrid(*[x] * dim, indexing="ij")], axis=1) if dim else np.zeros((1, 0))
    W = math.prod(np.meshgrid(*[w] * dim, indexing="ij")).reshape(-1) if dim else np.ones(1)
    if triangular and dim > 1:  # collapse the cube onto the simplex
        Y = X.copy()
        for i in range(1, dim):
            Y[:, i] = X[:, i] * (1 - Y[:, :i].sum(axis=1))
            W = W * (1 - Y[:, :i].sum(axis=1))
        X, W = Y, W / W.sum()
    return X, W


def _reference(P, m):
    """Element rule: points in the reference element, weights times its volume."""
    X, W = _rule(P["dim"], P["triangular"], m)
    if P["triangular"]:
        return X, W / math.factorial(P["dim"])
    return 2 * X - 1, W * 2 ** P["dim"]


def _vertices(P):
    if P["triangular"]:
        return np.concatenate([np.zeros((1, P["dim"])), np.eye(P["dim"])])
    return 2.0 * _corners(P["dim"]) - 1


def _jacobians(P, x):
    if P["triangular"]:
        return torch.stack([x[:, i + 1] - x[:, 0] for i in range(P["dim"])], dim=2)
    return torch.stack([(x[:, 1 << i] - x[:, 0]) / 2 for i in range(P["dim"])], dim=2)


def _initial(P, seed):
    """L2 projection of three seeded Fourier modes (the wave: pressure, velocity at rest), [E][vars][nb]."""
    rng = np.random.default_rng(seed)
    dim = P["dim"]
    k = _tensor(rng.integers(1, 4, size=(3, dim)) * rng.choice([-1.0, 1.0], size=(3, dim)))
    amplitude, phase = _tensor(rng.uniform(0.5, 1.0, 3)), _tensor(rng.uniform(0, 2 * math.pi, 3))
    X, W = _reference(P, P["order"] + 2)
    phi = _basis(P, X)
    project = _tensor(np.linalg.solve(np.einsum("q,qi,qj->ij", W, phi, phi), W * phi.T))
    x = _tensor(_lattice(P).astype(float)) / _tensor(np.array(P["cells"], dtype=float))
    J, centre = _jacobians(P, x), _tensor(_vertices(P)[0])
    u = torch.zeros(len(x), P["vars"], phi.shape[1], dtype=torch.float64, device=x.device)
    for e in range(0, len(x), 1 << 16):
        at = x[e:e + (1 << 16), None, 0] + torch.einsum("ecd,qd->eqc", J[e:e + (1 << 16)], _tensor(X) - centre)
        value = (amplitude * torch.sin(2 * math.pi * at @ k.T + phase)).sum(dim=2)
        u[e:e + (1 << 16), 0] = value @ project.T
    return u


class _Operator:
    """u -> M^{-1} (volume and face integrals), by quadrature on every element."""

    def __init__(self, P):
        self.P, dim, tri = P, P["dim"], P["triangular"]
        lattice = _lattice(P)
        n = np.array(P["cells"])
        x = _tensor(lattice.astype(float)) / _tensor(n.astype(float))
        J = _jacobians(P, x)
        self.Jinv, self.det = torch.linalg.inv(J), torch.linalg.det(J).abs()
        X, W = _reference(P, P["order"] + 2)
        phi, grad = _basis(P, X), _basis(P, X, True)
        self.minv = _tensor(np.linalg.inv(np.einsum("q,qi,qj->ij", W, phi, phi)))
        self.weak = _tensor(np.einsum("q,cqi,qj->cij", W, grad, phi))
        self.strong = _tensor(np.einsum("q,qi,cqj->cij", W, phi, grad))
        # faces: local vertex lists; a simplex face's points follow the order of its global node
        # numbers, so that both elements of a face have the same points
        if tri:
            faces = [[v for v in range(dim + 1) if v != f] for f in range(dim + 1)]
        else:
            faces = [[v for v in range(1 << dim) if (v >> a) & 1 == s] for a in range(dim) for s in (0, 1)]
        node = ((lattice % n) * np.concatenate([[1], np.cumprod(n)[:-1]])).sum(axis=2)
        F, W = _rule(dim - 1, tri, P["order"] + 2)
        if tri:
            shape = np.concatenate([1 - F.sum(axis=1, keepdims=True), F], axis=1)
        else:
            shape = math.prod([np.where(_corners(dim - 1)[None, :, i], F[:, None, i], 1 - F[:, None, i])
                               for i in range(dim - 1)]) if dim > 1 else np.ones((1, 1))
        E, nf = len(lattice), len(faces)
        ids = node[:, np.array(faces)]  # [E][face][vertex]
        order = np.argsort(ids, axis=2) if tri else np.broadcast_to(np.arange(ids.shape[2]), ids.shape)
        code = (order * ids.shape[2] ** np.arange(ids.shape[2])).sum(axis=2) + 10 ** 6 * np.arange(nf)
        kinds, which = np.unique(code, return_inverse=True)
        which = which.reshape(E, nf)
        tables = []
        for kind in range(len(kinds)):
            e, f = np.argwhere(which == kind)[0]
            tables.append(_basis(P, shape @ _vertices(P)[np.array(faces[f])[order[e, f]]]))
        tables = _tensor(np.stack(tables))
        self.trace = tables[_tensor(which)] if tri else tables[_tensor(which[:1])]  # [E or 1][face][point][nb]
        self.lift = self.trace * _tensor(W)[:, None]
        # neighbours: the two faces with the same nodes
        key = np.sort(ids, axis=2)[:, :, :3].astype(np.int64)
        key = (key * (int(n.prod()) + 1) ** np.arange(key.shape[2])).sum(axis=2).reshape(-1)
        by = np.argsort(key, kind="stable")
        other = np.empty(E * nf, dtype=np.int64)
        other[by[0::2]], other[by[1::2]] = by[1::2], by[0::2]
        self.other = _tensor(other)
        # outward normals and areas
        v = x[:, torch.as_tensor(np.array(faces), device=x.device)]  # [E][face][vertex][dim]
        if dim == 2:
            t = v[:, :, 1] - v[:, :, 0]
            normal = torch.stack([t[..., 1], -t[..., 0]], dim=2)
        else:
            normal = torch.linalg.cross(v[:, :, 1] - v[:, :, 0], v[:, :, 2] - v[:, :, 0]) * (0.5 if tri else 1.0)
        out = ((v.mean(dim=2) - x.mean(dim=1, keepdim=True)) * normal).sum(dim=2, keepdim=True)
        normal = normal * torch.sign(out)
        self.area = normal.norm(dim=2)
        self.normal = normal / self.area[..., None]

    def __call__(self, w):
        P, E, V = self.P, len(w), self.P["vars"]
        nb, nf, nq = w.shape[2], self.trace.shape[1], self.trace.shape[2]
        T = (w @ self.trace.reshape(-1, nf * nq, nb).transpose(1, 2)).reshape(E, V, nf, nq).permute(0, 2, 3, 1)
        T = T.contiguous()
        N = T.reshape(E * nf, nq, V)[self.other].reshape(E, nf, nq, V)
        if V == 1:
            a = _tensor(np.array(P["a"]))
            volume = torch.einsum("ec,cij,ej->ei", self.Jinv @ a, self.weak, w[:, 0])[:, None]
            an = self.normal @ a
            upwind = torch.where((an > 1e-12)[..., None], T[..., 0], torch.where((an < -1e-12)[..., None], N[..., 0],
                                                                                0.5 * (T[..., 0] + N[..., 0])))
            flux = -(an[..., None] * upwind)[..., None]
        else:
            D = torch.einsum("ecd,cij,evj->edvi", self.Jinv, self.strong, w)  # physical derivatives
            volume = torch.cat([sum(D[:, d, d + 1] for d in range(P["dim"]))[:, None], D[:, :, 0]], dim=1)
            jump = T - N
            jn = (jump[..., 1:] * self.normal[:, :, None, :]).sum(dim=3)
            penalty = 1.0 if P["physics"] == "wave_upwind" else 0.0
            flux = torch.cat([(-0.5 * jn - 0.5 * penalty * jump[..., 0])[..., None],
                              -0.5 * self.normal[:, :, None, :] * (jump[..., :1] + penalty * jn[..., None])], dim=3)
        flux = (flux * (self.area / self.det[:, None])[:, :, None, None]).reshape(E, nf * nq, V)
        faces = flux.transpose(1, 2) @ self.lift.reshape(-1, nf * nq, nb)
        return (volume + faces) @ self.minv
