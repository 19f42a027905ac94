"""The work that a user of the framework has it do, as cases that can be timed and compared.

A case is one pass through public entry points of ``mts_b200``:

* ``run``      a problem resident on the GPU is run for a number of steps from
               the caller's field in pinned host memory, and the result is read
               back (``Solver.advance_host_ptr``, the drop-in's call), with the
               error norms at the end as the reference's time loops print them;
* ``step``     the same for a single step and without norms: the drop-in's
               ``Solve_2nd`` with the field in host memory;
* ``batch``    many small problems advance together (``batch_advance_steps``)
               and every field is read back;
* ``request``  a problem from its description to its field: setup, upload,
               initial field, steps, norms, field (what the server does per
               request);
* ``setup``    the tags, crossings and MIB weights of a problem on the device.

Sizes, surfaces, coefficients and step counts are those of the repository's
tests, benchmark and request mix.
"""
from __future__ import annotations

import math
import os
import sys
from dataclasses import replace

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "matched-time-splitting-3d_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mts_b200 as M  # noqa: E402
from mts_b200 import workloads  # noqa: E402

TORUS = {"surface": "torus", "s0": 0.5, "s1": 0.2}
SPHERE = {"surface": "ellipsoid", "s0": 1.0, "s1": 1.0, "s2": 1.0, "s3": 0.49, "s4": 0.0, "s5": 0.0, "s6": 0.0}
ELLIPSOID = {"surface": "ellipsoid", "s0": 0.7001, "s1": 0.4999, "s2": 0.4001, "s3": 1.0, "s4": 0.0, "s5": 0.0,
             "s6": 0.0}
OFFSET = {"surface": "ellipsoid", "s0": 0.6123, "s1": 0.4517, "s2": 0.3739, "s3": 1.0, "s4": 0.0713, "s5": -0.1127,
          "s6": 0.0391}


def _case(name, do, n, surface, bi, bo, method, mib, steps, precision="plain", dt=None):
    h = min(2.0 / (k - 1) for k in n)
    c = {"do": do, "nx": n[0], "ny": n[1], "nz": n[2], "beta_in": bi, "beta_out": bo, "method": method, "mib": mib,
         "dt": dt if dt is not None else h, "steps": steps, "precision": precision, **surface}
    return {"name": name, **c} if name else c


def listed():
    return [
        # The drop-in on the reference's shipped 33^3 sphere: one Solve_2nd
        # per call, the field in host memory.  Latency and launches.
        _case("step_33_adi", "step", (33, 33, 33), SPHERE, 1.0, 10.0, "adi", 1, 1, dt=1.0 / 32),
        # A request of the served mix on an anisotropic grid, from its
        # description to its field.
        _case("request_33x49x25_lodie", "request", (33, 49, 25), OFFSET, 1.0, 37.5, "lod-ie", 2, 60),
        # The drop-in configuration's grid, dt = h, t = 0 to 1.
        _case("run_65_adi", "run", (65, 65, 65), TORUS, 1.0, 1000.0, "adi", 2, 32),
        # The next refinement, Crank-Nicolson splitting.
        _case("run_129_lodcn", "run", (129, 129, 129), ELLIPSOID, 1.0, 10.0, "lod-cn", 1, 64),
        # Trapezoidal splitting on a ragged grid.
        _case("run_113x97x141_ts", "run", (113, 97, 141), OFFSET, 1.0, 0.05, "ts", 2, 48),
        # The benchmark's grid in the bit-exact form, t = 0 to 1.
        _case("run_257_adi", "run", (257, 257, 257), TORUS, 1.0, 1000.0, "adi", 2, 128),
        # The benchmark's headline: the fast FP64 form, t = 0 to 1/2.
        _case("run_257_fast", "run", (257, 257, 257), TORUS, 1.0, 1000.0, "adi", 2, 64, "fast"),
        # The fast form on an ordinary ragged grid of even and odd lines.
        _case("run_131x118x150_fast", "run", (131, 118, 150), OFFSET, 1.0, 250.0, "adi", 2, 64, "fast"),
        # The mixed form on the benchmark's grid.
        _case("run_257_mixed", "run", (257, 257, 257), ELLIPSOID, 1.0, 1000.0, "adi", 1, 128, "mixed"),
        # The largest grid of the benchmark's precision sweep, mixed form.
        _case("run_385_mixed", "run", (385, 385, 385), TORUS, 1.0, 1e-3, "adi", 2, 48, "mixed"),
        # The batched family: 192 problems of 17 to 65 nodes per axis, all
        # four methods, 50 steps.
        {"name": "batch_192", "do": "batch", "count": 192, "family": 0, "steps": 50, "precision": "plain"},
        # The device setup of the benchmark's problem.
        _case("setup_257_torus", "setup", (257, 257, 257), TORUS, 1.0, 1000.0, "adi", 2, 0),
    ]


_LARGEST = 48 * 385**3  # node-steps of the largest listed case, the most a drawn one may take


def draw(rng):
    while True:
        c = _draw(rng)
        if c["do"] == "batch":
            return c
        try:
            counts = M.setup_host(_spec(c))[2]
        except M.MtsError:
            continue  # the interface passes through a grid node: refused by every setup
        if counts["singular_warnings"] == 0:  # (such problems amplify any rounding a thousandfold)
            return c


def _draw(rng):
    kind = rng.choices(("run", "step", "batch", "request", "setup"), (10, 2, 2, 2, 2))[0]
    if kind == "batch":
        return {"do": "batch", "count": int(math.exp(rng.uniform(math.log(16), math.log(192)))),
                "family": rng.randrange(1, 1000), "steps": rng.randrange(20, 80),
                "precision": rng.choice(("plain", "plain", "mixed"))}
    top = {"run": 340.0, "step": 140.0, "request": 129.0, "setup": 257.0}[kind]
    base = math.exp(rng.uniform(math.log(17.0), math.log(top)))
    n = tuple(max(17, min(385, round(base * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(3))
    method = rng.choice(("adi", "adi", "adi", "lod-ie", "lod-cn", "ts"))
    precision = rng.choice(("plain", "fast", "mixed")) if method == "adi" and kind in ("run", "step") else "plain"
    surface = dict(rng.choice((TORUS, SPHERE, ELLIPSOID, OFFSET, OFFSET)))
    if surface == OFFSET:
        for k, lo, hi in (("s0", 0.4, 0.7), ("s1", 0.35, 0.6), ("s2", 0.35, 0.6), ("s4", -0.15, 0.15),
                          ("s5", -0.15, 0.15), ("s6", -0.15, 0.15)):
            surface[k] = round(rng.uniform(lo, hi), 6)
    nodes = n[0] * n[1] * n[2]
    # (a high-contrast torus amplifies any rounding step by step: the forms
    # that round differently are drawn with runs short enough to compare)
    most = max(4, min({"plain": 128, "fast": 64, "mixed": 32}[precision], _LARGEST // 2 // nodes))
    steps = 0 if kind == "setup" else 1 if kind == "step" else rng.randrange(min(16, most), most + 1)
    bo = round(10.0 ** rng.uniform(-2.0, 3.0), 6)
    return _case(None, kind, n, surface, 1.0, bo, method, rng.choice((1, 2)), steps, precision)


def _spec(c):
    params = tuple(c[k] for k in ("s0", "s1", "s2", "s3", "s4", "s5", "s6") if k in c)
    return M.Spec(n=(c["nx"], c["ny"], c["nz"]), surface=c["surface"], surface_params=params, beta_in=c["beta_in"],
                  beta_out=c["beta_out"], method=c["method"], mib=c["mib"], dt=c["dt"],
                  setup="device" if c["do"] == "request" else "host")


def _nodes(c):
    return c["nx"] * c["ny"] * c["nz"]


def _family(c):
    return workloads.batched_problems(c["count"], c["family"])


def _t0(seed):
    return 0.25 * np.random.default_rng(seed).random()


def _start_field(c, tags, seed):
    """The exact solution at the start time by the nodes' side, and a smooth
    perturbation that vanishes on the faces; [z, y, x] like the solver's."""
    rng = np.random.default_rng(seed + 1)
    ax = [np.linspace(-1.0, 1.0, k) for k in (c["nx"], c["ny"], c["nz"])]
    s, co = [np.sin(2.0 * a) for a in ax], [np.cos(2.0 * a) for a in ax]
    x, y, z = ax
    out = (z * z)[:, None, None] + ((y * y)[:, None] + (x * x)[None, :])[None]
    u = np.multiply(s[2][:, None, None], (co[1][:, None] * s[0][None, :])[None])
    np.copyto(u, out, where=tags.reshape(u.shape) > 0)
    u *= math.exp(-_t0(seed))
    m = rng.integers(1, 5, 3)
    w = [np.sin(m[d] * np.pi * (ax[d] + 1.0) / 2.0) for d in range(3)]
    np.multiply((w[2] * (0.1 * rng.random()))[:, None, None], (w[1][:, None] * w[0][None, :])[None], out=out)
    u += out
    return u


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available())


class _Buffers:
    """A batch and its host buffer."""

    def __init__(self, solvers, out, where):
        self.solvers, self.out, self.where = solvers, out, where


def prepare(case, seed):
    do = case["do"]
    if do in ("run", "step"):
        s = M.Solver(_spec(case))
        if case["precision"] != "plain":
            s.set_precision(case["precision"])
        u_in, u_out = _pinned(_nodes(case)), _pinned(_nodes(case))
        u_in.numpy()[:] = _start_field(case, s.tags(), seed).reshape(-1)
        return {"case": case, "solver": s, "t0": _t0(seed), "in": u_in, "out": u_out}
    if do == "batch":
        solvers = [M.Solver(p) for p in _family(case)]
        for s in solvers:
            if case["precision"] == "mixed" and s.spec.method == "adi":
                s.set_precision("mixed")
        where = np.concatenate([[0], np.cumsum([s.spec.nodes for s in solvers])])
        return {"case": case, "t0": _t0(seed), "batch": _Buffers(solvers, _pinned(int(where[-1])), where)}
    if do == "setup":
        # the same geometry with other material: the weights change, the crossings do not
        r = np.random.default_rng(seed).random(2)
        spec = _spec(case)
        return {"case": case, "spec": replace(spec, beta_in=spec.beta_in * (1.0 + 0.2 * float(r[0])),
                                              beta_out=spec.beta_out * (1.0 + 0.2 * float(r[1])))}
    return {"case": case, "spec": _spec(case), "t0": _t0(seed)}


def run(state):
    c = state["case"]
    if c["do"] in ("run", "step"):
        s = state["solver"]
        s.time = state["t0"]
        s.advance_host_ptr(state["in"].data_ptr(), state["out"].data_ptr(), c["steps"])
        if c["do"] == "step":
            return state["out"]
        linf, l2, _ = s.norms()
        return {"u": state["out"], "linf": linf, "l2": l2}
    if c["do"] == "batch":
        b = state["batch"]
        for s in b.solvers:
            s.time = state["t0"]
            s.initialize()
        M.batch_advance_steps(b.solvers, [c["steps"]] * len(b.solvers))
        get, base = M.load().mts_get_solution, b.out.data_ptr()
        for s, o in zip(b.solvers, b.where):
            if get(s.handle, base + 8 * int(o)):
                raise RuntimeError("mts_get_solution")
        return b.out
    if c["do"] == "request":
        with M.Solver(state["spec"]) as s:
            s.time = state["t0"]
            s.initialize()
            s.advance(c["steps"])
            linf, l2, _ = s.norms()
            return {"u": s.solution(), "linf": linf, "l2": l2}
    tags, cr, counts = M.setup_device(state["spec"])
    return {"tags": tags, "counts": [counts["corner_pairs"], counts["singular_warnings"]],
            "where": np.stack([cr[k] for k in ("dir", "indx1", "indx2", "id", "left_loc", "nwei")]),
            "values": np.concatenate([cr[k].reshape(cr.size, -1)
                                      for k in ("coord", "gamma", "normal", "p", "weil", "weir")], axis=1)}


def work(case):
    """Per step of a node: the field read and written and the tag read, and
    about 60 operations (the stencils, three line solves, the source).  A
    call's host buffers cross the bus once each way.  The setup writes a tag
    per node and evaluates the level set (about 10 operations)."""
    if case["do"] == "setup":
        return {"bytes": _nodes(case), "flops": 10 * _nodes(case)}
    n = sum(p.nodes for p in _family(case)) if case["do"] == "batch" else _nodes(case)
    return {"bytes": n * (17 * case["steps"] + 16), "flops": 60 * n * case["steps"]}


def tolerance(case):
    if case["precision"] == "plain":
        return "exact"  # the bit-exact form, and the setup
    # the largest differences from the bit-exact form over tori and ellipsoids
    # of 97 to 385 nodes per axis, beta ratios to 1000, at the step counts
    # listed and drawn, times four
    if case["precision"] == "fast":
        return {"rel": 6e-10, "max": 4e-8}  # FP64 in another order: 1.6e-10, 8.4e-9
    return {"rel": 6e-5, "max": 5e-3}  # FP32 increments: 1.4e-5, 1.3e-3


# ---------------------------------------------------------------------------
# The same steps in numpy, from the crossing list the solver is given.

_EXACT_NODE_STEPS = 10_000_000  # about 15 s


class _Rows:
    """The MIB rows of one direction: two rows per single crossing, three per
    corner pair.  Row k of block b is node ``node[k]``; its three-point sum
    with fictitious points is sum_i coef[k, i] u[first[k] + i s] plus
    sum_i jc[k, i] (ju, jb)[c0 or c1]."""

    def __init__(self, c, tags, cr, d, vd):
        nx, ny = c["nx"], c["ny"]
        self.s = (1, nx, nx * ny)[d]
        self.groups = []
        cr = cr[cr["dir"] == d]
        at = np.flatnonzero(cr["dir"] == d)
        single = np.flatnonzero(cr["id"] > 0)
        left = np.flatnonzero(cr["id"] < 0)[0::2]
        for kind, c0 in ((2, single), (3, left)):
            if not c0.size:
                continue
            c1 = c0 + (kind == 3)
            i1, i2, L = (cr[k][c0].astype(np.int64) for k in ("indx1", "indx2", "left_loc"))
            base = (nx * (i1 + ny * i2), i1 + nx * ny * i2, i1 + nx * i2)[d]
            node = base[:, None] + (L[:, None] + np.arange(kind)) * self.s
            side = (tags[node] > 0).astype(int)
            v0, v1 = vd[side][:, :, 0], vd[side][:, :, 1]
            w = [cr["weil"][c0], cr["weir"][c0], cr["weil"][c1], cr["weir"][c1]]
            W = kind + 2  # columns L-1 .. L+kind
            coef = np.zeros((c0.size, kind, W))
            jc = np.zeros((c0.size, kind, 2 * (kind - 1)))
            for r in range(kind):
                for wt, low in ((w[1] if r == 0 else w[3], False), (w[0] if r <= 1 else w[2], True)):
                    if low and r == 0:
                        coef[:, r, 0] += v0[:, r]
                        continue
                    if not low and r == kind - 1:
                        coef[:, r, W - 1] += v0[:, r]
                        continue
                    coef[:, r, :] += v0[:, r, None] * wt[:, :W]
                    jc[:, r, :] += v0[:, r, None] * wt[:, W:W + 2 * (kind - 1)]
                coef[:, r, r + 1] += v1[:, r]
            self.groups.append({"kind": kind, "node": node, "first": node[:, 0] - self.s, "coef": coef, "jc": jc,
                                "c": np.stack([at[c0], at[c1]], 1)[:, :kind - 1], "L": L, "i1": i1, "i2": i2})

    def jumps(self, J):
        return [np.einsum("brj,bj->br", g["jc"], J[g["c"]].reshape(len(g["c"]), -1)) for g in self.groups]


def _exact_steps(spec, c, tags, cr, u, t0):
    n = spec.n
    shape = (n[2], n[1], n[0])
    h = [2.0 / (k - 1.0) for k in n]
    ax = [-1.0 + np.arange(k) * hd for k, hd in zip(n, h)]
    beta = np.array([spec.beta_in, spec.beta_out])
    out = (tags > 0).reshape(shape)
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    S = np.sin(2 * X) * np.cos(2 * Y) * np.sin(2 * Z)
    R2 = X * X + Y * Y + Z * Z
    dt = spec.dt
    half = spec.method in ("lod-cn", "ts")
    cdt = 0.5 * dt if half else dt
    F0 = np.where(out, -R2 - 6.0 * spec.beta_out, (12.0 * spec.beta_in - 1.0) * S)  # the source / e^{-t}
    face = np.ones(shape, bool)
    face[1:-1, 1:-1, 1:-1] = False
    nb = beta[out.astype(int)]

    # jump data / e^{-t}
    cx = cr["coord"]
    s, co = np.sin(2 * cx), np.cos(2 * cx)
    bu = np.stack([spec.beta_out * 2 * cx[:, 0] - spec.beta_in * 2 * co[:, 0] * co[:, 1] * s[:, 2],
                   spec.beta_out * 2 * cx[:, 1] + spec.beta_in * 2 * s[:, 0] * s[:, 1] * s[:, 2],
                   spec.beta_out * 2 * cx[:, 2] - spec.beta_in * 2 * s[:, 0] * co[:, 1] * co[:, 2]], 1)
    p = cr["p"].reshape(-1, 3, 3)
    pinv = np.linalg.inv(p)[np.arange(cr.size), cr["dir"], 0] if cr.size else np.zeros(0)
    J0 = np.stack([(cx * cx).sum(1) - s[:, 0] * co[:, 1] * s[:, 2], pinv * (p[:, 0] * bu).sum(1)], 1)

    rows, tri = [], []
    for d in range(3):
        vd = np.array([[b / h[d] ** 2, -2 * b / h[d] ** 2, b / h[d] ** 2] for b in beta])
        sel = np.flatnonzero(cr["dir"] == d)
        r = _Rows(c, tags, cr[sel], d, vd)
        r.sel = sel
        rows.append(r)
        # tridiagonal rows, node-shaped; MIB rows after elimination of the
        # columns outside the three diagonals
        lam = cdt * nb / h[d] ** 2
        a, b, cc = -lam, 1 + 2 * lam, -lam.copy()
        ends = [slice(None)] * 3
        for e in (0, -1):
            ends[2 - d] = e
            a[tuple(ends)], b[tuple(ends)], cc[tuple(ends)] = 0.0, 1.0, 0.0
        for g in r.groups:
            k = g["kind"]
            m = -cdt * g["coef"]
            for q in range(k):
                m[:, q, q + 1] += 1.0
            ops = [(1, 0, 0), (0, 1, 3)] if k == 2 else [(1, 0, 0), (2, 0, 0), (0, 2, 4), (1, 2, 4), (2, 1, 1), (0, 1, 3)]
            g["ops"] = []
            for to, by, col in ops:
                rate = m[:, to, col] / m[:, by, col]
                m[:, to] -= rate[:, None] * m[:, by]
                g["ops"].append((to, by, rate))
            for q in range(k):
                nd = g["node"][:, q]
                a.reshape(-1)[nd], b.reshape(-1)[nd], cc.reshape(-1)[nd] = m[:, q, q], m[:, q, q + 1], m[:, q, q + 2]
        A, B, C = (np.ascontiguousarray(np.moveaxis(v, 2 - d, 0)) for v in (a, b, cc))
        bet, gam = np.empty_like(A), np.zeros_like(A)
        bet[0] = B[0]
        for j in range(1, n[d]):
            gam[j] = C[j - 1] / bet[j - 1]
            bet[j] = B[j] - A[j] * gam[j]
        tri.append((A, bet, gam))

    def explicit(d, v, J):
        """beta v_dd by three-point sums, MIB rows with their fictitious points; J None: without jumps."""
        f = v.reshape(-1)
        w = np.zeros(shape)
        lo, mid, hi = ([slice(1, -1)] * 3 for _ in range(3))
        lo[2 - d], hi[2 - d] = slice(0, -2), slice(2, None)
        w[1:-1, 1:-1, 1:-1] = (v[tuple(lo)] - 2 * v[tuple(mid)] + v[tuple(hi)]) * nb[1:-1, 1:-1, 1:-1] / h[d] ** 2
        r = rows[d]
        js = r.jumps(J[r.sel]) if J is not None else [0.0] * len(r.groups)
        for g, j in zip(r.groups, js):
            k = g["kind"]
            cols = g["first"][:, None] + np.arange(k + 2) * r.s
            w.reshape(-1)[g["node"]] = np.einsum("brw,bw->br", g["coef"], f[cols]) + j
        return w

    def solve(d, v, J, ends, keep):
        """(1 - cdt beta D_dd) along every interior line; J: jump terms on the
        rows' right-hand sides; ends: values at the lines' ends and, unless
        keep, on the lines of the faces."""
        r = rows[d]
        rhs = v.copy()
        e = [slice(1, -1)] * 3
        for at in (0, -1):
            e[2 - d] = at
            rhs[tuple(e)] = ends[tuple(e)]
        js = r.jumps(J[r.sel]) if J is not None else [0.0] * len(r.groups)
        f = rhs.reshape(-1)
        for g, j in zip(r.groups, js):
            q = f[g["node"]] + cdt * j
            for to, by, rate in g["ops"]:
                q[:, to] -= rate * q[:, by]
            f[g["node"]] = q
        A, bet, gam = tri[d]
        y = np.moveaxis(rhs, 2 - d, 0).copy()
        y[0] /= bet[0]
        for j in range(1, n[d]):
            y[j] = (y[j] - A[j] * y[j - 1]) / bet[j]
        for j in range(n[d] - 2, -1, -1):
            y[j] -= gam[j + 1] * y[j + 1]
        x = np.moveaxis(y, 0, 2 - d)
        res = v.copy() if keep else np.where(face, ends, v)
        inner = [slice(1, -1)] * 3
        inner[2 - d] = slice(None)
        res[tuple(inner)] = x[tuple(inner)]
        return res

    t = t0
    for _ in range(c["steps"]):
        t1 = t + dt
        E, Eh, E0 = math.exp(-t1), math.exp(-(t1 - 0.5 * dt)), math.exp(-(t1 - dt))
        J, bc = J0 * E, R2 * E
        if spec.method == "adi":
            src = F0 * E
            for r in rows:
                for g, j in zip(r.groups, r.jumps(J[r.sel])):
                    src.reshape(-1)[g["node"]] += j
            w = np.where(face, bc, u + dt * (explicit(1, u, None) + explicit(2, u, None) + src))
            w = solve(0, w, None, bc, True)
            for d in (1, 2):
                w = solve(d, np.where(face, w, w - dt * explicit(d, u, None)), None, bc, d == 1)
            u = w
        elif spec.method == "ts":
            for d in (0, 1):
                u = np.where(face, R2 * Eh, u + 0.5 * dt * explicit(d, u, J))
            w = u + 0.5 * dt * explicit(2, u, J) + 0.5 * dt * (F0 * E0 + F0 * E)
            u = solve(2, w, J, bc, False)
            u = solve(1, u, J, bc, True)
            u = solve(0, u, J, bc, True)
        else:
            for d in range(3):
                w = u + 0.5 * dt * explicit(d, u, J) if spec.method == "lod-cn" else u
                u = solve(d, w, J, bc, False)
            u = u + dt * F0 * E
        t = t1
    return u, np.where(out, R2, S) * math.exp(-t)


def exact(case, seed):
    if case["do"] in ("setup", "batch") or _nodes(case) * max(1, case["steps"]) > _EXACT_NODE_STEPS:
        return None
    spec = _spec(case)
    tags, cr, _ = M.setup_host(spec)
    u = _start_field(case, tags, seed)
    if case["do"] == "request":
        x, y, z = (np.linspace(-1.0, 1.0, k) for k in spec.n)
        inside = np.sin(2 * z)[:, None, None] * np.cos(2 * y)[None, :, None] * np.sin(2 * x)[None, None, :]
        outside = (z * z)[:, None, None] + (y * y)[None, :, None] + (x * x)[None, None, :]
        u = np.where((tags > 0).reshape(u.shape), outside, inside) * math.exp(-_t0(seed))
    u, sol = _exact_steps(spec, case, tags, cr, u, _t0(seed))
    if case["do"] == "step":
        return u.reshape(-1)
    e = np.abs(u - sol)
    return {"u": u.reshape(-1), "linf": float(e.max()), "l2": float(np.sqrt(np.mean(e * e)))}
