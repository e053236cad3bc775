"""The calls a user of this framework makes, as measurable cases.

A simulation program builds a model once (mesh, material, loads) and then
calls it: residuals R(u) for a time stepper or another solver, tangent products
K(u) v, applications of the approximate-Jacobian preconditioner H0, whole
quasi-static solves, adjoint gradients, and batches of small solves.  Each case
is one of those calls (``path``) on one model:

  geometry  "box" (a cantilever, nx x ny x nz hexahedra, or six tetrahedra per
            hexahedron), "cap" (hollow cylinder with a top plate) or "finger"
            (block with internal chambers), as efem_b200.meshgen makes them;
  etype     C3D4, C3D8, C3D10, C3D20, ``reduced`` their reduced integration;
  law       nh, mr, yeoh;
  load      follower "pressure", directed pressure "dpressure", nodal "force";
  mixed     FP32 element kernels (the library's mixed precision).

Residual, tangent and H0 calls take CUDA tensors on the caller's stream (the
device_ptrs option); solves, gradients and batches take host arrays, the
default of the interface.
"""
import functools
import math

import numpy as np
import torch

from efem_b200 import api, meshgen as mg

DEV = "cuda"


# ------------------------------------------------------------------ the cases
def _case(name, path, geometry="box", etype="C3D8", law="nh", load="pressure", reduced=False, mixed=False, nx=0, ny=0,
          nz=0, transpose=False, members=0):
    c = {"path": path, "geometry": geometry, "etype": etype, "law": law, "load": load, "reduced": reduced,
         "mixed": mixed, "nx": nx, "ny": ny, "nz": nz, "transpose": transpose, "members": members}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest model in use (the repository's first benchmark mesh): launches and waits dominate
        _case("residual_c3d4_cantilever", "residual", etype="C3D4", nx=10, ny=4, nz=4),
        # the plain FP64 baseline mesh, one residual evaluation
        _case("residual_c3d8_beam", "residual", etype="C3D8", law="mr", load="force", nx=80, ny=16, nz=16),
        # quadratic tetrahedra with chamber pressure: what meshers deliver for soft robots
        _case("residual_c3d10_finger", "residual", "finger", "C3D10", "yeoh", nx=80, ny=12, nz=12),
        # the largest model, 27 Gauss points per element, FP32 element arithmetic
        _case("residual_c3d20_mixed", "residual", etype="C3D20", law="mr", load="dpressure", mixed=True, nx=97, ny=25,
              nz=25),
        # one Newton-Krylov or sensitivity product with the true tangent
        _case("tangent_c3d10_finger", "tangent", "finger", "C3D10", "yeoh", nx=80, ny=12, nz=12, transpose=True),
        # the preconditioner used by itself inside someone else's iteration
        _case("h0_c3d8_beam", "h0", etype="C3D8", law="mr", load="force", nx=80, ny=16, nz=16),
        _case("h0_c3d20r_cap", "h0", "cap", "C3D20", reduced=True, nx=64, ny=4, nz=24),
        # whole solves: small, the mixed-versus-FP64 benchmark mesh, the finger in mixed precision
        _case("solve_c3d4_cantilever", "solve", etype="C3D4", nx=10, ny=4, nz=4),
        _case("solve_c3d20r_cap", "solve", "cap", "C3D20", reduced=True, nx=64, ny=4, nz=24),
        _case("solve_c3d10_finger_mixed", "solve", "finger", "C3D10", "yeoh", mixed=True, nx=80, ny=12, nz=12),
        # dJ/dtheta of a tip displacement, the design-optimisation call
        _case("adjoint_c3d10_finger", "adjoint", "finger", "C3D10", "yeoh", nx=80, ny=12, nz=12),
        # many uneven load cases and material samples at once
        _case("batch_c3d4_mixed", "batch", etype="C3D4", mixed=True, members=32),
    ]


def draw(rng):
    path = rng.choice(["residual", "residual", "tangent", "h0", "solve", "adjoint", "batch"])
    if path == "batch":
        return _case(None, path, etype="C3D4", mixed=rng.random() < 0.5, members=rng.randint(3, 28))
    etype = rng.choice(["C3D4", "C3D8", "C3D10", "C3D20"])
    law = rng.choice(["nh", "mr", "yeoh"])
    load = rng.choice(["pressure", "dpressure", "force"]) if path in ("residual", "tangent") else "pressure"
    # one-point C3D10 has no positive-definite approximate Jacobian: residuals only
    reduced = ((etype == "C3D20" and path in ("residual", "h0", "solve")) or (etype == "C3D10" and path == "residual")) \
        and rng.random() < 0.5
    # hexahedra along x and across; nodes and work per hexahedron differ by type
    top = {"residual": {"C3D4": 36000, "C3D8": 120000, "C3D10": 18000, "C3D20": 36000},
           "tangent": {"C3D4": 18000, "C3D8": 6000, "C3D10": 8000, "C3D20": 700},
           "h0": {"C3D4": 30000, "C3D8": 30000, "C3D10": 4500, "C3D20": 8000},
           "solve": {"C3D4": 12000, "C3D8": 9000, "C3D10": 3500, "C3D20": 5000},
           "adjoint": {"C3D4": 9000, "C3D8": 6000, "C3D10": 3000, "C3D20": 500}}[path][etype]
    hexes = math.exp(rng.uniform(math.log(50), math.log(top)))
    aspect = rng.uniform(2.0, 5.0)
    n = (hexes / aspect) ** (1.0 / 3.0)
    ny, nz = (max(2, round(n * rng.uniform(0.8, 1.25))) for _ in range(2))
    nx = max(3, round(hexes / (ny * nz)))
    return _case(None, path, etype=etype, law=law, load=load, reduced=reduced, mixed=path in ("residual", "solve") and rng.random() < 0.4,
                 nx=nx, ny=ny, nz=nz, transpose=path == "tangent" and rng.random() < 0.5)


# ------------------------------------------------------------------ meshes and models
@functools.lru_cache(maxsize=None)
def _geometry(geometry, etype, reduced, nx, ny, nz):
    """Mesh, fixed nodes, loaded faces and loaded nodes (a user's mesh file)."""
    if geometry == "cap":
        c = mg.cylinder_cap_c3d20(n_theta=nx, n_r=ny, n_z=nz, reduced=reduced)
        return c.mesh, c.fix, c.pressure[0][1], None, None
    if geometry == "finger":
        c, tip = mg.finger_c3d10(nx=nx, nyz=ny)
        return c.mesh, c.fix, c.pressure[0][1], None, tip
    h = 0.0025
    L, W, H = nx * h, ny * h, nz * h
    base = mg.box_hex8(L, W, H, nx, ny, nz)
    m = {"C3D4": lambda: mg.hex8_to_tet4(base), "C3D8": lambda: base, "C3D20": lambda: mg.hex8_to_hex20(base),
         "C3D10": lambda: mg.tet4_to_tet10(mg.hex8_to_tet4(base))}[etype]()
    tol = 1e-9
    fix = np.nonzero(np.abs(m.X[:, 0]) < tol)[0]
    end = np.nonzero(np.abs(m.X[:, 0] - L) < tol)[0]
    # only the elements that touch the end face can own one of its faces
    near = np.isin(m.conn, end).sum(axis=1) >= 3
    faces = mg.boundary_faces(mg.Mesh(m.X, m.conn[near]), lambda P: bool(np.all(np.abs(P[:, 0] - L) < tol)))
    return m, fix, faces, end, int(end[0])


def _problem(case, seed):
    """The meshgen.Case of a case: material constants and load vary with the seed."""
    rng = np.random.default_rng([seed, 17])
    mesh, fix, faces, end, tip = _geometry(case["geometry"], case["etype"], case["reduced"], case["nx"], case["ny"], case["nz"])
    s = float(rng.uniform(0.9, 1.1))
    mat = {"nh": lambda: mg.mat_nh(C10=114000.0 * s), "mr": lambda: mg.mat_mr(C10=80000.0 * s, C01=20000.0 * s),
           "yeoh": lambda: mg.mat_yeoh(C10=110000.0 * s, C20=20000.0 * s, C30=-300.0 * s)}[case["law"]]()
    prob = mg.Case(mesh, [mat], fix, integration="reduced" if case["reduced"] else "full")
    if case["geometry"] == "cap":
        p = 1.0e4
    elif case["geometry"] == "finger":
        p = 3.0e4
    else:  # a third of the cantilever's Euler load at most: beyond it no straight equilibrium is stable
        span = mesh.X.max(axis=0)
        p = min(1.0e4, 0.3 * math.pi ** 2 * 6.0 * mat["C10"] * min(span[1], span[2]) ** 2 / (48.0 * span[0] ** 2))
    p *= float(rng.uniform(0.9, 1.1))
    if case["load"] == "pressure":
        prob.pressure.append((p, faces))
    elif case["load"] == "dpressure":
        prob.pressure.append(([0.0, 0.3 * p, -0.2 * p], faces))
    else:
        prob.force.append(([0.0, 0.0, -0.001 * p / len(end)], end))
    return prob, tip


def _displacement(X, seed):
    """A smooth deformation that vanishes at x = 0: bending, twist, stretch of a few
    per cent, with a small irregular part, as solver iterates have."""
    rng = np.random.default_rng([seed, 29])
    span = X.max(axis=0) - X.min(axis=0)
    q = (X - X.min(axis=0)) / span
    u = np.zeros_like(X)
    for c in range(3):
        a = rng.uniform(-1.0, 1.0, 5)
        u[:, c] = 0.02 * span.min() * q[:, 0] * (a[0] + a[1] * q[:, 0] + a[2] * q[:, 1] + a[3] * q[:, 2]
                                                 + a[4] * np.sin(3.0 * q[:, 0] + 2.0 * q[:, 1]))
    return u + 2e-6 * q[:, :1] * rng.normal(size=X.shape)


def _free(prob):
    free = np.ones(prob.mesh.X.shape[0], dtype=bool)
    free[prob.fix] = False
    return np.nonzero(free)[0]


@functools.lru_cache(maxsize=4)
def _batch_meshes(members):
    return mg.batch_beams(n=members, seed=1000, el_max=20000)


def _batch(case, seed):
    """One set of meshes; each member's material constants and pressure vary with the seed."""
    rng = np.random.default_rng([seed, 53])
    out = []
    for c in _batch_meshes(case["members"]):
        mat = dict(c.materials[0])
        s = float(rng.uniform(0.8, 1.25))
        for k in ("C10", "C01"):
            if k in mat:
                mat[k] *= s
        p, faces = c.pressure[0]
        out.append(mg.Case(c.mesh, [mat], c.fix, pressure=[(p * s * float(rng.uniform(0.7, 1.0)), faces)]))
    return out


def _vectors(case, prob, seed):
    """(u, v): a displacement and a direction (or load) on the free DOFs."""
    free = _free(prob)
    u = _displacement(prob.mesh.X, seed)[free].ravel()
    v = np.random.default_rng([seed, 41]).normal(size=u.size)
    return u, v


def _options(case):
    o = api.default_options()
    o.precision = api.MIXED if case["mixed"] else api.FP64
    # converged well inside the configs' 1e-6 N, so that the answer is defined to more digits than the test asks
    o.residual_criterion = 1e-8
    return o


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        probs = _batch(case, seed)
        return {"path": path, "models": [api.Model.from_case(p, _options(case)) for p in probs]}
    prob, tip = _problem(case, seed)
    o = _options(case)
    st = {"path": path, "transpose": case["transpose"]}
    if path in ("residual", "tangent", "h0"):
        o.device_ptrs = 1
        st["model"] = m = api.Model.from_case(prob, o)
        st["stream"] = torch.cuda.Stream()
        m.set_stream(st["stream"].cuda_stream)
        u, v = _vectors(case, prob, seed)
        st["u"], st["v"] = (torch.from_numpy(x).to(DEV) for x in (u, v))
        st["out"] = torch.zeros_like(st["u"])
        if path == "h0":  # the factor is the plan that such a program keeps
            torch.cuda.synchronize()
            m.precond_apply(st["v"].clone())
        return st
    st["model"] = m = api.Model.from_case(prob, o)
    if path == "adjoint":
        st["u"], _ = m.solve()
        g = np.zeros(m.n_dof)
        g[3 * int(np.searchsorted(_free(prob), tip)) + 2] = 1.0
        st["g"] = g
    return st


def run(st):
    path = st["path"]
    if path == "residual":
        return st["model"].residual(st["u"], st["out"])
    if path == "tangent":
        with torch.cuda.stream(st["stream"]):
            return st["model"].hvp(st["u"], st["v"], transpose=st["transpose"])
    if path == "h0":
        with torch.cuda.stream(st["stream"]):
            st["out"].copy_(st["v"])
            return st["model"].precond_apply(st["out"])
    if path == "solve":
        return st["model"].solve()[0]
    if path == "adjoint":
        dtheta, lam, _ = st["model"].adjoint(st["u"], st["g"], want_lambda=True)
        return {"dtheta": dtheta, "lambda": lam}
    us, _ = api.batch_solve(st["models"])
    return np.concatenate(us)


# ------------------------------------------------------------------ what a pass cannot do without
_NGP = {("C3D4", False): 1, ("C3D10", False): 4, ("C3D10", True): 1, ("C3D8", False): 8, ("C3D20", False): 27, ("C3D20", True): 8}
_NEN = {"C3D4": 4, "C3D8": 8, "C3D10": 10, "C3D20": 20}


def _size(case):
    """(nodes, elements) without building the mesh."""
    nx, ny, nz, t = case["nx"], case["ny"], case["nz"], case["etype"]
    if case["geometry"] == "cap":
        ne = nx * ny * nz + 2 * (19 * nx + (nx // 4) ** 2)
        return 4.95 * ne, ne
    hexes = nx * ny * nz
    if case["geometry"] == "finger":
        hexes = 8448 * hexes / 11520
    node = {"C3D4": 1.0, "C3D8": 1.0, "C3D10": 8.0, "C3D20": 4.0}[t]
    if case["geometry"] == "finger":
        return 9.6 * hexes, 6 * hexes
    return node * (nx + 1) * (ny + 1) * (nz + 1), hexes * (6 if t in ("C3D4", "C3D10") else 1)


def _residual_work(case):
    nn, ne = _size(case)
    law = {"nh": 260.0, "mr": 510.0, "yeoh": 270.0}[case["law"]]
    nen, ngp = _NEN[case["etype"]], _NGP[case["etype"], case["reduced"]]
    # connectivity, reference coordinates, u read once; r written once
    return 4.0 * nen * ne + 72.0 * nn, ngp * (36.0 * nen + law) * ne


def _factor_nnz(nn):
    return 8.0 * nn ** (4.0 / 3.0)  # nested dissection of a 3D mesh, as the beam's factor measures


def _solve_work(case, iters):
    nn, _ = _size(case)
    rb, rf = _residual_work(case)
    # per iteration: a residual, the factor read by both sweeps, the twelve history vectors read twice
    per = rb + 16.0 * _factor_nnz(nn) + 24.0 * 3.0 * nn * 8.0
    return iters * per, iters * (rf + 12.0 * _factor_nnz(nn)) + 60.0 * nn ** 2


def work(case):
    path = case["path"]
    if path == "batch":
        one = dict(case, etype="C3D4", geometry="box", nx=50, ny=5, nz=5, law="nh", reduced=False)
        b, f = _solve_work(one, 100)
        return {"bytes": case["members"] * b, "flops": case["members"] * f}
    nn, _ = _size(case)
    if path == "residual":
        b, f = _residual_work(case)
    elif path == "tangent":
        b, f = _residual_work(case)
        b, f = b + 24.0 * nn, 2.0 * f
    elif path == "h0":
        b, f = 16.0 * _factor_nnz(nn) + 48.0 * nn, 12.0 * _factor_nnz(nn)
    elif path == "solve":
        b, f = _solve_work(case, 100)
    else:  # GMRES: per iteration H0, a tangent product and the basis twice
        b, f = _solve_work(case, 100)
        b += 100 * 2 * 50 * 24.0 * nn
    return {"bytes": b, "flops": f}


def tolerance(case):
    path = case["path"]
    if path in ("residual", "tangent"):
        return {"rel": 4e-6, "max": 1e-3} if case["mixed"] else {"rel": 4e-12, "max": 1e-9}
    if path == "h0":
        return {"rel": 1e-11, "max": 1e-9}
    if path == "adjoint":  # GMRES to a relative residual of 1e-8
        return {"rel": 1e-5, "max": 1e-3}
    # solves stop inside a ball of 1e-8 N
    return {"rel": 1e-4, "max": 1e-2}


# ------------------------------------------------------------------ 64-bit answers in plain torch
_HEX8 = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)
_HEX20 = np.array([[1, -1, 1], [1, 1, 1], [1, 1, -1], [1, -1, -1], [-1, -1, 1], [-1, 1, 1], [-1, 1, -1], [-1, -1, -1]], float)
_EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]


def _shape(etype, p):
    """N and dN/dxi at one local point, the derivatives by autograd."""
    def N_of(q):
        x, y, z = q[0], q[1], q[2]
        if etype == "C3D4":
            return torch.stack([x, y, z, 1 - x - y - z])
        if etype == "C3D10":
            L = 1 - x - y - z
            return torch.stack([L * (2 * L - 1), x * (2 * x - 1), y * (2 * y - 1), z * (2 * z - 1), 4 * L * x, 4 * x * y,
                                4 * y * L, 4 * z * L, 4 * x * z, 4 * y * z])
        if etype == "C3D8":
            return torch.stack([(1 + s[0] * x) * (1 + s[1] * y) * (1 + s[2] * z) / 8 for s in _HEX8])
        out = [(1 + s[0] * x) * (1 + s[1] * y) * (1 + s[2] * z) * (s[0] * x + s[1] * y + s[2] * z - 2) / 8 for s in _HEX20]
        for a, b in _EDGES:
            c = 0.5 * (_HEX20[a] + _HEX20[b])
            f = [(1 - t * t) if ck == 0 else (1 + ck * t) for ck, t in zip(c, (x, y, z))]
            out.append(f[0] * f[1] * f[2] / 4)
        return torch.stack(out)

    q = torch.tensor(p, dtype=torch.float64)
    return N_of(q), torch.autograd.functional.jacobian(N_of, q)


def _rule(etype, reduced):
    if etype == "C3D4" or (etype == "C3D10" and reduced):
        return [[0.25] * 3], [1.0]
    if etype == "C3D10":
        a, b = 0.58541020, 0.13819660  # the discretisation's own 8-digit constants
        return [[a, b, b], [b, a, b], [b, b, a], [b, b, b]], [0.25] * 4
    if etype == "C3D8" or reduced:
        return (_HEX8 / math.sqrt(3.0)).tolist(), [0.125] * 8
    c, q, w = math.sqrt(0.6), [-1, 0, 1], [5 / 18, 8 / 18, 5 / 18]
    return ([[c * q[i], c * q[j], c * q[k]] for k in range(3) for j in range(3) for i in range(3)],
            [w[i] * w[j] * w[k] for k in range(3) for j in range(3) for i in range(3)])


def _face_points(etype, miss):
    """Local points and weights of the face that lacks the given element corner(s)."""
    if etype == "C3D4":
        p = [1 / 3] * 3
        if miss < 3:
            p[miss] = 0.0
        return [p], [1.0]
    if etype == "C3D10":
        pts = []
        for g in range(3):
            if miss == 0:
                pts.append([2 / 3 if k == g else 1 / 6 for k in range(3)])
            else:
                o = [k for k in range(3) if k != miss - 1]
                p = [0.0] * 3
                p[o[0]], p[o[1]] = (2 / 3 if g == 0 else 1 / 6), (2 / 3 if g == 1 else 1 / 6)
                pts.append(p)
        return pts, [1 / 3] * 3
    ax, val = ([(2, 1), (1, 1), (0, 1), (1, -1), (0, -1), (2, -1)] if etype == "C3D8"
               else [(0, -1), (2, -1), (1, 1), (2, 1), (1, -1), (0, 1)])[miss]
    o = [k for k in range(3) if k != ax]
    if etype == "C3D8":
        t, w = [-math.sqrt(1 / 3), math.sqrt(1 / 3)], [0.5, 0.5]
    else:
        t, w = [-math.sqrt(0.6), 0.0, math.sqrt(0.6)], [5 / 18, 8 / 18, 5 / 18]
    pts, ws = [], []
    for i in range(len(t)):
        for j in range(len(t)):
            p = [0.0] * 3
            p[ax], p[o[0]], p[o[1]] = val, t[i], t[j]
            pts.append(p)
            ws.append(w[i] * w[j])
    return pts, ws


def _stress(F, theta, law):
    C10, C01, C20, C30, D1 = theta
    I = torch.eye(3, dtype=F.dtype, device=F.device)
    J = torch.linalg.det(F)[..., None, None]
    FiT = torch.linalg.inv(F).transpose(-1, -2)
    C = F.transpose(-1, -2) @ F
    I1 = C.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
    Jm = (J * J) ** (-1.0 / 3.0)
    t = I1 * Jm - 3
    coef = C10 + 2 * C20 * t + 3 * C30 * t * t if law == "yeoh" else C10
    P = coef * Jm * (2 * F - 2.0 / 3.0 * I1 * FiT) + 2 / D1 * (J - 1) * J * FiT
    if law == "mr":
        I2 = 0.5 * (I1 * I1 - (C @ C).diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None])
        P = P + C01 * Jm * Jm * (2 * F @ (I1 * I - C) - 4.0 / 3.0 * I2 * FiT)
    return P


class _Plain:
    """The discrete problem in 64-bit torch."""

    def __init__(self, case, prob):
        self.etype, self.law = case["etype"], case["law"]
        T = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
        X, conn = T(prob.mesh.X), T(prob.mesh.conn)
        free = T(_free(prob))
        self.nn, self.nf, self.free, self.conn = X.shape[0], free.numel(), free, conn
        self.slot = torch.full((self.nn,), self.nf, dtype=torch.long, device=DEV)
        self.slot[free] = torch.arange(self.nf, device=DEV)
        pts, w = _rule(self.etype, case["reduced"])
        self.dN = torch.stack([_shape(self.etype, p)[1] for p in pts]).to(DEV)          # (g, a, 3)
        Y = X[conn]
        J0 = torch.einsum("eai,gak->egik", Y, self.dN)
        self.B = torch.einsum("gak,egki->egai", self.dN, torch.linalg.inv(J0))          # dN/dX
        if self.etype in ("C3D4", "C3D10"):
            vol = torch.linalg.det(Y[:, 1:4] - Y[:, :1]).abs() / 6
        else:
            vol = 0
            for f in [(0, 3, 2, 1), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7)]:
                a, b, c, d = (Y[:, k] for k in f)
                vol = vol + (a * (torch.cross(b, c, dim=1) + torch.cross(c, d, dim=1))).sum(1)
            vol = vol.abs() / 6
        self.wv = vol[:, None] * T(np.array(w))[None]
        m = prob.materials[0]
        self.theta = [float(m.get(k, 0.0)) for k in ("C10", "C01", "C20", "C30", "D1")]
        self.kappa = 2.94001 * self.theta[0] + 2 / self.theta[4] + (3.818 * self.theta[1] if self.law == "mr" else 0)
        if self.law == "yeoh":
            self.kappa += 3.51194 * self.theta[2] + 3.3154 * self.theta[3]
        self.fext = torch.zeros(self.nf + 1, 3, dtype=torch.float64, device=DEV)
        for value, nodes in prob.force:
            n = T(np.asarray(nodes))
            self.fext.index_add_(0, self.slot[n], T(np.asarray(value, float)).expand(n.numel(), 3).contiguous())
        self.faces, self.value = [], None
        if prob.pressure:
            self.value, faces = prob.pressure[0]
            self._set_faces(np.asarray(faces), prob.mesh, X)

    def _set_faces(self, faces, mesh, X):
        nc = 3 if self.etype in ("C3D4", "C3D10") else 4
        corners = 4 if nc == 3 else 8
        on = np.isin(mesh.conn[:, :corners], np.unique(faces[:, :nc]))
        groups = {}
        pairs = [(0, 2), (0, 5), (0, 7), (6, 3), (6, 1), (6, 4)]
        owner = {}
        for e in np.nonzero(on.sum(1) >= nc)[0]:
            for v in mesh.conn[e, :corners]:
                owner.setdefault(int(v), []).append(e)
        for f in faces:
            key = set(int(v) for v in f[:nc])
            e = next(e for e in owner[int(f[0])] if key <= set(mesh.conn[e, :corners].tolist()))
            has = [int(v) in key for v in mesh.conn[e, :corners]]
            miss = has.index(False) if nc == 3 else next(k for k, p in enumerate(pairs) if not has[p[0]] and not has[p[1]])
            groups.setdefault(miss, []).append((e, f))
        for miss, g in groups.items():
            e = torch.as_tensor(np.array([x[0] for x in g]), device=DEV)
            f = torch.as_tensor(np.array([x[1] for x in g]), device=DEV)
            ref = X[self.conn[e, miss if nc == 3 else pairs[miss][0]]]
            P = [X[f[:, k]] for k in range(nc)]

            def area(a, b, c):
                A = 0.5 * torch.cross(c - a, b - a, dim=1)
                return torch.where((((ref - P[0]) * A).sum(1) < 0)[:, None], -A, A)
            A0 = area(P[0], P[1], P[2]) if nc == 3 else area(P[0], P[1], P[2]) + area(P[3], P[2], P[0])
            pts, w = _face_points(self.etype, miss)
            sh = [_shape(self.etype, p) for p in pts]
            N, dN = torch.stack([s[0] for s in sh]).to(DEV), torch.stack([s[1] for s in sh]).to(DEV)
            J0 = torch.einsum("eai,gak->egik", X[self.conn[e]], dN)
            B = torch.einsum("gak,egki->egai", dN, torch.linalg.inv(J0))
            self.faces.append((self.conn[e], A0, N * torch.tensor(w, dtype=torch.float64, device=DEV)[:, None], B))

    def _nodal(self, u):
        full = torch.zeros(self.nn, 3, dtype=u.dtype, device=u.device)
        return full.index_copy(0, self.free, u.reshape(-1, 3))

    def residual(self, u, theta=None, scale=None):
        U = self._nodal(u)
        I = torch.eye(3, dtype=u.dtype, device=u.device)
        F = I + torch.einsum("eai,egaj->egij", U[self.conn], self.B)
        S = _stress(F, self.theta if theta is None else theta, self.law) * self.wv[..., None, None]
        f = torch.einsum("egij,egaj->eai", S, self.B)
        r = torch.zeros_like(self.fext).index_add(0, self.slot[self.conn].reshape(-1), f.reshape(-1, 3)) - self.fext
        for conn, A0, wN, B in self.faces:
            F = I + torch.einsum("eai,egaj->egij", U[conn], B)
            cA = torch.linalg.det(F)[..., None] * torch.einsum("egji,ej->egi", torch.linalg.inv(F), A0)
            if isinstance(self.value, (list, tuple)):
                v = torch.tensor(self.value, dtype=u.dtype, device=u.device) * (1.0 if scale is None else scale)
                f = torch.einsum("ga,eg->ea", wN, cA.norm(dim=-1))[..., None] * v
            else:
                f = torch.einsum("ga,egi->eai", wN, cA) * (self.value if scale is None else scale)
            r = r.index_add(0, self.slot[conn].reshape(-1), -f.reshape(-1, 3))
        return r[:self.nf].reshape(-1)

    def tangent(self, u, v, transpose):
        if transpose:
            u = u.clone().requires_grad_(True)
            return torch.autograd.grad(self.residual(u), u, v)[0]
        return torch.func.jvp(self.residual, (u,), (v,))[1]

    def dense_tangent(self, u):
        x = u.clone().requires_grad_(True)
        r = self.residual(x)
        return torch.stack([torch.autograd.grad(r[i], x, retain_graph=True)[0] for i in range(x.numel())])

    def h0(self, v):
        L = torch.zeros(self.nf + 1, self.nf + 1, dtype=torch.float64, device=DEV)
        s = self.slot[self.conn]
        for c in range(0, s.shape[0], 4096):
            B, w, q = self.B[c:c + 4096], self.wv[c:c + 4096] * self.kappa, s[c:c + 4096]
            K = torch.einsum("egai,egbi,eg->eab", B, B, w)
            L.view(-1).index_add_(0, (q[:, :, None] * (self.nf + 1) + q[:, None, :]).reshape(-1), K.reshape(-1))
        L = L[:self.nf, :self.nf].contiguous()
        L = torch.linalg.cholesky(L)
        return torch.cholesky_solve(v.reshape(-1, 3), L).reshape(-1)

    def solve(self):
        u = torch.zeros(3 * self.nf, dtype=torch.float64, device=DEV)
        for _ in range(12):
            r = self.residual(u)
            if float(r.abs().max()) < 1e-11:
                break
            u = u - torch.linalg.solve(self.dense_tangent(u), r)
        return u


_DENSE = 1500  # unknowns up to which the tangent is formed whole


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        return None
    prob, tip = _problem(case, seed)
    dof = 3 * _free(prob).size
    if path in ("solve", "adjoint") and dof > _DENSE:
        return None
    P = _Plain(case, prob)
    u, v = (torch.from_numpy(x).to(DEV) for x in _vectors(case, prob, seed))
    if path == "residual":
        return P.residual(u)
    if path == "tangent":
        return P.tangent(u, v, case["transpose"])
    if path == "h0":
        return P.h0(v)
    u = P.solve()
    if path == "solve":
        return u.cpu().numpy()
    g = torch.zeros(dof, dtype=torch.float64, device=DEV)
    g[3 * int(np.searchsorted(_free(prob), tip)) + 2] = 1.0
    lam = torch.linalg.solve(P.dense_tangent(u).T, g)
    theta = [torch.tensor(t, dtype=torch.float64, device=DEV, requires_grad=True) for t in P.theta + [P.value]]
    d = torch.autograd.grad(P.residual(u, theta[:5], theta[5]), theta, -lam, allow_unused=True)
    return {"dtheta": np.array([0.0 if x is None else float(x) for x in d]), "lambda": lam.cpu().numpy()}
