"""The work that a user of the framework has it do, as cases to be timed.

Every case is a call sequence through the public API of
xcalibre_tw.jl_b200/xcal: fields in, SIMPLE or PISO iterations, fields and
histories out; a user-built equation assembled and solved; a stream of cases
served.  Meshes come from the repository's own generators at the sizes of its
configurations, tests and benchmark and in between.

What a user's program holds before the call (mesh, context with the uploaded
mesh and case, host fields) is made in prepare(); the seed sets the viscosity
and the initial fields, a smooth flow as a restart from an earlier run has.

kinds of case
    run        X.Solver kept by the caller: set_field, run, get_field
    simple     X.simple, the drop-in call: context, upload, run and read-back
    operators  xcal.operators: assemble a convection-diffusion equation, solve
               it, and take the gradient of the solution
    serve      X.Server: open, submit a stream of cases, collect, close
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xcalibre_tw.jl_b200"))

import xcal as X  # noqa: E402
from xcal import _abi, cases as C, meshgen, operators as op  # noqa: E402

FIELDS = (_abi.FIELD_UX, _abi.FIELD_UY, _abi.FIELD_UZ, _abi.FIELD_P)
TURB = (_abi.FIELD_K, _abi.FIELD_OMEGA, _abi.FIELD_NUT)


def listed():
    return [
        # the drop-in call on the reference's own example size, set-up included
        {"name": "simple_cavity_40", "kind": "simple", "geom": "cavity2d", "n": 40, "prec": "fp64", "scheme": "upwind",
         "iters": 20},
        # the smallest mesh on a kept context: a phase is launch and barrier latency
        {"name": "cavity_40", "kind": "run", "geom": "cavity2d", "n": 40, "prec": "fp64", "scheme": "upwind",
         "iters": 20},
        # transient run on a small non-orthogonal mesh (Euler time, two correctors)
        {"name": "piso_bfs_4k", "kind": "run", "geom": "bfs", "n": 8, "prec": "fp64", "scheme": "piso", "iters": 10},
        # an ordinary 2D case in mixed precision, odd size
        {"name": "cavity_157_mixed", "kind": "run", "geom": "cavity2d", "n": 157, "prec": "mixed", "scheme": "upwind",
         "iters": 10},
        # the laminar backward-facing step of the benchmark
        {"name": "bfs_47k", "kind": "run", "geom": "bfs", "n": 27, "prec": "fp64", "scheme": "upwind", "iters": 10},
        # the turbulent flat plate of the benchmark: two more transport equations
        {"name": "flatplate_150k_mixed", "kind": "run", "geom": "flatplate", "n": 600, "m": 250, "prec": "mixed",
         "scheme": "upwind", "iters": 8},
        # the largest 2D mesh, central schemes and the corrected gradient
        {"name": "cavity_400_midpoint", "kind": "run", "geom": "cavity2d", "n": 400, "prec": "fp64",
         "scheme": "midpoint", "iters": 8},
        # 3D: small, ragged in mixed precision, and the benchmark's 2.1 M cells
        {"name": "cavity3d_32", "kind": "run", "geom": "cavity3d", "n": 32, "prec": "fp64", "scheme": "upwind",
         "iters": 10},
        {"name": "cavity3d_101_mixed", "kind": "run", "geom": "cavity3d", "n": 101, "prec": "mixed",
         "scheme": "upwind", "iters": 4},
        {"name": "cavity3d_128", "kind": "run", "geom": "cavity3d", "n": 128, "prec": "fp64", "scheme": "upwind",
         "iters": 4},
        # a user-built equation in the caller's own numbering (a level-scheduled preconditioner)
        {"name": "operators_bfs_7k", "kind": "operators", "geom": "bfs", "n": 10},
        # a stream of small cases in flight together
        {"name": "serve_16", "kind": "serve", "n": 16, "stream": 5, "nmax": 200, "prec": "mixed", "iters": 60},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(("cavity2d", "cavity2d", "bfs", "bfs", "flatplate", "cavity3d", "cavity3d", "simple",
                       "operators", "serve"))
    prec = rng.choice(("fp64", "mixed"))
    if kind == "operators":
        return {"kind": "operators", "geom": "bfs", "n": log(3, 11)}
    if kind == "serve":
        return {"kind": "serve", "n": rng.randint(6, 16), "stream": rng.randint(0, 999), "nmax": rng.randint(80, 200),
                "prec": prec, "iters": rng.randint(30, 80)}
    c = {"kind": "run", "geom": kind, "prec": prec, "scheme": "upwind", "iters": rng.randint(4, 8)}
    if kind == "simple":
        c.update(kind="simple", geom="cavity2d", n=log(24, 80), iters=rng.randint(10, 30))
    elif kind == "flatplate":
        c.update(n=log(150, 600), m=rng.randint(60, 250))
    elif kind == "cavity3d":
        c.update(n=log(16, 120), iters=4)
    else:
        c["scheme"] = rng.choice(("upwind", "upwind", "piso") + (("midpoint",) if kind == "cavity2d" else ()))
        c["n"] = log(40, 400) if kind == "cavity2d" else log(5, 49)
    return c


# ------------------------------------------------------------------ meshes
@functools.lru_cache(maxsize=None)
def _mesh(geom, n, m=0):
    if geom == "cavity2d":
        return X.build_mesh(C._unv("cavity", meshgen.cavity_unv, n=n, L=0.1))
    if geom == "bfs":
        return X.build_mesh(C._unv("bfs", meshgen.bfs_unv, cells_per_h=n))
    if geom == "flatplate":
        return X.build_mesh(C._unv("flatplate", meshgen.flatplate_unv, nx=n, ny=m))
    return X.Mesh2.from_dict(meshgen.hex_cavity(n))


def _cells(case):
    n = case["n"]
    return {"cavity2d": n * n, "bfs": 65 * n * n, "flatplate": n * case.get("m", 0), "cavity3d": n ** 3}[case["geom"]]


# ------------------------------------------------------------------- cases
def _model(geom, mesh, iters, scheme, rng):
    """Model, configuration and pref of a run; the Reynolds number from the seed."""
    kw = {}
    if scheme == "midpoint":
        kw = dict(divergence=X.Linear, gradient=X.Midpoint)
    if geom == "cavity2d":
        _, model, config, pref = C.cavity2d(iterations=iters, nu=0.1 / rng.uniform(50.0, 400.0), mesh=mesh, **kw)
    elif geom == "bfs":
        _, model, config, pref = C.bfs(iterations=iters, nu=0.5 * 0.01 / rng.uniform(20.0, 60.0), mesh=mesh, **kw)
    elif geom == "flatplate":
        _, model, config, pref = C.flatplate(iterations=iters, mesh=mesh)
    else:
        model, config, pref = _cavity3d(mesh, iters, 1.0 / rng.uniform(200.0, 1000.0))
    if scheme == "piso":
        config["schemes"]["U"] = X.set_schemes(time=X.Euler, divergence=X.Upwind)
        config["runtime"] = X.set_runtime(iterations=iters, write_interval=-1, time_step=2e-4)
    return model, config, pref


def _cavity3d(mesh, iters, nu):
    model = X.RANS(X.Laminar, mesh=mesh, viscosity=X.ConstantScalar(nu))
    walls = ("xmin", "xmax", "ymin", "zmin", "zmax")
    X.assign(model, "U", *[X.Dirichlet(w, [0.0, 0.0, 0.0]) for w in walls], X.Dirichlet("lid", [1.0, 0.0, 0.0]))
    X.assign(model, "p", *[X.Neumann(w, 0.0) for w in walls + ("lid",)])
    schemes = dict(U=X.set_schemes(divergence=X.Upwind), p=X.set_schemes(divergence=X.Upwind))
    config = X.Configuration(solvers=C.solvers_for(model), schemes=schemes,
                             runtime=X.set_runtime(iterations=iters, write_interval=-1, time_step=1))
    return model, config, 0.0


def _smooth(cc, rng, modes=4):
    """A smooth field of a few random waves over the mesh, of order one."""
    lo = cc.min(axis=0)
    s = (cc - lo) / max(float((cc.max(axis=0) - lo).max()), 1e-300)
    f = np.zeros(len(cc))
    for _ in range(modes):
        k = rng.uniform(0.5, 3.0, 3) * math.pi
        f += rng.uniform(-1.0, 1.0) * np.sin(s @ k + rng.uniform(0.0, 2.0 * math.pi))
    return f / modes


def _initial(model, geom, rng):
    """Initial fields: the case's own start plus a smooth flow, as a restart has."""
    mesh = model.mesh
    cc = mesh.cell_centres()
    speed = {"cavity2d": 0.2, "bfs": 0.1, "flatplate": 0.2, "cavity3d": 0.2}[geom]
    start = {"bfs": 0.25, "flatplate": 10.0}.get(geom, 0.0)
    model.U.x.values[:] = start + speed * _smooth(cc, rng)
    model.U.y.values[:] = 0.2 * speed * _smooth(cc, rng)
    model.U.z.values[:] = 0.2 * speed * _smooth(cc, rng) if mesh.dim == 3 else 0.0
    model.p.values[:] = 0.1 * speed * speed * _smooth(cc, rng)
    out = [f.values.copy() for f in (model.U.x, model.U.y, model.U.z, model.p)]
    if model.turbulence is not None:
        t = model.turbulence
        for f in (t.k, t.omega, t.nut):
            f.values[:] *= 1.0 + 0.2 * _smooth(cc, rng)
            out.append(f.values.copy())
    return out


def _serve_stream(case, seed):
    """Sizes from the case, Reynolds numbers and initial fields from the seed."""
    sizes, rng = np.random.default_rng(case["stream"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["n"]):
        bfs = sizes.random() < 0.5
        N = int(round(math.exp(sizes.uniform(math.log(40), math.log(case["nmax"])))))
        geom, n = ("bfs", max(2, int(round(N / math.sqrt(65.0))))) if bfs else ("cavity2d", N)
        model, config, pref = _model(geom, _mesh(geom, n), 1, "upwind", rng)
        _initial(model, geom, rng)
        out.append((model, config, pref))
    return out


def _precision(case):
    return _abi.PREC_MIXED if case["prec"] == "mixed" else _abi.PREC_FP64


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "serve":
        return {"kind": kind, "case": case, "stream": _serve_stream(case, seed)}
    mesh = _mesh(case["geom"], case["n"], case.get("m", 0))
    if kind == "operators":
        return dict(_equation(mesh, rng), kind=kind)
    model, config, pref = _model(case["geom"], mesh, case["iters"], case["scheme"], rng)
    st = {"kind": kind, "model": model, "config": config, "pref": pref, "prec": _precision(case),
          "fields": _initial(model, case["geom"], rng), "iters": case["iters"], "piso": case["scheme"] == "piso"}
    if kind == "run":
        st["solver"] = X.Solver(mesh)
        c, st["keep"] = X.make_case(model, config, pref, st["prec"])
        st["solver"].setup(c)
        st["which"] = FIELDS + (TURB if model.turbulence is not None else ())
    return st


# --------------------------------------------------------------- operators
def _equation(mesh, rng):
    cc = mesh.cell_centres()
    n, nf = mesh.ncells, mesh.nfaces
    E = op.Equation(mesh)
    phi = X.ScalarField(mesh, _smooth(cc, rng))
    flux = 1e-4 * mesh.face_area * _smooth(mesh.face_centre.reshape(-1, 3), rng)
    gamma = 1e-3 * (1.0 + 0.3 * rng.random(nf))
    src = _smooth(cc, rng)
    si = 20.0 + rng.random(n)   # keeps the matrix diagonally dominant
    model = (op.Divergence[op.Upwind](flux, phi) - op.Laplacian[op.Linear](gamma, phi) + op.Si(si, phi)
             == op.Source(src))
    bcs = (X.Dirichlet("inlet", float(rng.uniform(0.5, 1.5))), X.Neumann("outlet", 0.0), X.Dirichlet("wall", 0.0),
           X.Neumann("top", 0.0))
    setup = X.set_solver(phi, solver=X.BicgstabSolver, preconditioner=X.DILU(), convergence=1e-7, relax=1.0,
                         itmax=400, atol=1e-13, rtol=1e-10)
    return {"mesh": mesh, "eqn": model >> E, "bcs": bcs, "setup": setup, "flux": flux, "gamma": gamma, "src": src,
            "si": si}


def _run_operators(st):
    op.discretise(st["eqn"])
    A, b = op.apply_boundary_conditions(st["eqn"], st["bcs"])
    x = op.run(st["eqn"], st["setup"])
    return {"A": A.copy(), "b": b.copy(), "x": x, "grad": op.grad(st["eqn"], x, st["bcs"])}


def run(st):
    kind = st["kind"]
    if kind == "operators":
        return _run_operators(st)
    if kind == "serve":
        return _run_serve(st)
    if kind == "simple":
        m = st["model"]
        for f, v in zip((m.U.x, m.U.y, m.U.z, m.p), st["fields"]):
            f.values[:] = v
        R = X.simple(m, st["config"], pref=st["pref"], precision=st["prec"])
        return {"R": list(R), "fields": [f.values.copy() for f in (m.U.x, m.U.y, m.U.z, m.p)]}
    s = st["solver"]
    for which, v in zip(st["which"], st["fields"]):
        s.set_field(which, v)
    out = s.run(st["iters"], piso=st["piso"])
    return {"R": [out["R_ux"], out["R_uy"], out["R_uz"], out["R_p"]], "krylov": out["krylov"], "done": out["done"],
            "fields": [s.get_field(w) for w in st["which"]]}


def _run_serve(st):
    case = st["case"]
    srv = X.Server(slots=64, max_iterations=case["iters"], tolerance=1e-6, precision=_precision(case),
                   device_bytes=4e8, host_bytes=2.5e8)
    try:
        tickets = [srv.submit(*c) for c in st["stream"]]
        got = [srv.poll(t, wait_ms=-1) for t in tickets]
    finally:
        srv.close()
    return {"iterations": [g["iterations"] for g in got], "U": np.concatenate([g["U"].ravel() for g in got]),
            "p": np.concatenate([g["p"] for g in got])}


# -------------------------------------------------------------------- work
def _iteration_work(n, dim, prec, turb, piso):
    """Bytes and operations of one SIMPLE iteration over n cells.  Krylov work
    per iteration: the matrix (values and int32 columns) and the operand
    vectors read, the result written, for the product and for the two sweeps
    of the preconditioner, and the vector updates.  The pressure solve takes
    about two iterations per cell across the domain up to its limit of 100,
    the transport solves about two in all."""
    ns, row = (3, 7) if dim == 3 else (2, 5)
    s = 4 if prec == "mixed" else 8
    across = n ** (1.0 / dim)
    p_its, t_its = min(100.0, 2.0 * across), 2.0
    matrix = row * n * (s + 4)
    cg = 2 * matrix + 13 * n * s
    bicg = 4 * matrix + 20 * n * ns * s
    faces = (row - 1) / 2 * n
    asm = 2 * (faces * 56 + row * n * 8) + n * 8 * (6 + 5 * ns)
    corr = 2 if piso else 1
    nbytes = corr * p_its * cg + t_its * bicg + (1 + corr) * asm
    flops = corr * p_its * n * (4 * row + 12) + t_its * n * ns * (8 * row + 20) + (1 + corr) * n * 60
    if turb:
        nbytes += 2 * (t_its * (4 * matrix + 20 * n * s) + asm)
        flops += 2 * (t_its * n * (8 * row + 20) + n * 60)
    return nbytes, flops


def work(case):
    if case["kind"] == "serve":
        sizes, total = np.random.default_rng(case["stream"]), [0.0, 0.0]
        for _ in range(case["n"]):
            bfs = sizes.random() < 0.5
            N = int(round(math.exp(sizes.uniform(math.log(40), math.log(case["nmax"])))))
            n = 65 * max(2, int(round(N / math.sqrt(65.0)))) ** 2 if bfs else N * N
            b, f = _iteration_work(n, 2, case["prec"], False, False)
            total = [total[0] + case["iters"] * b, total[1] + case["iters"] * f]
        return {"bytes": total[0], "flops": total[1]}
    n = _cells(case)
    if case["kind"] == "operators":
        # assembly and gradient once; about 30 BiCGSTAB iterations to 1e-10
        b = 30 * (4 * 5 * n * 12 + 20 * n * 8) + 2 * n * 56 * 2 + 5 * n * 12 + 6 * n * 8
        return {"bytes": float(b), "flops": float(30 * n * 60 + n * 80)}
    b, f = _iteration_work(n, 3 if case["geom"] == "cavity3d" else 2, case["prec"], case["geom"] == "flatplate",
                           case["scheme"] == "piso")
    return {"bytes": case["iters"] * b, "flops": case["iters"] * f}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The equation of the operators case assembled in numpy, solved directly,
    and its gradient.  The iterates of a SIMPLE run after a given number of
    steps have no value of their own beside the algorithm's."""
    if case["kind"] != "operators":
        return None
    mesh = _mesh(case["geom"], case["n"])
    st = _Plain(mesh, np.random.default_rng(seed))
    return st.solve()


class _Plain:
    """The operators case restated on the mesh arrays."""

    def __init__(self, mesh, rng):
        self.mesh = mesh
        cc = mesh.cell_centres()
        _smooth(cc, rng)   # the phi of the equation: drawn, not used by it
        self.flux = 1e-4 * mesh.face_area * _smooth(mesh.face_centre.reshape(-1, 3), rng)
        self.gamma = 1e-3 * (1.0 + 0.3 * rng.random(mesh.nfaces))
        self.src = _smooth(cc, rng)
        self.si = 20.0 + rng.random(mesh.ncells)
        self.inlet = float(rng.uniform(0.5, 1.5))

    def solve(self):
        m = self.mesh
        n, nb = m.ncells, m.nbfaces
        own = m.face_owner.reshape(-1, 2) - 1
        a, c = own[nb:, 0], own[nb:, 1]
        cond = self.gamma[nb:] * m.face_area[nb:] / m.face_delta[nb:]
        # outward flux of each side: the sign of the face in the cell's list
        cell = np.repeat(np.arange(n), np.diff(m.cell_faces_ptr))
        face = m.cell_faces - 1
        sign = np.zeros((m.nfaces, 2))
        first = own[face, 0] == cell
        sign[face[first], 0] = m.cell_nsign[first]
        sign[face[~first], 1] = m.cell_nsign[~first]
        A = torch.zeros((n, n), dtype=torch.float64)
        Av = A.numpy()
        diag = self.si * m.cell_volume
        b = self.src * m.cell_volume
        for side, (i, j) in enumerate(((a, c), (c, a))):
            out = self.flux[nb:] * sign[nb:, side]
            np.add.at(diag, i, np.maximum(out, 0.0) + cond)
            np.add.at(Av, (i, j), -np.maximum(-out, 0.0) - cond)
        value = {"inlet": self.inlet, "wall": 0.0}
        bface = np.zeros(nb)
        fixed = np.zeros(nb, dtype=bool)
        for name, faces, cells in m.boundaries:
            f, i = faces - 1, cells - 1
            if name in value:
                g = self.gamma[f] * m.face_area[f] / m.face_delta[f]
                np.add.at(diag, i, g)
                np.add.at(b, i, (g - self.flux[f]) * value[name])
                bface[f], fixed[f] = value[name], True
            else:
                np.add.at(diag, i, np.maximum(self.flux[f], 0.0))
        Av[np.arange(n), np.arange(n)] = diag
        rows = np.concatenate([a, c, np.arange(n)])
        cols = np.concatenate([c, a, np.arange(n)])
        at = np.unique(rows.astype(np.int64) * n + cols)
        vals = Av.reshape(-1)[at]
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        x = torch.linalg.solve(A.to(dev), torch.from_numpy(b).to(dev)).cpu().numpy()
        # Green-Gauss gradient of x with the interpolation weight of the mesh
        w = m.face_weight[nb:]
        xf = np.empty(m.nfaces)
        xf[nb:] = w * x[a] + (1.0 - w) * x[c]
        xf[:nb] = np.where(fixed, bface, x[own[:nb, 0]])
        S = m.face_normal.reshape(-1, 3) * m.face_area[:, None]
        g = np.zeros((3, n))
        for d in range(3):
            np.add.at(g[d], cell, xf[face] * S[face, d] * m.cell_nsign)
            np.add.at(g[d], own[:nb, 0], xf[:nb] * S[:nb, d])
        return {"A": vals, "b": b, "x": x, "grad": g / m.cell_volume}
