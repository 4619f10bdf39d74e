"""The work a program built on yafel_b200 has it do, as cases to be timed and checked.

Every case is one of seven kinds of call sequence, all through the public
classes (FESystem, CGAssembly, DirichletBC, the preconditioners, solve, Batch):

analysis   a linear analysis on a numbered mesh: assemble the tangent and the
           load, Dirichlet conditions, Jacobi preconditioner, PCG to a 1e-10
           relative residual (FP64 or mixed precision), the solution downloaded.
newton     one residual evaluation of a parameter study or Newton loop: the
           tangent and load re-assembled with the pass's material, then
           r = F - K u, downloaded.
inexact    one inexact-Newton (or time) step: re-assembly, Dirichlet conditions
           and a fixed, short number of PCG iterations from the last state.
explicit   a march of explicit steps x -= dt K x with the operator kept.
ilu        an analysis preconditioned with ILU(0), factorisation included.
advection  SUPG advection-diffusion solved by BiCGSTAB with Jacobi.
batch      many 2D systems of different sizes solved together, FP64 or mixed.

The listed sizes are those of the repository's benchmark (64 x 64 Q1 Poisson,
Q2/Q3 hexahedral elasticity cubes, seeded batches of 2D problems, SUPG with
Peclet numbers 1-100) and smaller and larger relatives of them.  Results leave
the device the way a program takes them: DeviceVector.numpy().
"""
import math
import random

import numpy as np
import torch

import yafel_b200 as yb
from yafel_b200 import meshgen, workloads

TOL = 1e-10


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the smallest analysis of the benchmark: 4,225 dofs, launches and latency
        {"name": "poisson2d_q1_64", "kind": "analysis", "phys": "poisson", "dim": 2, "p": 1, "n": 64, "prec": "fp64"},
        # an everyday plane-elasticity mesh of triangles and quadrilaterals (2x2 blocks)
        {"name": "elast2d_p2_mixed_mesh", "kind": "analysis", "phys": "elasticity", "dim": 2, "p": 2, "n": 61,
         "prec": "fp64", "jitter": True},
        # a mid-size solid: matrix a little over L2
        {"name": "elast3d_q2_15", "kind": "analysis", "phys": "elasticity", "dim": 3, "p": 2, "n": 15, "prec": "fp64"},
        # a large solid, HBM bound, FP64: the headline workload at a third of its dofs
        {"name": "elast3d_q2_40", "kind": "analysis", "phys": "elasticity", "dim": 3, "p": 2, "n": 40, "prec": "fp64"},
        # mixed precision, order 3 (rows of up to 343 blocks)
        {"name": "elast3d_q3_14_mixed", "kind": "analysis", "phys": "elasticity", "dim": 3, "p": 3, "n": 14,
         "prec": "mixed"},
        # the Newton-loop side: assembly of a large solid and of a scalar field in CSR
        {"name": "newton_elast3d_q2_33", "kind": "newton", "phys": "elasticity", "dim": 3, "p": 2, "n": 33},
        {"name": "newton_poisson3d_q2_37", "kind": "newton", "phys": "poisson", "dim": 3, "p": 2, "n": 37},
        # a time step on a trilinear mesh: assembly, conditions and 24 iterations
        {"name": "inexact_elast3d_q1_48", "kind": "inexact", "phys": "elasticity", "dim": 3, "p": 1, "n": 48, "its": 24},
        # 32 explicit steps of 3D heat conduction with the CSR operator
        {"name": "explicit_poisson3d_q2_48", "kind": "explicit", "phys": "poisson", "dim": 3, "p": 2, "n": 48,
         "steps": 32, "prec": "fp64"},
        # ILU(0)-PCG on a small solid: dependency levels
        {"name": "ilu_elast3d_q2_7", "kind": "ilu", "phys": "elasticity", "dim": 3, "p": 2, "n": 7},
        # a served advection-diffusion request
        {"name": "supg3d_q2_25", "kind": "advection", "phys": "supg", "dim": 3, "p": 2, "n": 25, "peclet": 8.0},
        # a batch of seeded 2D problems, 1e3-4e4 dofs, orders 1-3
        {"name": "batch_2d_24", "kind": "batch", "count": 24, "lo": 1000.0, "hi": 40000.0, "prec": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, then a size spread over the logarithm of its range."""
    kind = rng.choice(["analysis", "analysis", "analysis", "newton", "newton", "inexact", "explicit", "ilu",
                       "advection", "batch"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 24), "lo": 1000.0,
                "hi": float(_log_int(rng, 4000, 40000)), "prec": prec}
    if kind == "advection":
        dim = rng.choice([2, 3])
        p = rng.choice([1, 2])
        n = _log_int(rng, 20, 220 // p) if dim == 2 else _log_int(rng, 6, 50 // p)
        return {"kind": kind, "phys": "supg", "dim": dim, "p": p, "n": n, "peclet": math.exp(rng.uniform(0.0, math.log(100.0)))}
    if kind == "ilu":
        phys = rng.choice(["poisson", "elasticity"])
        dim = rng.choice([2, 3])
        p = rng.choice([1, 2])
        n = _log_int(rng, 8, 24 // p) if dim == 2 else _log_int(rng, 4, 14 // p)
        return {"kind": kind, "phys": phys, "dim": dim, "p": p, "n": n}
    phys = rng.choice(["poisson", "elasticity"])
    dim = rng.choice([2, 3, 3])
    p = rng.choice([1, 2, 2, 3])
    # cells per side: 2D 16..500/p, 3D up to the sizes of the listed cases
    if dim == 2:
        n = _log_int(rng, 12, 500 // p if kind != "analysis" else 250 // p)
    else:
        n = _log_int(rng, 4, {1: 60, 2: 32, 3: 14}[p])
    c = {"kind": kind, "phys": phys, "dim": dim, "p": p, "n": n}
    if kind == "analysis":
        c["prec"] = prec
        c["jitter"] = dim == 2 and n <= 120 and rng.random() < 0.5
    elif kind == "inexact":
        c["its"] = rng.randint(10, 40)
    elif kind == "explicit":
        c["steps"] = rng.randint(8, 32)
        c["prec"] = prec
    return c


# ------------------------------------------------------------------ states and passes

def _dpn(case):
    return case["dim"] if case["phys"] == "elasticity" else 1


def _draws(case, seed):
    """What the seed decides: the material, the loads and the current state."""
    rng = np.random.Generator(np.random.PCG64(seed))
    m = {"E": float(rng.uniform(0.8, 1.2)), "nu": float(rng.uniform(0.25, 0.35)),
         "f": float(rng.uniform(0.5, 1.5)), "body": tuple(float(v) for v in rng.uniform(-1.0, 1.0, 3))}
    dofs = _dpn(case) * (case["p"] * case["n"] + 1) ** case["dim"]
    return rng, m, dofs


def _physics(case, m):
    dim = case["dim"]
    if case["phys"] == "poisson":
        return yb.PoissonEquation(dim, f=m["f"])
    if case["phys"] == "elasticity":
        return yb.LinearElasticity(dim, E=m["E"], nu=m["nu"], body=m["body"][:dim])
    h = 1.0 / case["n"]
    return yb.AdvectionDiffusionSUPG(dim, k=h / (2.0 * case["peclet"]), h=h, U0=1.0, Q=m["f"])


def _jittered(n, p, seed):
    """Quadrilaterals and triangle pairs; quadrilaterals alone at order 3, where the
    number of merged nodes depends on which cells are split."""
    return meshgen.jittered_mixed(n, n, seed=seed, tri_fraction=0.5 if p < 3 else 0.0, order=meshgen.corner_order(p))


def _load(rng, case, dofs):
    """Nodal loads beside the body force: i.i.d., of the size of a cell's share."""
    return rng.standard_normal(dofs) / case["n"] ** case["dim"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    rng, m, dofs = _draws(case, seed)
    dim, p, n, dpn = case["dim"], case["p"], case["n"], _dpn(case)
    if case.get("jitter"):
        mesh = _jittered(n, p, seed)
        dm = yb.DoFManager(mesh, p, dpn)
    else:
        dm = yb.DoFManager.box(dim, (n,) * dim, polyOrder=p, dof_per_node=dpn)
    fe = yb.FESystem(dm, dim, format=yb.CSR if dpn == 1 else yb.BCSR)
    s = {"case": case, "fe": fe, "phys": _physics(case, m)}
    # the first assembly of a dofmap builds its pattern, which a program keeps
    yb.CGAssembly(s["phys"], fe, [yb.AssemblyRequirement.Tangent])
    if kind in ("analysis", "inexact", "ilu", "advection"):
        bcs = [yb.DirichletBC(dm, 0.0, c) for c in range(dpn)]
        for bc in bcs:
            bc.selectByFunction(lambda X: np.abs(X[:, 0]) < 1e-9)
        s["bcs"] = bcs
        s["load"] = yb.DeviceVector(_load(rng, case, dm.ndofs))
    if kind in ("newton", "explicit"):
        s["u0"] = yb.DeviceVector(rng.standard_normal(dm.ndofs))
        s["y"] = yb.DeviceVector(dm.ndofs)
    if kind == "explicit":
        s["x"] = yb.DeviceVector(dm.ndofs)
        if case["prec"] == "mixed":
            fe.getGlobalTangent().make_fp32()
    if kind == "advection":
        _assemble_and_constrain(s)
        s["M"] = yb.JacobiPreconditioner(fe.getGlobalTangent())
    return s


def _assemble_and_constrain(s):
    fe = s["fe"]
    F = fe.getGlobalResidual()
    F.fill(0.0)
    yb.CGAssembly(s["phys"], fe)
    F.axpy(1.0, s["load"])
    for bc in s["bcs"]:
        bc.apply(fe.getGlobalTangent(), F)
    return fe.getGlobalTangent(), F


_PREC = {"fp64": yb.PREC_FP64, "mixed": yb.PREC_MIXED}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "batch":
        return _run_batch(s)
    fe = s["fe"]
    if kind == "analysis":
        K, F = _assemble_and_constrain(s)
        x, _ = yb.solve(K, F, M=yb.JacobiPreconditioner(K), tol=TOL, precision=_PREC[case["prec"]])
        return x.numpy()
    if kind == "ilu":
        K, F = _assemble_and_constrain(s)
        x, _ = yb.solve(K, F, M=yb.ILUPreconditioner(K), tol=TOL)
        return x.numpy()
    if kind == "inexact":
        K, F = _assemble_and_constrain(s)
        x, _ = yb.solve(K, F, M=yb.JacobiPreconditioner(K), tol=1e-30, maxiter=case["its"])
        return x.numpy()
    if kind == "advection":
        x, _ = yb.solve(fe.getGlobalTangent(), fe.getGlobalResidual(), M=s["M"], method="bicgstab", tol=TOL)
        return x.numpy()
    if kind == "newton":
        F = fe.getGlobalResidual()
        F.fill(0.0)
        yb.CGAssembly(s["phys"], fe)
        F.axpy(-1.0, fe.getGlobalTangent().spmv(s["u0"], s["y"]))
        return F.numpy()
    # explicit: x -= dt K x from the state u0
    K, x, y = fe.getGlobalTangent(), s["x"], s["y"]
    x.fill(0.0)
    x.axpy(1.0, s["u0"])
    prec = yb.SPMV_MIXED_CORRECTED if case["prec"] == "mixed" else yb.PREC_FP64
    for _ in range(case["steps"]):
        K.spmv(x, y, prec)
        x.axpy(-_dt(case), y)
    return x.numpy()


def _dt(case):
    """A stable explicit step: the element matrices scale with h^(dim-2)."""
    return 0.02 * case["n"] ** (case["dim"] - 2) / case["p"] ** 2


def _prepare_batch(case, seed):
    r = random.Random(seed)
    base = r.randrange(1 << 30)
    ctx = yb.default_context()
    batch = yb.Batch(case["count"])
    s = {"case": case, "batch": batch, "x": []}
    for i in range(case["count"]):
        # sizes at the case's quantiles, so that every seed asks for the same work
        # in another order of problems; meshes, loads and orders are the seed's
        t = case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / case["count"])
        p, kind = 1 + i % 3, ("poisson", "elasticity")[(i // 3) % 2]
        dpn = 2 if kind == "elasticity" else 1
        n = workloads.grid_for_dofs(t, p, dpn)
        spec = {"index": i, "seed": base + i, "order": p, "kind": kind, "dim": 2, "dpn": dpn, "n": n}
        _, K, b, _ = workloads.assemble(spec, ctx, _jittered(n, p, base + i))
        x = yb.DeviceVector(K.rows())
        batch.add(K, b, x, tol=TOL, precision=_PREC[case["prec"]])
        s["x"].append(x)
    batch.tune()
    return s


def _run_batch(s):
    for x in s["x"]:
        x.fill(0.0)
    s["batch"].reset()
    s["batch"].run()
    return [x.numpy() for x in s["x"]]


# ------------------------------------------------------------------ what a pass cannot do without

def _sizes(case):
    """dofs, node pairs of the pattern, block size and cells of a structured case."""
    dim, p, n, B = case["dim"], case["p"], case["n"], _dpn(case)
    nodes = (p * n + 1) ** dim
    # a node couples to the nodes of its cells: per direction, corner nodes of two
    # cells see 2p+1 nodes (p+1 at the ends), inner nodes p+1
    pairs = (n * (p - 1) * (p + 1) + (n - 1) * (2 * p + 1) + 2 * (p + 1)) ** dim
    return nodes * B, pairs, B, n ** dim


def _spmv_bytes(case, val=8):
    dofs, pairs, B, _ = _sizes(case)
    return pairs * (val * B * B + 4) + 4 * (dofs // B + 1) + 16 * dofs


def _iterations(case):
    """Krylov iterations these systems take to 1e-10 with Jacobi (ILU(0): the ILU count)."""
    side = case["p"] * case["n"]
    if case["kind"] == "advection":
        return 2 * side + 10
    per = {"poisson": 4.2 if case["dim"] == 2 else 6.0, "elasticity": 15.5 if case["dim"] == 2 else 18.7}[case["phys"]]
    return int(per * side * (0.2 if case["kind"] == "ilu" else 1.3 if case["p"] == 3 and case["dim"] == 3 else 1.0))


def work(case):
    if case["kind"] == "batch":
        total = 0.0
        flops = 0.0
        for i in range(case["count"]):
            t = case["lo"] * (case["hi"] / case["lo"]) ** ((i + 0.5) / case["count"])
            p, kind = 1 + i % 3, ("poisson", "elasticity")[(i // 3) % 2]
            c = {"kind": "analysis", "phys": kind, "dim": 2, "p": p,
                 "n": workloads.grid_for_dofs(t, p, 2 if kind == "elasticity" else 1)}
            dofs, pairs, B, _ = _sizes(c)
            total += _iterations(c) * (_spmv_bytes(c, 4 if case["prec"] == "mixed" else 8) + 72 * dofs)
            flops += _iterations(c) * (2 * pairs * B * B + 12 * dofs)
        return {"bytes": total, "flops": flops}
    dofs, pairs, B, cells = _sizes(case)
    kind = case["kind"]
    nen = (case["p"] + 1) ** case["dim"]
    # the symmetric half of sum_q w G^T G per cell; every value written once
    asm_flops = cells * nen * nen * case["dim"] * B * nen
    asm_bytes = pairs * B * B * 8 + 24 * dofs // B + 4 * nen * cells + 8 * dofs
    val = 4 if case.get("prec") == "mixed" else 8
    step = _spmv_bytes(case, val) + 72 * dofs
    if kind == "newton":
        return {"bytes": asm_bytes + _spmv_bytes(case), "flops": asm_flops + 2 * pairs * B * B}
    if kind == "explicit":
        return {"bytes": case["steps"] * (_spmv_bytes(case, val) + 24 * dofs), "flops": case["steps"] * 2 * pairs * B * B}
    its = case["its"] if kind == "inexact" else _iterations(case)
    if kind == "advection":
        return {"bytes": its * (2 * _spmv_bytes(case) + 150 * dofs), "flops": its * 4 * pairs}
    if kind == "ilu":
        step += pairs * B * B * 12
        asm_flops += 2 * pairs * B * B * nen
    return {"bytes": asm_bytes + its * step, "flops": asm_flops + its * 2 * pairs * B * B}


# ------------------------------------------------------------------ 64-bit values without the package

def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return x, w


def _lobatto(n):
    if n == 2:
        return np.array([-1.0, 1.0])
    c = np.zeros(n)
    c[-1] = 1.0
    return np.concatenate([[-1.0], np.sort(np.polynomial.legendre.Legendre(c).deriv().roots().real), [1.0]])


def _element(case, m):
    """Element matrix and load of the uniform cube's cell, nodes x fastest."""
    dim, p, n = case["dim"], case["p"], case["n"]
    t = _lobatto(p + 1)
    gx, gw = _gauss(p + 1)
    V = np.ones((gx.size, p + 1))
    D = np.zeros((gx.size, p + 1))
    for j in range(p + 1):
        o = np.delete(t, j)
        den = np.prod(t[j] - o)
        V[:, j] = np.prod(gx[:, None] - o, axis=1) / den
        for k in range(o.size):
            D[:, j] += np.prod(gx[:, None] - np.delete(o, k), axis=1) / den
    h = 1.0 / n

    def kron(fs):  # fs in z, y, x order
        out = fs[0]
        for f in fs[1:]:
            out = np.einsum("qa,rb->qrab", out, f).reshape(out.shape[0] * f.shape[0], -1)
        return out

    N = kron([V] * dim)
    G = np.stack([kron([D if dim - 1 - k == d else V for k in range(dim)]) for d in range(dim)], axis=2) * (2.0 / h)
    w = gw
    for _ in range(dim - 1):
        w = np.outer(w, gw).ravel()
    w = w * (h / 2.0) ** dim
    nen = N.shape[1]
    if case["phys"] == "poisson":
        return np.einsum("q,qad,qbd->ab", w, G, G), m["f"] * (w @ N)
    if case["phys"] == "elasticity":
        lam = m["E"] * m["nu"] / ((1 + m["nu"]) * (1 - 2 * m["nu"]))
        mu = m["E"] / (2 * (1 + m["nu"]))
        M = np.einsum("q,qai,qbk->aibk", w, G, G)
        Ke = lam * M + mu * M.transpose(0, 3, 2, 1)
        tr = np.einsum("aibi->ab", M)
        for i in range(dim):
            Ke[:, i, :, i] += mu * tr
        return Ke.reshape(nen * dim, nen * dim), np.outer(w @ N, np.array(m["body"][:dim])).ravel()
    # steady SUPG advection-diffusion as the reference states it: the advection
    # term counted once per dimension, the stabilised diffusion tensor
    k, U = (1.0 / n) / (2.0 * case["peclet"]), 1.0
    Pe = U * (1.0 / n) / (2 * k)
    alpha = np.cosh(Pe) / np.sinh(Pe) - 1.0 / Pe
    Kd = k * np.eye(dim)
    Uv = np.zeros(dim)
    Uv[0] = U
    Kd = Kd + (alpha * (1.0 / n) / (2 * U)) * np.outer(Uv, Uv)
    adv = dim * np.einsum("q,qa,qbd,d->ab", w, N, G, Uv)
    Ke = adv + np.einsum("q,qai,qbj,ij->ab", w, G, G, Kd)
    Uh = (alpha * (1.0 / n) / 2) * Uv / U
    Fe = -(dim * m["f"] * (w @ N) + np.einsum("q,qai,i->a", w, G, Uh))
    return Ke, Fe


def _cells(case):
    dim, p, n, B = case["dim"], case["p"], case["n"], _dpn(case)
    side = p * n + 1
    loc = np.arange(p + 1)
    start = p * np.arange(n)
    one = start[:, None] + loc[None, :]  # cells x local nodes along one axis
    if dim == 2:
        c = (one[:, None, :, None] * side + one[None, :, None, :]).reshape(n * n, -1)
    else:
        c = ((one[:, None, None, :, None, None] * side + one[None, :, None, None, :, None]) * side
             + one[None, None, :, None, None, :]).reshape(n ** 3, -1)
    return (c[:, :, None] * B + np.arange(B)).reshape(c.shape[0], -1)


class _Operator:
    """y = K x cell by cell in FP64 torch, on the GPU when there is one."""

    def __init__(self, case, m):
        Ke, Fe = _element(case, m)
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.Ke = torch.tensor(Ke, device=self.dev)
        self.conn = torch.tensor(_cells(case), device=self.dev)
        side = case["p"] * case["n"] + 1
        self.n = _dpn(case) * side ** case["dim"]
        self.F = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        self.F.index_add_(0, self.conn.reshape(-1), torch.tensor(Fe, device=self.dev).repeat(self.conn.shape[0]))
        self.fixed = (torch.arange(self.n, device=self.dev) // _dpn(case)) % side == 0
        self.diag = torch.zeros_like(self.F)
        self.diag.index_add_(0, self.conn.reshape(-1), self.Ke.diagonal().repeat(self.conn.shape[0]))

    def __call__(self, x, constrained=True):
        v = torch.where(self.fixed, 0.0, x) if constrained else x
        y = torch.zeros_like(x)
        y.index_add_(0, self.conn.reshape(-1), (v[self.conn] @ self.Ke.T).reshape(-1))
        return torch.where(self.fixed, x, y) if constrained else y


def _pcg(A, b, its, tol):
    d = 1.0 / torch.where(A.fixed, 1.0, A.diag)
    x = torch.zeros_like(b)
    r = b.clone()
    p = d * r
    rz = torch.dot(r, p)
    nb = float(b.norm())
    for k in range(its):
        q = A(p)
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        z = d * r
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
        if tol and k % 10 == 9 and float(r.norm()) <= tol * nb:
            break
    return x


def _solve(A, b):
    """FP64 solution refined by restarts from the true residual."""
    x = torch.zeros_like(b)
    for _ in range(2):
        x = x + _pcg(A, b - A(x), 4000, 1e-9)
    return x


def _bicgstab(A, b):
    d = 1.0 / torch.where(A.fixed, 1.0, A.diag)
    x = torch.zeros_like(b)
    nb = float(b.norm())
    for _ in range(6):
        r = b - A(x)
        if float(r.norm()) <= 1e-14 * nb:
            break
        target = max(1e-15 * nb, 1e-8 * float(r.norm()))
        r0, p = r.clone(), r.clone()
        rho = torch.dot(r0, r)
        for _ in range(2000):
            ph = d * p
            v = A(ph)
            a = rho / torch.dot(r0, v)
            s = r - a * v
            sh = d * s
            t = A(sh)
            om = torch.dot(t, s) / torch.dot(t, t)
            x = x + a * ph + om * sh
            r = s - om * t
            if float(r.norm()) <= target:
                break
            new = torch.dot(r0, r)
            p = r + (new / rho) * (a / om) * (p - om * v)
            rho = new
    return x


def exact(case, seed):
    """The same outputs in 64 bits, for the structured meshes."""
    if case["kind"] == "batch" or case.get("jitter"):
        return None
    rng, m, dofs = _draws(case, seed)
    A = _Operator(case, m)
    kind = case["kind"]
    if kind in ("newton", "explicit"):
        u = torch.tensor(rng.standard_normal(dofs), device=A.dev)
        if kind == "newton":
            return (A.F - A(u, False)).cpu().numpy()
        for _ in range(case["steps"]):
            u = u - _dt(case) * A(u, False)
        return u.cpu().numpy()
    b = A.F + torch.tensor(_load(rng, case, dofs), device=A.dev)
    b[A.fixed] = 0.0
    if kind == "advection":
        return _bicgstab(A, b).cpu().numpy()
    if kind == "inexact":
        return _pcg(A, b, case["its"], 0.0).cpu().numpy()
    return _solve(A, b).cpu().numpy()
