"""What a program built on this library spends its GPU time in, as timed cases.

Each case is one pass through the public Python entry points (the ctypes
mirror of the C ABI) on seeded synthetic systems: the solves of a SIMPLE /
PISO run (pressure PCG, momentum BiCGSTAB on three right-hand sides, energy
through host buffers), the solverC drop-in, batches of uneven systems, the
differentiable solve, and the device assembly with the gradients it reads.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges,
``prepare`` what a program holds before the call, ``run`` the call,
``work`` its unavoidable bytes and flops, ``exact`` the 64-bit value of what
``run`` returns, from plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sfr3d_b200 import adjoint, assembly, solver, systems

# Solves of the nearly singular diffusion systems go to 1e-12 (the adjoint's
# default): the solution is then known to about 1e-11, whatever the order of a
# sum.  The diagonally dominant momentum and energy systems go to 1e-10.
POISSON_TOL, MOMENTUM_TOL = 1e-12, 1e-10
MAXIT = 10000


def listed():
    return [
        # The smallest call: a coarse pressure system, a few hundred short
        # iterations, all latency.
        {"name": "pcg-16", "kind": "pcg", "nx": 16, "ny": 16, "nz": 16, "precision": "fp64",
         "call": "device"},
        # The drop-in as the reference's own cavity example calls it: 64,000
        # cells, symmetric CSRC, everything in host memory, values uploaded
        # on each call.
        {"name": "solverc-cavity-40", "kind": "pcg", "nx": 40, "ny": 40, "nz": 40,
         "precision": "fp64", "call": "solverC"},
        # The headline: FP64 pressure correction on 128^3 cells.
        {"name": "pcg-128", "kind": "pcg", "nx": 128, "ny": 128, "nz": 128, "precision": "fp64",
         "call": "device"},
        # Mixed-precision pressure correction, an ordinary box.
        {"name": "pcg-mixed-80x72x96", "kind": "pcg", "nx": 80, "ny": 72, "nz": 96,
         "precision": "mixed", "call": "device"},
        # u, v, w in one call, FP64, ragged edges.
        {"name": "momentum-61x47x53", "kind": "momentum", "nx": 61, "ny": 47, "nz": 53,
         "peclet": 50.0, "precision": "fp64"},
        # The largest momentum solve: mixed, 128^3, three right-hand sides.
        {"name": "momentum-mixed-128", "kind": "momentum", "nx": 128, "ny": 128, "nz": 128,
         "peclet": 50.0, "precision": "mixed"},
        # Energy (or a species) assembled on the host: new ELLPACK values and
        # one right-hand side from host buffers on each outer iteration.
        {"name": "energy-ell-48x40x51", "kind": "energy", "nx": 48, "ny": 40, "nz": 51,
         "peclet": 20.0},
        # Many small independent boxes, FP64, one launch.
        {"name": "batch-24", "kind": "batch", "count": 24, "nmin": 8, "nmax": 48, "shapes": 11,
         "precision": "fp64"},
        # The uneven batch of 64 boxes of 8 to 96 cells an edge, mixed.
        {"name": "batch-mixed-64", "kind": "batch", "count": 64, "nmin": 8, "nmax": 96,
         "shapes": 4, "precision": "mixed"},
        # Training through the solve: forward and backward of the autograd
        # function, gradients of every coefficient and of b.
        {"name": "adjoint-48", "kind": "adjoint", "nx": 48, "ny": 48, "nz": 48, "peclet": 20.0},
        # One outer iteration's assembly, resident: both gradients, momentum,
        # pressure correction and diffusion, and the products A u of explicit
        # residual checks.
        {"name": "assembly-96x88x101", "kind": "assembly", "nx": 96, "ny": 88, "nz": 101},
        # A whole SIMPLE iteration, resident, on an ordinary cavity mesh.
        {"name": "simple-56x60x52", "kind": "simple", "nx": 56, "ny": 60, "nz": 52},
    ]


def _edges(rng, lo, hi):
    """A box whose edges spread around one log-uniform length in [lo, hi]."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return {a: max(lo, min(hi, round(n * math.exp(rng.uniform(-0.25, 0.25)))))
            for a in ("nx", "ny", "nz")}


def draw(rng):
    kind = rng.choice(["pcg", "pcg", "pcg", "momentum", "momentum", "energy", "batch",
                       "adjoint", "assembly", "simple"])
    if kind == "pcg":
        call = rng.choice(["device", "device", "solverC"])
        return {"kind": kind, **_edges(rng, 12, 80 if call == "solverC" else 128),
                "precision": "fp64" if call == "solverC" else rng.choice(["fp64", "mixed"]),
                "call": call}
    if kind == "momentum":
        return {"kind": kind, **_edges(rng, 12, 128), "peclet": rng.choice([20.0, 50.0]),
                "precision": rng.choice(["fp64", "mixed"])}
    if kind == "batch":
        # mixed batches reach from small boxes to the 96-cell ones
        precision = rng.choice(["fp64", "mixed"])
        return {"kind": kind, "count": rng.randint(8, 64), "nmin": 8,
                "nmax": rng.randint(24, 96 if precision == "mixed" else 64),
                "shapes": rng.randint(1, 10**6), "precision": precision}
    if kind in ("energy", "adjoint"):
        return {"kind": kind, **_edges(rng, 12, 72), "peclet": rng.choice([20.0, 50.0])}
    return {"kind": kind, **_edges(rng, 16, 104 if kind == "assembly" else 80)}


# ------------------------------------------------------------- the systems --

def _poisson(case, seed):
    """Pressure-correction system: jittered hexahedra, cell diffusivity over
    four decades, permuted then RCM-numbered, right-hand side U[-1, 1]."""
    return systems.build(systems.params(n=(case["nx"], case["ny"], case["nz"]), jitter=0.2,
                                        log10k=(-2.0, 2.0), permute=True, seed=seed))


def _convection(case, seed, nrhs):
    """Upwind convection-diffusion in the divergence-free vortex field, one
    implicit time step, right-hand sides N(0, 1)."""
    return systems.build(systems.params(
        kind=systems.SFR_SYS_CONVDIFF, n=(case["nx"], case["ny"], case["nz"]),
        lengths=(math.pi,) * 3, dirichlet=systems.ALL_FACES, nrhs=nrhs, rhs_normal=True,
        peclet=case["peclet"], nu=1e-3, dt=1e-2, seed=seed))


def _boxes(case, seed):
    """The batch's boxes: shapes from the case, coefficients' seeds from
    ``seed``."""
    out = []
    rng = np.random.default_rng(seed)
    for p in systems.batch_params(case["count"], case["nmin"], case["nmax"], case["shapes"]):
        p.seed = int(rng.integers(1 << 31))
        p.log10k_lo = p.log10k_hi = rng.uniform(-1.0, 1.0)
        out.append(systems.build(p))
    return out


LID, WALL = 1, 2  # load numbers: the moving lid (z max), the static walls
VEL_SIDES, PRES_SIDES = [WALL] * 5 + [LID], [1, 0, 0, 0, 0, 0]


def _cavity(case, seed):
    """A lid-driven cavity's mesh and fields (numpy): static walls, the z-max
    lid moving, the pressure fixed on x = 0."""
    s = _poisson(case, seed)
    m = s.mesh()
    rng = np.random.default_rng(seed)
    n = m.numel
    return s, m, {
        "cc": m.xm[m.cellface[:, 0] - 1] - m.xmcc[:, 0, :],
        "prop": np.array([[1e-3, 1.0] + [0.0] * 8]),
        "pres": rng.standard_normal(n) * 1e-2, "vel": rng.standard_normal((n, 3)) * 0.1,
        "u0": rng.standard_normal(n), "dfield": rng.uniform(0.5, 1.0, (n, 3)),
    }


def _loads():
    return ([assembly.Load(assembly.MOVEWALL, (1.0, 0.0, 0.0, 0.0)),
             assembly.Load(assembly.STATICWALL, ())],
            [assembly.Load(assembly.DIRICHLET, (0.0,))])


def _gpu(a):
    return torch.from_numpy(np.array(a, dtype=np.float64, order="C")).cuda()


def _precision(case):
    return solver.MIXED if case["precision"] == "mixed" else solver.FP64


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "stream": torch.cuda.Stream()}
    if kind == "pcg":
        s = _poisson(case, seed)
        st["precision"], st["call"] = _precision(case), case["call"]
        if case["call"] == "solverC":
            ia, ja, a = s.csrc()
            st.update(neq=s.neq, ia=ia, ja=ja, al=a[:len(ja)].copy(), ad=s.ad, b=s.b[0])
            return st
        g = solver.GpuSystem(s.neq, s.ia, s.ja, solver.CSRD, True)
        g.set_values(s.al, s.ad)
        st.update(g=g, b=_gpu(s.b[0]), x=_gpu(np.zeros(s.neq)))
    elif kind == "momentum":
        s = _convection(case, seed, 3)
        g = solver.GpuSystem(s.neq, s.ia, s.ja, solver.CSRD, True)
        g.set_values(s.al, s.ad)
        st.update(g=g, b=_gpu(s.b), x=_gpu(np.zeros((3, s.neq))), precision=_precision(case))
    elif kind == "energy":
        s = _convection(case, seed, 1)
        ja, a = s.ell()
        ia = np.array([s.width, s.neq * s.width], np.int32)
        st.update(g=solver.GpuSystem(s.neq, ia, ja, solver.ELLPACK, True), a=a, ad=s.ad,
                  b=s.b[0])
    elif kind == "batch":
        boxes = _boxes(case, seed)
        g = solver.GpuBatch([(s.neq, s.ia, s.ja) for s in boxes], solver.CSRD, True)
        g.set_values([s.al for s in boxes], [s.ad for s in boxes])
        st.update(g=g, b=[s.b[0] for s in boxes], precision=_precision(case))
    elif kind == "adjoint":
        s = _convection(case, seed, 1)
        w = np.random.default_rng(seed).standard_normal(s.neq)
        st.update(g=solver.GpuSystem(s.neq, s.ia, s.ja, solver.CSRD, True), w=_gpu(w),
                  leaves=[_gpu(v).requires_grad_() for v in (s.al, s.ad, s.b[0])])
    else:
        s, m, f = _cavity(case, seed)
        st["prop"] = f["prop"]
        for k in ("pres", "vel", "u0", "dfield"):
            st[k] = _gpu(f[k])
        st["cdiff"] = _gpu(m.cdiff)
        st["gradvel"] = _gpu(np.zeros((m.numel, 3, 3)))
        st["gradpres"] = _gpu(np.zeros((m.numel, 3)))
        fv, fp = m.face_r(VEL_SIDES), m.face_r(PRES_SIDES)
        system = lambda: solver.GpuSystem(s.neq, s.ia, s.ja, solver.CSRD, True)  # noqa: E731
        st.update(gvel=assembly.GradPlan(m, fv), gpres=assembly.GradPlan(m, fp),
                  av=system(), ap=system())
        st.update(vplan=assembly.VelPlan(st["av"], m, fv, f["cc"]),
                  pplan=assembly.PresPlan(st["ap"], m, fp, fv))
        new = lambda k: _gpu(np.zeros(k))  # noqa: E731
        n = s.neq
        st.update(ad3=new(3 * n), b3=new(3 * n), bp=new(n), rcell3=new(3 * n), rcellp=new(n))
        if kind == "assembly":
            st["ad_"] = system()
            st["dplan"] = assembly.DifPlan(st["ad_"], m, fp)
            st.update(bd=new(n), rcelld=new(n), yv=new(n), yp=new(n), yd=new(n))
        else:
            st.update(x3=new(3 * n), xp=new(n))
    return st


def _assemble(st, residual):
    """Gradients, momentum and pressure correction of one SIMPLE iteration."""
    sp = st["stream"].cuda_stream
    p = {k: v.data_ptr() for k, v in st.items() if isinstance(v, torch.Tensor)}
    lvel, lpres = _loads()
    st["gvel"].grad_device(lvel, st["prop"], 3, p["vel"], p["gradvel"], sp)
    st["gpres"].grad_device(lpres, st["prop"], 1, p["pres"], p["gradpres"], sp)
    st["vplan"].assemble_device(lvel, st["prop"], p["pres"], p["gradpres"], p["vel"],
                                p["gradvel"], p["dfield"], d_ad3=p["ad3"], d_b3=p["b3"],
                                d_rcell3=p["rcell3"], fres=residual, time=(0, 1e-2, 1e-2),
                                stream=sp)
    return p, lvel, lpres, sp


def _pressure(st, p, lvel, lpres, sp):
    st["pplan"].assemble_device(lvel, lpres, st["prop"], p["pres"], p["gradpres"], p["vel"],
                                p["dfield"], d_b=p["bp"], d_rcell=p["rcellp"], stream=sp)


def run(st):
    kind, sp = st["kind"], st["stream"].cuda_stream
    if kind == "pcg" and st["call"] == "solverC":
        x = np.zeros(st["neq"])
        rc = solver.solverC(st["neq"], st["neq"], len(st["ja"]), 0, st["ia"], st["ja"], st["al"],
                            st["ad"], None, st["b"], x, POISSON_TOL, MAXIT, solver.CSRC,
                            solver.PCG, newX=True, unSym=False, name="pressure")
        if rc != solver.OK:
            raise RuntimeError(f"solverC: {rc}")
        return x
    if kind == "pcg":
        st["g"].solve_device(solver.PCG, st["b"].data_ptr(), st["x"].data_ptr(), tol=POISSON_TOL,
                             maxit=MAXIT, precision=st["precision"], stream=sp)
        return st["x"]
    if kind == "momentum":
        st["g"].solve_multi_device(solver.PBICGSTAB, 3, st["b"].data_ptr(), st["x"].data_ptr(),
                                   tol=MOMENTUM_TOL, maxit=MAXIT, precision=st["precision"],
                                   stream=sp)
        return st["x"]
    if kind == "energy":
        st["g"].set_values(st["a"], st["ad"])
        return st["g"].solve(solver.PBICGSTAB, st["b"], tol=MOMENTUM_TOL, maxit=MAXIT)[0]
    if kind == "batch":
        # the mixed batch to 1e-10, as its refinement is specified
        tol = POISSON_TOL if st["precision"] == solver.FP64 else 1e-10
        xs, _ = st["g"].solve(solver.PCG, st["b"], tol=tol, maxit=MAXIT,
                              precision=st["precision"])
        return np.concatenate(xs)
    if kind == "adjoint":
        al, ad, b = st["leaves"]
        x = adjoint.linear_solve(st["g"], al, ad, b)
        return [x.detach(), *torch.autograd.grad((st["w"] * x).sum(), st["leaves"])]
    if kind == "assembly":
        p, lvel, lpres, sp = _assemble(st, True)
        _pressure(st, p, lvel, lpres, sp)
        st["dplan"].assemble_device(lpres, p["u0"], p["cdiff"], d_b=p["bd"],
                                    d_rcell=p["rcelld"], stream=sp)
        for g, y in (("av", "yv"), ("ap", "yp"), ("ad_", "yd")):
            st[g].spmv(p["u0"], p[y], stream=sp)
        return [st[k] for k in ("gradvel", "gradpres", "ad3", "b3", "rcell3", "dfield", "bp",
                                "rcellp", "bd", "rcelld", "yv", "yp", "yd")]
    p, lvel, lpres, sp = _assemble(st, False)
    st["av"].solve_multi_device(solver.PBICGSTAB, 3, p["b3"], p["x3"], d_ad_k=p["ad3"],
                                tol=MOMENTUM_TOL, maxit=MAXIT, stream=sp)
    _pressure(st, p, lvel, lpres, sp)
    st["ap"].solve_device(solver.PCG, p["bp"], p["xp"], tol=POISSON_TOL, maxit=MAXIT, stream=sp)
    return [st[k] for k in ("gradvel", "gradpres", "ad3", "b3", "dfield", "bp", "x3", "xp")]


# ------------------------------------------------------------------- work --

def work(case):
    """Inputs read once and outputs written once; flops of the iterations the
    method takes on these systems (Jacobi-PCG: about 17 an edge cell of the
    box to 1e-12; BiCGSTAB: about 0.12 an edge cell, 3 at least)."""
    kind = case["kind"]
    if kind == "batch":
        n = iters_n = 0
        for p in systems.batch_params(case["count"], case["nmin"], case["nmax"],
                                      case["shapes"]):
            rows = p.nx * p.ny * p.nz
            n += rows
            iters_n += 17 * rows ** (1 / 3) * rows
        return {"bytes": n * (6 * 12 + 8 * 3), "flops": iters_n * (13 + 12)}
    n = case["nx"] * case["ny"] * case["nz"]
    edge = n ** (1 / 3)
    matrix = n * (6 * 12 + 8)
    if kind == "pcg":
        offdiag = n * 3 * 12 if case["call"] == "solverC" else n * 6 * 12
        return {"bytes": offdiag + 8 * 3 * n, "flops": 17 * edge * n * (13 + 12)}
    its = max(3.0, 0.12 * edge)
    if kind == "momentum":
        return {"bytes": matrix + 3 * 16 * n, "flops": 3 * its * n * (26 + 24)}
    if kind == "energy":
        return {"bytes": matrix + 16 * n, "flops": its * n * (26 + 24)}
    if kind == "adjoint":
        return {"bytes": 2 * matrix + 8 * 5 * n + 6 * 8 * n, "flops": 3 * its * n * (26 + 24)}
    # the mesh (per face: neighbour, centre, vectors, areas), the cell fields,
    # the gradients, the systems written
    mesh = n * (6 * (4 + 8 + 24) + 8) + 3 * n * (3 * 24 + 3 * 8 + 8)
    fields = n * 8 * (1 + 3 + 12 + 3)
    systems_out = n * 8 * ((6 + 3 + 3 + 3) + (6 + 1 + 2))
    if kind == "assembly":
        return {"bytes": mesh + fields + systems_out + n * 8 * (1 + 1 + 9) + 3 * (matrix + 16 * n),
                "flops": n * 1500}
    return {"bytes": mesh + fields + systems_out + n * 8 * 4,
            "flops": n * 1200 + 17 * edge * n * 25 + 3 * its * n * 50}


# ------------------------------------------------------------------ exact --

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev())


def _csr(n, rows, cols, vals, diag):
    d = torch.arange(n, device=vals.device)
    ij = torch.stack([torch.cat([d, rows]), torch.cat([d, cols])])
    return torch.sparse_coo_tensor(ij, torch.cat([diag, vals]), (n, n)).coalesce().to_sparse_csr()


def _system(s, transpose=False):
    rows = torch.repeat_interleave(torch.arange(s.neq, device=_dev()),
                                   _t(np.diff(s.ia.astype(np.int64))))
    cols = _t(s.ja.astype(np.int64))
    if transpose:
        rows, cols = cols, rows
    return _csr(s.neq, rows, cols, _t(s.al), _t(s.ad))


def _cg(A, m, r, rtol):
    """Jacobi-PCG on A d = r from zero."""
    d, z = torch.zeros_like(r), m * r
    p, rz = z.clone(), torch.dot(r, z)
    stop = rz * rtol * rtol
    for j in range(20000):
        q = A @ p
        alpha = rz / torch.dot(p, q)
        d += alpha * p
        r = r - alpha * q
        z = m * r
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
        if j % 20 == 19 and bool(rz <= stop):
            break
    return d


def _bicgstab(A, m, r, rtol):
    """Jacobi-BiCGSTAB on A d = r from zero."""
    d, r0, p = torch.zeros_like(r), r.clone(), r.clone()
    rho, stop = torch.dot(r, r), rtol * torch.linalg.vector_norm(r)
    for _ in range(2000):
        z = m * p
        v = A @ z
        alpha = rho / torch.dot(r0, v)
        d += alpha * z
        s = r - alpha * v
        y = m * s
        t = A @ y
        omega = torch.dot(t, s) / torch.dot(t, t)
        d += omega * y
        r = s - omega * t
        if bool(torch.linalg.vector_norm(r) <= stop):
            break
        new = torch.dot(r0, r)
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return d


def _solve(A, diag, b, step):
    """A x = b with defect correction to working accuracy."""
    x, m = torch.zeros_like(b), 1.0 / diag
    for _ in range(3):
        r = b - A @ x
        if not bool((r != 0).any()):
            break
        x = x + step(A, m, r, 1e-9)
    return x


def _dot3(a, b):
    return (a * b).sum(-1)


class _Mesh:
    """The mesh per (cell, face slot), as tensors: neighbour (itself on the
    boundary), interior mask, outward vectors and the face's numbers."""

    def __init__(self, s, m):
        self.n = m.numel
        self.rows = _t(m.id.astype(np.int64)) - 1
        nb = _t(m.nelcon.astype(np.int64)) - 1
        self.inside = nb > -1
        me = torch.arange(self.n, device=nb.device)[:, None].expand_as(nb)
        self.nb = torch.where(self.inside, nb, me)
        face = _t(m.cellface.astype(np.int64)) - 1
        sign = torch.where(_t(m.owner.astype(np.int64))[face, 0] - 1 == me, 1.0, -1.0)
        sign = sign.to(torch.float64)
        self.mk, self.area = _t(m.mksi)[face], _t(m.area)[face]
        self.ksi = sign[..., None] * _t(m.ksi)[face]
        self.nrm = sign[..., None] * _t(m.normal)[face]
        self.xmcc, self.dcca, self.xm = _t(m.xmcc), _t(m.dcca), _t(m.xm)[face]
        self.alpha = torch.linalg.vector_norm(_t(m.vskew)[face] + self.xmcc, dim=-1) / self.mk
        self.volume = _t(m.volume)
        self.cdiff = _t(m.cdiff)
        side = torch.arange(6, device=nb.device).expand_as(nb)
        self.boundary = lambda sides: ~self.inside & torch.tensor(  # noqa: E731
            sides, device=nb.device)[side].bool()

    def matrix(self, coef, diag):
        """The matrix with off-diagonals -coef at the interior faces."""
        cell, slot = self.inside.nonzero(as_tuple=True)
        d = torch.empty_like(diag)
        d[self.rows] = diag
        return _csr(self.n, self.rows[cell], self.rows[self.nb[cell, slot]],
                    -coef[cell, slot], d), d

    def by_row(self, v):
        out = torch.empty_like(v)
        out[self.rows] = v
        return out


def _lsq(M, u, fixed, value):
    """Least-squares gradient of u (n, k): weights 1/|ksi|^2, du = value - u
    on the faces ``fixed``, zero on a wall, extrapolated where no load is."""
    w = 1.0 / M.mk ** 2
    dx = M.ksi * M.mk[..., None]
    inv = torch.linalg.inv(torch.einsum("cf,cfi,cfj->cij", w, dx, dx))
    lsq = torch.einsum("cf,cfj,cij->cif", w, dx, inv)
    du = torch.where(M.inside[..., None], u[M.nb] - u[:, None, :], 0.0)
    load, free = fixed
    du = torch.where(load[..., None], value - u[:, None, :], du)
    g = torch.einsum("cif,cfk->cki", lsq, du)
    du = torch.where(free[..., None], torch.einsum("cki,cfi->cfk", g, M.xmcc), du)
    return torch.einsum("cif,cfk->cki", lsq, du)


def _exact_gradients(M, f):
    lid = M.boundary([0, 0, 0, 0, 0, 1])
    none = torch.zeros_like(lid)
    gv = _lsq(M, f["vel"], (lid, none), torch.tensor([1.0, 0.0, 0.0], device=lid.device,
                                                     dtype=torch.float64))
    fixed, free = M.boundary([1, 0, 0, 0, 0, 0]), M.boundary([0, 1, 1, 1, 1, 1])
    gp = _lsq(M, f["pres"][:, None], (fixed, free), torch.zeros((), device=lid.device,
                                                                dtype=torch.float64))
    return gv, gp[:, 0, :]


def _exact_momentum(M, f, gp):
    """Laminar SIMPLE momentum: orthogonal diffusion, first-order upwind,
    second-order face pressure, walls by their tangential stress, Euler time
    term, under-relaxation 0.7.  (coef, ad (3, n), force (3, n), D, residual)."""
    mu, rho, dt, under = 1e-3, 1.0, 1e-2, 0.7
    vel, pres = f["vel"], f["pres"]
    al, zero = M.alpha, torch.zeros((), device=vel.device, dtype=torch.float64)
    dfd = mu * M.area / M.mk
    wf = (1 - al)[..., None] * vel[:, None, :] + al[..., None] * vel[M.nb]
    cv = torch.where(M.inside, rho * _dot3(wf, M.nrm) * M.area, zero)
    coef = torch.where(M.inside, dfd - torch.clamp(cv, max=0.0), zero)
    rv = M.xm - f["cc"][M.nb]
    p1 = pres[:, None] + _dot3(gp[:, None, :], M.xmcc)
    p2 = pres[M.nb] + _dot3(gp[M.nb], rv)
    pf = torch.where(M.inside, 0.5 * (p1 + p2), pres[:, None].expand_as(p1))
    force = -((pf * M.area)[..., None] * M.nrm).sum(1)
    ap = torch.where(M.inside, zero, mu * M.area / M.dcca)[..., None]
    vb = torch.zeros((M.n, 6, 3), device=vel.device, dtype=torch.float64)
    vb[..., 0] = torch.where(M.boundary([0, 0, 0, 0, 0, 1]), 1.0, 0.0)
    dv = vel[:, None, :] - vb
    tang = _dot3(dv, M.nrm)[..., None] * M.nrm - dv * M.nrm ** 2
    force += (ap * (vb * (1 - M.nrm ** 2) + tang)).sum(1)
    wall = (ap * (1 - M.nrm ** 2)).sum(1)
    total = coef.sum(1)
    ad = ((cv.sum(1) + rho * M.volume / dt + total)[:, None] + wall) / under
    force += (1 - under) * ad * vel
    res = (coef[..., None] * torch.where(M.inside[..., None], vel[M.nb], zero)).sum(1)
    res = res + force - ad * vel
    return coef, ad, force, M.volume[:, None] / ad, res


def _exact_pressure(M, f, gp, dfield):
    rho, vel, pres = 1.0, f["vel"], f["pres"]
    a1, a = (1 - M.alpha)[..., None], M.alpha[..., None]
    zero = torch.zeros((), device=vel.device, dtype=torch.float64)
    df = a1 * dfield[:, None, :] + a * dfield[M.nb]
    coef = rho * M.area * torch.linalg.vector_norm(df * M.nrm, dim=-1) / M.mk
    coef = torch.where(M.inside, coef, zero)
    wfn = _dot3(a1 * vel[:, None, :] + a * vel[M.nb], M.nrm)
    g1 = _dot3(a1 * gp[:, None, :] + a * gp[M.nb], M.ksi) - (pres[M.nb] - pres[:, None]) / M.mk
    wfn = wfn + g1 * _dot3(df * M.ksi, M.nrm)
    force = -torch.where(M.inside, rho * wfn * M.area, zero).sum(1)
    side = M.area * torch.linalg.vector_norm(dfield[:, None, :] * M.nrm, dim=-1) / M.dcca
    ad = coef.sum(1) + torch.where(M.boundary(PRES_SIDES), rho * side, zero).sum(1)
    return coef, ad, force


def _exact_diffusion(M, u0):
    """Orthogonal diffusion, harmonic face diffusivity, u = 0 on x = 0, in
    residual form."""
    k = M.cdiff
    zero = torch.zeros((), device=u0.device, dtype=torch.float64)
    kf = 1.0 / (M.alpha / k[:, None] + (1 - M.alpha) / k[M.nb])
    coef = torch.where(M.inside, kf * M.area / M.mk, zero)
    side = torch.where(M.boundary(PRES_SIDES), k[:, None] * M.area / M.dcca, zero)
    ad = coef.sum(1) + side.sum(1)
    res = (coef * torch.where(M.inside, u0[M.nb], zero)).sum(1) - ad * u0
    return coef, ad, res


def exact(case, seed):
    kind = case["kind"]
    if kind == "pcg":
        s = _poisson(case, seed)
        return _solve(_system(s), _t(s.ad), _t(s.b[0]), _cg)
    if kind == "momentum":
        s = _convection(case, seed, 3)
        A = _system(s)
        return torch.stack([_solve(A, _t(s.ad), _t(b), _bicgstab) for b in s.b])
    if kind == "energy":
        s = _convection(case, seed, 1)
        return _solve(_system(s), _t(s.ad), _t(s.b[0]), _bicgstab)
    if kind == "batch":
        return torch.cat([_solve(_system(s), _t(s.ad), _t(s.b[0]), _cg)
                          for s in _boxes(case, seed)])
    if kind == "adjoint":
        s = _convection(case, seed, 1)
        w = _t(np.random.default_rng(seed).standard_normal(s.neq))
        x = _solve(_system(s), _t(s.ad), _t(s.b[0]), _bicgstab)
        lam = _solve(_system(s, transpose=True), _t(s.ad), w, _bicgstab)
        rows = _t(np.repeat(np.arange(s.neq), np.diff(s.ia)))
        return [x, -lam[rows] * x[_t(s.ja.astype(np.int64))], -lam * x, lam]
    s, m, f = _cavity(case, seed)
    M = _Mesh(s, m)
    f = {k: _t(v) for k, v in f.items()}
    gv, gp = _exact_gradients(M, f)
    coef, ad3, force, dfield, res = _exact_momentum(M, f, gp)
    blocks = lambda v: torch.cat([M.by_row(v[:, k].contiguous()) for k in range(3)])  # noqa: E731
    cp, adp, fp = _exact_pressure(M, f, gp, dfield)
    if kind == "assembly":
        cd, add, resd = _exact_diffusion(M, f["u0"])
        y = [M.matrix(c, d)[0] @ f["u0"]
             for c, d in ((coef, ad3[:, 0].contiguous()), (cp, adp), (cd, add))]
        rc3 = torch.cat([res[:, k] for k in range(3)])
        return [gv, gp, blocks(ad3), blocks(res), rc3, dfield, M.by_row(fp), fp,
                M.by_row(resd), resd, *y]
    x3 = []
    for k in range(3):
        A, d = M.matrix(coef, ad3[:, k].contiguous())
        x3.append(_solve(A, d, M.by_row(force[:, k].contiguous()), _bicgstab))
    A, d = M.matrix(cp, adp)
    return [gv, gp, blocks(ad3), blocks(force), dfield, M.by_row(fp), torch.cat(x3),
            _solve(A, d, M.by_row(fp), _cg)]
