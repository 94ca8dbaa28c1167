"""The work that a user of the heat framework has it do, as measurable cases.

Sizes follow the repository's benchmarks and tests: FE_Q(1..6) on boxes from the 16^3-cell
correctness case (35,937 DoFs) to the 128^3-cell FE_Q(3) scan (57 M DoFs), uniform and deformed
meshes, constant and temperature-dependent conductivity, FP64 and FP32 vectors, the three-phase
melt-pool operator with convection, a locally refined mesh, and the guess network.

Kinds of case and what a pass of each is:
  vmult     one application of the tangent operator (op.vmult)
  picard    one application of the FP32 Picard operator of the mixed-precision preconditioner
  assemble  what a time step forms before its solve: create_rhs and the inverse diagonal
  solve     one Jacobi-CG solve (LinearSolver.solve) from a zero guess
  step      one implicit heat step, mixed precision (FP64 flexible CG, FP32 p-multigrid)
  meltpool  one implicit step of the three-phase law with convection (flexible GMRES)
  amr       one implicit step on a mesh with a refined region (Jacobi-CG)
  train     forward and backward of the guess network on one training sample
"""
import functools
import math

import numpy as np
import torch
import torch.nn.functional as F

from meltpooldg_b200 import _lib as L
from meltpooldg_b200 import heat as H
from meltpooldg_b200 import learned as LG
from meltpooldg_b200.amr import AmrHeatOperator

K0, K1 = 1.0, 0.5  # k(T) = 1 + 0.5 T
DT = 5e-4
DEV = "cuda:0"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the correctness problem (FE_Q(2), 16^3): the smallest call, where latency counts
        dict(name="vmult_p2_16_f64", kind="vmult", degree=2, mx=16, my=16, mz=16, perturb=0.0,
             law="constant", dtype="f64"),
        # the outer operator of the scan benchmark, 57 M DoFs
        dict(name="vmult_p3_128_kT_f64", kind="vmult", degree=3, mx=128, my=128, mz=128,
             perturb=0.0, law="linear_k", dtype="f64"),
        # the outer operator of the production run: deformed mesh, degree 4, 57 M DoFs
        dict(name="vmult_p4_96_deformed_kT_f64", kind="vmult", degree=4, mx=96, my=96, mz=96,
             perturb=0.2, law="linear_k", dtype="f64"),
        # high degree of the operator sweep, constant law, odd cell counts
        dict(name="vmult_p5_53x49x51_f64", kind="vmult", degree=5, mx=53, my=49, mz=51,
             perturb=0.0, law="constant", dtype="f64"),
        # FP32 on a deformed mesh, odd and unequal cell counts
        dict(name="vmult_p2_91x103x97_deformed_f32", kind="vmult", degree=2, mx=91, my=103, mz=97,
             perturb=0.2, law="constant", dtype="f32"),
        # the preconditioner's operator, the one that a mixed-precision step calls most
        dict(name="picard_p3_97x101x89_f32", kind="picard", degree=3, mx=97, my=101, mz=89,
             perturb=0.0, law="linear_k", dtype="f32"),
        # residual and Jacobi diagonal on a deformed mesh
        dict(name="assemble_p3_64_deformed", kind="assemble", degree=3, mx=64, my=64, mz=64,
             perturb=0.2, law="linear_k", dtype="f64"),
        # the correctness problem's solve to 1e-10: many small launches
        dict(name="solve_p2_16", kind="solve", degree=2, mx=16, my=16, mz=16, perturb=0.0,
             law="constant", dtype="f64"),
        # one step of the scan benchmark
        dict(name="step_p3_128", kind="step", degree=3, mx=128, my=128, mz=128, perturb=0.0,
             law="linear_k", dtype="f64"),
        # one melt-pool step, nonsymmetric operator
        dict(name="meltpool_p3_48", kind="meltpool", degree=3, mx=48, my=48, mz=48, perturb=0.0,
             law="three_phase", dtype="f64"),
        # one step on a mesh with its middle refined once
        dict(name="amr_step_p3_24", kind="amr", degree=3, mx=24, my=24, mz=24, perturb=0.0,
             law="linear_k", dtype="f64"),
        # one training sample of the guess network on its training grid
        dict(name="train_97", kind="train", mx=97, my=97, mz=97),
    ]


def draw(rng):
    kind = rng.choice(["vmult"] * 5 + ["picard"] * 2 + ["assemble", "solve", "step", "step",
                                                       "meltpool", "amr", "train"])

    def box(degree, lo, hi):
        """Three cell counts for lo..hi DoFs, spread over the logarithm, mostly unequal."""
        per = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1.0 / 3.0) / degree
        m = [max(3, int(round(per * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(3)]
        return dict(zip(("mx", "my", "mz"), m))

    if kind == "train":
        d = [rng.randint(33, 113) for _ in range(3)]
        return dict(kind=kind, mx=d[0], my=d[1], mz=d[2])
    if kind == "vmult":
        p = rng.randint(1, 6)
        return dict(kind=kind, degree=p, **box(p, 2e4, 4e7), perturb=rng.choice([0.0, 0.2]),
                    law=rng.choice(["constant", "linear_k"]), dtype=rng.choice(["f64", "f32"]))
    if kind == "picard":
        p = rng.randint(1, 4)
        return dict(kind=kind, degree=p, **box(p, 2e4, 4e7), perturb=rng.choice([0.0, 0.2]),
                    law="linear_k", dtype="f32")
    if kind == "assemble":
        p = rng.randint(1, 5)
        return dict(kind=kind, degree=p, **box(p, 2e4, 2e7), perturb=rng.choice([0.0, 0.2]),
                    law="linear_k", dtype="f64")
    if kind == "solve":
        p = rng.randint(1, 4)
        return dict(kind=kind, degree=p, **box(p, 2e4, 2e6), perturb=rng.choice([0.0, 0.2]),
                    law="constant", dtype="f64")
    if kind == "step":  # cell counts that the multigrid can coarsen at least once
        p = rng.randint(2, 4)
        c = box(p, 2e5, 1e7)
        return dict(kind=kind, degree=p, **{k: 4 * max(2, (v + 2) // 4) for k, v in c.items()},
                    perturb=rng.choice([0.0, 0.2]), law="linear_k", dtype="f64")
    if kind == "meltpool":
        p = rng.randint(2, 3)
        return dict(kind=kind, degree=p, **box(p, 1e5, 2e6), perturb=rng.choice([0.0, 0.1]),
                    law="three_phase", dtype="f64")
    m = rng.randint(8, 22)
    return dict(kind="amr", degree=rng.randint(1, 3), mx=m, my=m + rng.randint(-3, 3),
                mz=m + rng.randint(-3, 3), perturb=0.0, law="linear_k", dtype="f64")


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gll(n):
    """Gauss-Lobatto points of n nodes on [0, 1]."""
    inner = np.polynomial.legendre.Legendre.basis(n - 1).deriv().roots()
    return 0.5 * (1.0 + np.concatenate([[-1.0], np.sort(inner.real), [1.0]]))


def _nodes_1d(p, m):
    g = _gll(p + 1)
    x = (np.arange(m)[:, None] + g[None, :-1]).reshape(-1) / m
    return torch.tensor(np.append(x, 1.0), dtype=torch.float64, device=DEV)


def _rand(shape, seed, k, lo, hi, dtype=torch.float64):
    """Uniform values in [lo, hi] of a seed and a field number k."""
    g = torch.Generator(device=DEV).manual_seed(1000 * int(seed) + k)
    return torch.rand(shape, dtype=dtype, device=DEV, generator=g) * (hi - lo) + lo


def _bump(xs, centre, radius):
    """exp(-|x - centre|^2 / radius^2) at the nodes, z slowest (the lexicographic DoF order)."""
    e = [torch.exp(-((x - c) / radius) ** 2) for x, c in zip(xs, centre)]
    return (e[2][:, None, None] * e[1][None, :, None]) * e[0][None, None, :]


def _shape(xs):
    """1 in the box, 0 on its faces."""
    e = [torch.tanh(8.0 * x) * torch.tanh(8.0 * (1.0 - x)) for x in xs]
    return (e[2][:, None, None] * e[1][None, :, None]) * e[0][None, None, :]


def _history(case, seed):
    """T, T_old and the source of a scan: a warm track behind the beam, the beam at z = 0.95."""
    xs = [_nodes_1d(case["degree"], case[k]) for k in ("mx", "my", "mz")]
    r = np.random.default_rng(seed)
    y, x0 = r.uniform(0.3, 0.7), r.uniform(0.35, 0.7)
    amp = r.uniform(0.3, 0.6, 4)
    hull = _shape(xs)

    def track(x_beam):
        t = 0.05
        for i in range(4):
            t = t + amp[i] * _bump(xs, (x_beam - 0.06 * i, y, 0.9), 0.06 + 0.03 * i)
        return (hull * t).reshape(-1).contiguous()

    q = (500.0 * _bump(xs, (x0 + DT, y, 0.95), 0.05)).reshape(-1).contiguous()
    return track(x0), track(x0 - DT), q


def _mesh(case):
    return H.box_mesh(case["degree"], (case["mx"], case["my"], case["mz"]),
                      perturb=case["perturb"], seed=1)


def _operator(case):
    op = H.HeatDiffuseOperator(_mesh(case))
    if case["law"] == "three_phase":
        op.set_material(H.material(law=L.LAW_GAS_LIQUID_SOLID, rho=1.0, cp=1.0, k=1.0, rho_s=1.0,
                                   cp_s=1.2, k_s=1.5, T_solidus=0.3, T_liquidus=0.5, rho_g=0.1,
                                   cp_g=1.0, k_g=0.05))
    elif case["law"] == "linear_k":
        op.set_material(H.material(law=L.LAW_LINEAR_K, k=K0, k1=K1))
    else:
        op.set_material(H.material(law=L.LAW_CONSTANT, k=1.0))
    return op


def _dt(case):
    return 1e-3 if case["kind"] == "solve" else DT


def _free(case):
    """1 at the DoFs off the boundary (all faces are Dirichlet faces), 0 on it."""
    dims = [case["degree"] * case[k] + 1 for k in ("mz", "my", "mx")]
    m = torch.zeros(dims, dtype=torch.float64, device=DEV)
    m[1:-1, 1:-1, 1:-1] = 1.0
    return m.reshape(-1)


def _refined(case):
    """The refinement flags of an `amr` case: the middle half of every direction."""
    m = (case["mz"], case["my"], case["mx"])
    ref = np.zeros(m, dtype=np.uint8)
    ref[m[0] // 4:m[0] - m[0] // 4, m[1] // 4:m[1] - m[1] // 4, m[2] // 4:m[2] - m[2] // 4] = 1
    return ref


def _train_inputs(case, seed):
    """A training sample's three channels and target, and the weights."""
    dims = (case["mx"], case["my"], case["mz"])
    xs = [torch.linspace(0, 1, d, dtype=torch.float64, device=DEV) for d in dims]
    r = np.random.default_rng(seed)
    c = (r.uniform(0.3, 0.7), r.uniform(0.3, 0.7), 0.9)
    chans = [_bump(xs, c, 0.06) - 0.8 * _bump(xs, (c[0] - 0.03, c[1], c[2]), 0.07),
             _bump(xs, (c[0], c[1], 0.95), 0.05), _bump(xs, (c[0] - 0.05, c[1], 0.9), 0.15)]
    x = torch.stack([(10.0 * v).reshape(-1) for v in chans]).float().contiguous()
    t = (0.5 * _bump(xs, (c[0] + 0.01, c[1], c[2]), 0.05)).reshape(-1).float().contiguous()
    w = []
    for i, (ci, co) in enumerate(LG.LAYERS):
        b = math.sqrt(6.0 / (27.0 * ci))
        w.append(_rand(ci * co * 27, seed, 2 * i, -b, b, torch.float32))
        w.append(_rand(co, seed, 2 * i + 1, -0.1, 0.1, torch.float32))
    return x.reshape(-1), t, torch.cat(w)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "train":
        x, t, w = _train_inputs(case, seed)
        net = LG.UNet((case["mx"], case["my"], case["mz"]), seed=1)
        net.set_params(w)
        s.update(net=net, x=x, target=t)
        return s
    if kind == "amr":
        op = AmrHeatOperator(_mesh(case), _refined(case), device=0)
        op.set_material(H.material(law=L.LAW_LINEAR_K, k=K0, k1=K1), DT)
        pos = torch.tensor(op.support_points(), device=DEV)
        r = np.random.default_rng(seed)
        c = torch.tensor([r.uniform(0.4, 0.6), r.uniform(0.4, 0.6), 0.7], dtype=torch.float64,
                         device=DEV)
        hull = torch.prod(torch.tanh(8.0 * pos) * torch.tanh(8.0 * (1.0 - pos)), dim=1)

        def field(centre, radius, amp):
            return (hull * amp * torch.exp(-((pos - centre) ** 2).sum(1) / radius ** 2)).contiguous()

        s.update(op=op, T0=field(c, 0.1, 0.8), q=field(c, 0.06, 400.0))
        c[0] -= DT
        s["T1"] = field(c, 0.1, 0.8)
        s["T"], s["T_old"] = torch.empty_like(s["T0"]), torch.empty_like(s["T0"])
        prm = H.step_params()
        prm.linear.rel_tolerance, prm.linear.abs_tolerance = 1e-8, 0.0
        s["prm"] = prm
        return s
    op = _operator(case)
    op.reset_time_increment(_dt(case))
    s["op"] = op
    n = op.n_dofs
    if kind in ("vmult", "picard"):
        dtype = torch.float32 if case["dtype"] == "f32" else torch.float64
        s["src"] = _rand(n, seed, 0, -1.0, 1.0).to(dtype)
        s["dst"] = op.new_vector(dtype)
        if case["law"] == "linear_k":
            s["T"] = _history(case, seed)[0]
            op.set_linearization(s["T"], s["T"])
    elif kind == "assemble":
        s["T"], s["T_old"], s["q"] = _history(case, seed)
        s["rhs"], s["diag"] = op.new_vector(), op.new_vector()
    elif kind == "solve":
        s["b"] = _rand(n, seed, 0, 0.0, 1.0).mul_(_free(case)).mul_(1.0 / n)
        s["x"] = op.new_vector()
        s["jacobi"] = H.JacobiPreconditioner(op)
        s["data"] = H.LinearSolverData(rel_tolerance=1e-10)
    else:
        if kind == "meltpool":
            xs = [_nodes_1d(case["degree"], case[k]) for k in ("mx", "my", "mz")]
            one = [torch.ones_like(x) for x in xs]

            def grid(fx, fy, fz):
                return ((fz[:, None, None] * fy[None, :, None]) * fx[None, None, :]).reshape(-1)

            hs = grid(one[0], one[1], 0.5 + 0.5 * torch.tanh((0.9 - xs[2]) / 0.02))
            vel = torch.stack([
                0.2 * grid(torch.sin(math.pi * xs[0]), one[1], torch.cos(math.pi * xs[2])),
                torch.zeros(n, dtype=torch.float64, device=DEV),
                -0.2 * grid(torch.cos(math.pi * xs[0]), one[1], torch.sin(math.pi * xs[2]))])
            s["fields"] = (hs.contiguous(), vel.contiguous())
            op.set_fields(*s["fields"])
            data = H.LinearSolverData(solver_type=L.SOLVER_GMRES,
                                      preconditioner_type=L.PRECOND_CHEBYSHEV_JACOBI_F32,
                                      cheb_degree=6, rel_tolerance=1e-8, abs_tolerance=0.0,
                                      cheb_eig_reuse=True)
        else:
            data = H.LinearSolverData(preconditioner_type=L.PRECOND_MG_F32, rel_tolerance=1e-8,
                                      abs_tolerance=0.0, cheb_picard=True, cheb_eig_reuse=True)
        s["T0"], s["T1"], q = _history(case, seed)
        s["opn"] = H.HeatDiffuseOperation(op, data, predictor=L.PREDICTOR_LINEAR,
                                          single_linearization=True)
        s["opn"].heat_source = q
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["case"]["kind"]
    if kind == "vmult":
        return s["op"].vmult(s["dst"], s["src"])
    if kind == "picard":
        return s["op"].vmult_picard_f32(s["dst"], s["src"])
    if kind == "assemble":
        s["op"].set_linearization(s["T"], s["T_old"])
        s["rhs"].zero_()
        s["op"].create_rhs(s["rhs"], s["T_old"], s["q"])
        return s["rhs"], s["op"].compute_inverse_diagonal_from_matrixfree(s["diag"])
    if kind == "solve":
        s["x"].zero_()
        s["jacobi"].update()
        H.LinearSolver.solve(s["op"], s["x"], s["b"], s["data"], s["jacobi"])
        return s["x"]
    if kind in ("step", "meltpool"):
        opn = s["opn"]
        opn.T.copy_(s["T0"])
        opn.T_old.copy_(s["T1"])
        opn.dt_old = DT
        opn.solve(DT)
        return opn.T
    if kind == "amr":
        s["T"].copy_(s["T0"])
        s["T_old"].copy_(s["T1"])
        s["op"].time_step(s["T"], s["T_old"], DT, DT, s["q"], s["prm"])
        return s["T"]
    y = s["net"].forward(s["x"])
    return y, s["net"].backward((y - s["target"]) * (2.0 / y.numel()))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once; operations of the sum-factorised cell loops
    (even-odd 1D contractions) at typical iteration counts for the solves."""
    if case["kind"] == "train":
        d = [(case["mx"], case["my"], case["mz"])]
        for _ in range(3):
            d.append(tuple((v + 1) // 2 for v in d[-1]))
        pts = [a * b * c for a, b, c in d]
        level = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0]
        mac = sum(27 * ci * co * pts[lv] for (ci, co), lv in zip(LG.LAYERS, level))
        w = sum(27 * ci * co + co for ci, co in LG.LAYERS)
        return {"bytes": 4.0 * (5 * pts[0] + 2 * w), "flops": 6.0 * mac}
    p, m = case["degree"], (case["mx"], case["my"], case["mz"])
    n, cells = p + 1, m[0] * m[1] * m[2]
    if case["kind"] == "amr":
        cells += 7 * int(_refined(case).sum())
    dofs = (cells * p ** 3 if case["kind"] == "amr" else
            (p * m[0] + 1) * (p * m[1] + 1) * (p * m[2] + 1))
    s = 4 if case["dtype"] == "f32" else 8
    geo = 24.0 * (m[0] + 1) * (m[1] + 1) * (m[2] + 1) if case["perturb"] else 0.0
    apply = cells * (12.0 * n ** 4 + 24.0 * n ** 3)
    lin = 0 if case["law"] == "constant" else 8
    vectors, applications = {"vmult": (2 * s + lin, 1), "picard": (2 * s + lin, 1),
                             "assemble": (6 * 8, 3), "solve": (2 * 8 + lin, 60),
                             "step": (4 * 8, 40), "meltpool": (8 * 8, 200),
                             "amr": (4 * 8, 60)}[case["kind"]]
    return {"bytes": vectors * float(dofs) + geo, "flops": applications * apply}


# ---------------------------------------------------------------------------
# the same results in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _vertices(case):
    """Vertices of the box mesh, interior ones moved by at most perturb x h from a hash."""
    m = (case["mx"], case["my"], case["mz"])
    a, b, c = np.meshgrid(*(np.arange(k + 1) for k in m), indexing="ij")
    idx = np.stack([a, b, c], -1).transpose(2, 1, 0, 3)  # [z][y][x][3]
    v = (idx[..., 0] + (m[0] + 1) * (idx[..., 1] + (m[1] + 1) * idx[..., 2])).astype(np.uint64)
    inner = np.all((idx > 0) & (idx < np.array(m)), axis=-1)
    x = np.empty(idx.shape)
    for e in range(3):
        h = 1.0 / m[e]
        x[..., e] = h * idx[..., e]
        r = np.uint64(0xD1B54A32D192ED03) + np.uint64(3) * v + np.uint64(e)
        r = r + np.uint64(0x9E3779B97F4A7C15)
        r = (r ^ (r >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        r = (r ^ (r >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        r = r ^ (r >> np.uint64(31))
        u = 2.0 * ((r >> np.uint64(11)).astype(np.float64) * (1.0 / 9007199254740992.0)) - 1.0
        x[..., e] += np.where(inner, case["perturb"] * h * u, 0.0)
    return torch.tensor(x, device=DEV)


@functools.lru_cache(maxsize=None)
def _tables(n):
    """Values and derivatives of the Lagrange basis on GLL nodes at the Gauss points, [q][i]."""
    xl = _gll(n)
    xg, wg = np.polynomial.legendre.leggauss(n)
    xg, wg = 0.5 * (1.0 + xg), 0.5 * wg
    S, D = np.empty((n, n)), np.empty((n, n))
    for i in range(n):
        c = np.poly1d(np.delete(xl, i), r=True)
        c = c / c(xl[i])
        S[:, i], D[:, i] = c(xg), c.deriv()(xg)
    return xg, wg, S, D


class _Exact:
    """The heat operator, residual and diagonal on a box mesh, slab by slab of cell layers."""

    def __init__(self, case, dt):
        self.p, self.n = case["degree"], case["degree"] + 1
        self.m = (case["mx"], case["my"], case["mz"])
        self.dims = [self.p * k + 1 for k in self.m]
        self.dt, self.free = dt, _free(case)
        self.lin = case["law"] == "linear_k"
        self.xg, self.wg, S, D = _tables(self.n)
        self.S = torch.tensor(S, device=DEV)
        self.D = torch.tensor(D, device=DEV)
        self.vert = _vertices(case) if case["perturb"] else None
        layer = self.m[0] * self.m[1] * self.n ** 3
        step = max(1, int(1.2e7 / layer))
        self.slabs = [(z, min(z + step, self.m[2])) for z in range(0, self.m[2], step)]

    def cells(self, u, z):
        """Nodal values per cell, [cz][cy][cx][k][j][i]."""
        p, n = self.p, self.n
        u = u.view(self.dims[2], self.dims[1], self.dims[0])[p * z[0]:p * z[1] + 1]
        return u.unfold(0, n, p).unfold(1, n, p).unfold(2, n, p)

    def scatter(self, out, v, z):
        p = self.p
        o = out.view(self.dims[2], self.dims[1], self.dims[0])[p * z[0]:p * z[1] + 1]
        e = [p * (z[1] - z[0] - 1) + 1, p * (self.m[1] - 1) + 1, p * (self.m[0] - 1) + 1]
        for k in range(self.n):
            for j in range(self.n):
                for i in range(self.n):
                    o[k:k + e[0]:p, j:j + e[1]:p, i:i + e[2]:p] += v[..., k, j, i]

    @staticmethod
    def tensor(u, A, B, C):
        """A along z, B along y, C along x."""
        u = torch.matmul(u, C.T)
        u = torch.matmul(B, u)
        return torch.einsum("qk,...kji->...qji", A, u)

    def at_points(self, u, z):
        c, S, D = self.cells(u, z), self.S, self.D
        return (self.tensor(c, S, S, S),
                [self.tensor(c, S, S, D), self.tensor(c, S, D, S), self.tensor(c, D, S, S)])

    def integrate(self, val, f):
        S, D = self.S.T, self.D.T
        return (self.tensor(val, S, S, S) + self.tensor(f[0], S, S, D) +
                self.tensor(f[1], S, D, S) + self.tensor(f[2], D, S, S))

    def geometry(self, z):
        """JxW and the six values of JxW J^-1 J^-T (xx xy xz yy yz zz) at the points."""
        w = torch.tensor(self.wg, device=DEV)
        w3 = (w[:, None, None] * w[None, :, None]) * w[None, None, :]
        if self.vert is None:
            h = [1.0 / k for k in self.m]
            det = h[0] * h[1] * h[2]
            zero = torch.zeros_like(w3)
            return det * w3, [det / h[0] ** 2 * w3, zero, zero, det / h[1] ** 2 * w3, zero,
                              det / h[2] ** 2 * w3]
        xg = torch.tensor(self.xg, device=DEV)
        N, d = torch.stack([1 - xg, xg], 1), torch.tensor([[-1.0, 1.0]], dtype=torch.float64,
                                                          device=DEV).expand(self.n, 2)
        c = self.vert[z[0]:z[1] + 1].unfold(0, 2, 1).unfold(1, 2, 1).unfold(2, 2, 1)
        J = [[self.tensor(c[:, :, :, e], *t) for t in ((N, N, d), (N, d, N), (d, N, N))]
             for e in range(3)]  # J[e][f] = dx_e / dxi_f
        cof = [[J[(e + 1) % 3][(f + 1) % 3] * J[(e + 2) % 3][(f + 2) % 3] -
                J[(e + 1) % 3][(f + 2) % 3] * J[(e + 2) % 3][(f + 1) % 3] for f in range(3)]
               for e in range(3)]
        det = sum(J[0][f] * cof[0][f] for f in range(3))
        G = [w3 / det * sum(cof[e][a] * cof[e][b] for e in range(3))
             for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
        return det * w3, G

    @staticmethod
    def flux(G, g):
        return [G[0] * g[0] + G[1] * g[1] + G[2] * g[2], G[1] * g[0] + G[3] * g[1] + G[4] * g[2],
                G[2] * g[0] + G[4] * g[1] + G[5] * g[2]]

    def vmult(self, u, T, picard=False):
        u, out = u * self.free, torch.zeros_like(u)
        for z in self.slabs:
            jxw, G = self.geometry(z)
            v, g = self.at_points(u, z)
            if self.lin:
                t, gt = self.at_points(T, z)
                k = K0 + K1 * t
                g = [k * a + (0.0 if picard else K1 * b * v) for a, b in zip(g, gt)]
            self.scatter(out, self.integrate(v * jxw / self.dt, self.flux(G, g)), z)
        return out * self.free

    def rhs(self, T, T_old, q):
        out = torch.zeros_like(T)
        for z in self.slabs:
            jxw, G = self.geometry(z)
            t, g = self.at_points(T, z)
            w = self.at_points((T - T_old) / self.dt - q, z)[0]
            k = K0 + K1 * t if self.lin else K0
            self.scatter(out, self.integrate(-w * jxw, [-a for a in self.flux(G, [k * a for a in g])]), z)
        return out * self.free

    def diagonal(self, T):
        """phi_i J phi_i summed over the cells (squares of the 1D tables)."""
        out = torch.zeros_like(T)
        S, D = self.S, self.D
        P, Q, R = (S * S).T, (D * D).T, (S * D).T
        for z in self.slabs:
            jxw, G = self.geometry(z)
            t, gt = self.at_points(T, z)
            one = torch.ones_like(t)
            k, dk = (K0 + K1 * t, K1) if self.lin else (K0 * one, 0.0)
            b = self.flux(G, [dk * a for a in gt])
            x = self.tensor
            d = x(jxw / self.dt * one, P, P, P)
            d = d + x(k * G[0], P, P, Q) + x(k * G[3], P, Q, P) + x(k * G[5], Q, P, P)
            d = d + x(2 * k * G[1], P, R, R) + x(2 * k * G[2], R, P, R) + x(2 * k * G[4], R, R, P)
            d = d + x(b[0], P, P, R) + x(b[1], P, R, P) + x(b[2], R, P, P)
            self.scatter(out, d, z)
        return out * self.free

    def inverse_diagonal(self, T):
        d = self.diagonal(T)
        return torch.where(d.abs() > 1e-10, 1.0 / torch.where(d == 0, torch.ones_like(d), d),
                           torch.ones_like(d))

    def solve(self, b, T, tol):
        """Jacobi-preconditioned BiCGStab (the k(T) tangent is not symmetric)."""
        inv = self.inverse_diagonal(T) * self.free
        x, r = torch.zeros_like(b), b * self.free
        r0, p, rr, stop = r.clone(), r.clone(), float(r @ r), tol * float(r.norm())
        for _ in range(600):
            pz = inv * p
            v = self.vmult(pz, T)
            a = rr / float(r0 @ v)
            s = r - a * v
            sz = inv * s
            t = self.vmult(sz, T)
            w = float(t @ s) / float(t @ t)
            x += a * pz + w * sz
            r = s - w * t
            if float(r.norm()) <= stop:
                break
            rr, old = float(r0 @ r), rr
            p = r + (rr / old) * (a / w) * (p - w * v)
        return x


def _exact_train(case, seed):
    dims = (case["mz"], case["my"], case["mx"])
    x, t, w = _train_inputs(case, seed)
    w = w.double().requires_grad_(True)
    layers, off = [], 0
    for ci, co in LG.LAYERS:
        layers.append((w[off:off + ci * co * 27].view(co, ci, 3, 3, 3),
                       w[off + ci * co * 27:off + ci * co * 27 + co]))
        off += ci * co * 27 + co

    def conv(i, v):
        return F.conv3d(v, layers[i][0], layers[i][1], padding=1)

    def pool(v):
        pad = [b for k in (4, 3, 2) for b in (0, v.shape[k] % 2)]
        one = F.pad(torch.ones_like(v[:, :1]), pad)
        return F.avg_pool3d(F.pad(v, pad), 2) / F.avg_pool3d(one, 2)

    def up(v, like):
        for k in (2, 3, 4):
            v = v.repeat_interleave(2, dim=k).narrow(k, 0, like.shape[k])
        return v

    v, skips = x.double().view(1, 3, *dims), []
    for lv in range(4):
        v = conv(2 * lv, v if lv == 0 else pool(v)).relu()
        v = conv(2 * lv + 1, v).relu()
        skips.append(v)
    for lv in (2, 1, 0):
        i = 8 + 2 * (2 - lv)
        v = (conv(i, up(v, skips[lv])) + skips[lv]).relu()
        v = conv(i + 1, v).relu()
    y = conv(14, v).reshape(-1)
    gy = ((y - t.double()) * (2.0 / y.numel())).detach()
    (g,) = torch.autograd.grad(y, w, gy)
    return y.detach(), g


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    # no second way to number a refined mesh's DoFs here, and no second nonsymmetric solver
    if kind in ("amr", "meltpool"):
        return None
    e = _Exact(case, _dt(case))
    n = e.dims[0] * e.dims[1] * e.dims[2]
    T = torch.zeros(n, dtype=torch.float64, device=DEV)
    if case["law"] == "linear_k":
        T, T_old, q = _history(case, seed)
    if kind in ("vmult", "picard"):
        src = _rand(n, seed, 0, -1.0, 1.0)
        src = src.float().double() if case["dtype"] == "f32" else src
        return e.vmult(src, T, picard=kind == "picard")
    if kind == "assemble":
        return e.rhs(T, T_old, q), e.inverse_diagonal(T)
    if kind == "solve":
        b = _rand(n, seed, 0, 0.0, 1.0).mul_(_free(case)).mul_(1.0 / n)
        return e.solve(b, T, 1e-14)
    if n > 1.2e7:  # a Krylov solve of this size with plain torch takes too long
        return None
    guess = (2.0 * T - T_old) * e.free
    b = e.rhs(guess, T, q)
    return guess + e.solve(b, guess, 1e-13)
