"""The timed cases: what a topology-optimisation program has this library do,
through its public entry points, from the smallest mesh to the largest.

A case is a dict of plain values; its "kind" picks the call:

  solve     one Helmholtz / Poisson solve from a zero guess (ksp.solve)
  sequence  the next solve of a design sequence with the learned guess
            (SolveSequence.solve: prediction, solve, online training)
  filter    the PDE density filter, forward and backward
  operator  the assembled operator in FP64: Ax, gather-scatter, Dirichlet mask
  inner     the FP32 pieces of the mixed solver: Ax, gather-scatter, mask and
            one application of the two-level Schwarz preconditioner
  residuals the Pn/Pn pressure and velocity residuals of a time step
  dealias   the dealiased adjoint or linearised advection term
  advect    both advection terms without dealiasing and the minimum-
            dissipation forcing
  mma       one design update of the MMA optimiser

Meshes are boxes of ex x ey x ez hexahedra with lx^3 GLL nodes each,
deformed by a seeded sinusoid of 5% of the element size, x fastest.
"""
import math

import numpy as np
import torch

from __graft_entry__ import load_package

DEV = "cuda"
RTOL = 1e-10


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    def box(e, lx):
        return {"ex": e[0], "ey": e[1], "ez": e[2], "lx": lx}

    return [
        # an 8^3 design mesh, FP64 Jacobi-PCG: the small solves of a first
        # design study, where launches and latency count
        dict(name="solve_small_fp64", kind="solve", method="cg", op="brinkman", **box((8, 8, 8), 8)),
        # the pressure Poisson solve of an ordinary mesh
        dict(name="solve_poisson", kind="solve", method="cg_mixed", op="poisson", **box((32, 32, 32), 8)),
        # a Brinkman-penalised pressure solve of the largest mesh (134M nodes)
        dict(name="solve_brinkman_large", kind="solve", method="cg_mixed", op="brinkman", **box((64, 64, 64), 8)),
        # the channel sequence: learned guess, solve, 20 training steps
        dict(name="sequence_channel", kind="sequence", **box((64, 16, 16), 8)),
        # the density filter of every design update and its transpose
        dict(name="filter_design", kind="filter", radius=0.01, **box((24, 24, 24), 8)),
        # the FP64 operator of plain CG and of every residual replacement
        dict(name="operator_fp64", kind="operator", **box((32, 32, 32), 8)),
        # one inner iteration's operator and preconditioner on a ragged mesh of lower order
        dict(name="inner_fp32_ragged", kind="inner", **box((21, 13, 17), 6)),
        # the residuals on either side of a time step's solves
        dict(name="residuals", kind="residuals", **box((24, 24, 24), 8)),
        # the advection term of every adjoint step, over-integrated
        dict(name="dealias_adjoint", kind="dealias", mode="adjoint", **box((24, 24, 24), 8)),
        # the linearised one on a small ragged mesh of lower order
        dict(name="dealias_linear_small", kind="dealias", mode="linear", **box((5, 7, 9), 6)),
        # the terms of a run without dealiasing, odd order, ragged mesh
        dict(name="advect_ragged", kind="advect", **box((19, 13, 11), 7)),
        # the optimiser's update, one variable per node of a 32^3 mesh
        dict(name="mma_update", kind="mma", n=32 ** 3 * 512, m=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, cells):
    """Ragged element counts whose product is near `cells`."""
    side = cells ** (1.0 / 3.0)
    a = max(2, int(round(side * rng.uniform(0.6, 1.6))))
    b = max(2, int(round(side * rng.uniform(0.7, 1.4))))
    c = max(2, int(round(cells / (a * b))))
    return {"ex": a, "ey": b, "ez": c}


def draw(rng):
    kind = rng.choice(["solve", "solve", "sequence", "filter", "operator", "operator", "inner", "residuals", "dealias",
                       "dealias", "advect", "mma"])
    if kind == "solve":
        method = rng.choice(["cg", "cg_mixed", "cg_mixed"])
        lx = rng.choice([4, 6, 8, 8])
        op = rng.choice(["poisson", "brinkman"])
        cells = _log_int(rng, 60, 3000 if method == "cg" else 20000)
        return {"kind": kind, "method": method, "op": op, "lx": lx, **_dims(rng, cells)}
    if kind == "sequence":
        return {"kind": kind, "lx": 8, **_dims(rng, _log_int(rng, 500, 16000))}
    if kind == "filter":
        return {"kind": kind, "radius": round(rng.uniform(0.005, 0.05), 4), "lx": rng.choice([4, 5, 6, 7, 8, 8]),
                **_dims(rng, _log_int(rng, 60, 12000))}
    if kind == "operator":
        return {"kind": kind, "lx": rng.choice([4, 5, 6, 7, 8, 8, 8]), **_dims(rng, _log_int(rng, 40, 32000))}
    if kind == "inner":
        return {"kind": kind, "lx": rng.choice([4, 6, 8, 8]), **_dims(rng, _log_int(rng, 40, 32000))}
    if kind == "residuals":
        return {"kind": kind, "lx": rng.choice([4, 5, 6, 7, 8, 8, 8]), **_dims(rng, _log_int(rng, 40, 16000))}
    if kind == "dealias":
        return {"kind": kind, "mode": rng.choice(["adjoint", "linear"]), "lx": rng.choice([4, 5, 6, 7, 8, 8, 8]),
                **_dims(rng, _log_int(rng, 40, 14000))}
    if kind == "advect":
        return {"kind": kind, "lx": rng.choice([4, 5, 6, 7, 8, 8]), **_dims(rng, _log_int(rng, 40, 14000))}
    return {"kind": "mma", "n": _log_int(rng, 3000, 16_000_000), "m": rng.choice([1, 1, 2, 3])}


# ---------------------------------------------------------------------------
# meshes and fields
# ---------------------------------------------------------------------------
def _legendre(n, x):
    p0, p1 = np.ones_like(x), x
    for k in range(2, n + 1):
        p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
    return (p0, p0) if n == 0 else (p1, p0)


def _gll(lx):
    """GLL nodes, weights and differentiation matrix."""
    n = lx - 1
    x = -np.cos(np.pi * np.arange(lx) / n)
    for _ in range(50):
        p, q = _legendre(n, x)
        x = x - (x * p - q) / (lx * p)
    x[0], x[-1] = -1.0, 1.0
    x = 0.5 * (x - x[::-1])
    p = _legendre(n, x)[0]
    d = np.zeros((lx, lx))
    for i in range(lx):
        for j in range(lx):
            if i != j:
                d[i, j] = p[i] / (p[j] * (x[i] - x[j]))
    d[0, 0], d[-1, -1] = -n * lx / 4.0, n * lx / 4.0
    return x, 2.0 / (n * lx * p * p), d


def _rng(seed, stream):
    return np.random.default_rng([int(seed), stream])


class Mesh:
    """Coordinates (flat, i fastest), global node ids and the nodes of the face x = max."""

    def __init__(self, case, seed):
        ex, ey, ez, lx = (int(case[k]) for k in ("ex", "ey", "ez", "lx"))
        self.dims, self.lx, self.nelv, self.n = (ex, ey, ez), lx, ex * ey * ez, ex * ey * ez * lx ** 3
        # elements of one size, the longest side of the box 1
        h = 1.0 / max(ex, ey, ez)
        self.lo, self.hi = (0.0, 0.0, 0.0), (ex * h, ey * h, ez * h)
        t = torch.as_tensor((_gll(lx)[0] + 1.0) / 2.0, device=DEV)
        t[0], t[-1] = 0.0, 1.0

        def axis(d, e, i):  # positions in elements, as [ez, ey, ex, k, j, i]
            shape = [1] * 6
            shape[2 - d], shape[5 - d] = e, i
            c = torch.arange(e, device=DEV, dtype=torch.float64)[:, None] + t[None, :]
            return c.reshape(shape)

        s = [axis(d, self.dims[d], lx) for d in range(3)]
        r = _rng(seed, 1)
        full = (ez, ey, ex, lx, lx, lx)
        self.xyz = []
        for d in range(3):
            k, ph = r.integers(1, 4, 3), r.uniform(0, 2 * math.pi)
            wave = torch.sin(2 * math.pi / 16 * (k[0] * s[0] + k[1] * s[1] + k[2] * s[2]) + ph)
            self.xyz.append((h * (s[d] + 0.05 * wave)).expand(full).contiguous().reshape(-1))
        ids = []
        for d in range(3):
            shape = [1] * 6
            shape[2 - d], shape[5 - d] = self.dims[d], lx
            g = torch.arange(self.dims[d], device=DEV)[:, None] * (lx - 1) + torch.arange(lx, device=DEV)[None, :]
            ids.append(g.reshape(shape))
        nx, ny, nz = (e * (lx - 1) + 1 for e in self.dims)
        self.nu = nx * ny * nz
        self.gid = (ids[0] + nx * (ids[1] + ny * ids[2])).expand(full).contiguous().reshape(-1)
        self.face = torch.nonzero((ids[0] == nx - 1).expand(full).reshape(-1)).reshape(-1)

    def coef(self):
        pkg = load_package()
        c = pkg.coef_t(self.nelv, self.lx, *self.xyz, self.gid)
        c.box_dims, c.lo, c.hi = self.dims, self.lo, self.hi
        return c

    def mask(self):  # 1-based, as Neko's masks
        return (self.face + 1).to(torch.int32)


def _field(mesh, seed, stream, modes=8, kmax=4, noise=0.0):
    """A seeded sum of Fourier modes with amplitudes ~ 1/|k|^2, continuous across elements."""
    r = _rng(seed, stream)
    f = torch.zeros(mesh.n, dtype=torch.float64, device=DEV)
    for _ in range(modes):
        k, a, ph = r.integers(1, kmax + 1, 3), r.uniform(-1, 1), r.uniform(0, 2 * math.pi)
        arg = 2 * math.pi * (k[0] * mesh.xyz[0] + k[1] * mesh.xyz[1] + k[2] * mesh.xyz[2]) + ph
        f.add_(arg.cos_(), alpha=a * 3.0 / float((k ** 2).sum()))
    if noise:
        g = torch.Generator(device=DEV).manual_seed(int(seed) * 64 + stream)
        f.add_(torch.randn(mesh.nu, dtype=torch.float64, device=DEV, generator=g)[mesh.gid], alpha=noise)
    return f


def _density(mesh, seed, stream):
    """12 Gaussian blobs clamped to [0, 1]: a material distribution."""
    r = _rng(seed, stream)
    rho = torch.zeros(mesh.n, dtype=torch.float64, device=DEV)
    for _ in range(12):
        c = [r.uniform(mesh.lo[d], mesh.hi[d]) for d in range(3)]
        rho += torch.exp(-50.0 * sum((mesh.xyz[d] - c[d]) ** 2 for d in range(3)))
    return rho.clamp_(0.0, 1.0)


def _permeability(rho):
    """RAMP (q = 8, chi_max = 1e4) of the void fraction."""
    t = 1.0 - rho
    return 1e4 * t / (1.0 + 8.0 * (1.0 - t))


# ---------------------------------------------------------------------------
# plain torch restatement in 64 bits (for exact)
# ---------------------------------------------------------------------------
class Plain:
    def __init__(self, mesh):
        self.m = mesh
        lx = mesh.lx
        _, w, d = _gll(lx)
        self.D = torch.as_tensor(d, device=DEV)
        w = torch.as_tensor(w, device=DEV)
        self.w3 = (w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(1, lx, lx, lx)
        g = [self.rgrad(self.e(c)) for c in mesh.xyz]  # g[c] = (c_r, c_s, c_t)
        (xr, xs, xt), (yr, ys, yt), (zr, zs, zt) = g
        # cofactors cof[d][c] = jac * d(r_d)/d(x_c)
        self.cof = [[ys * zt - yt * zs, xt * zs - xs * zt, xs * yt - xt * ys],
                    [yt * zr - yr * zt, xr * zt - xt * zr, xt * yr - xr * yt],
                    [yr * zs - ys * zr, xs * zr - xr * zs, xr * ys - xs * yr]]
        self.jac = xr * self.cof[0][0] + yr * self.cof[0][1] + zr * self.cof[0][2]
        self.B = self.w3 * self.jac
        self.mult = 1.0 / self.gs(torch.ones_like(self.B))

    def e(self, f):
        lx = self.m.lx
        return f.reshape(self.m.nelv, lx, lx, lx)  # [e, k, j, i]

    def rgrad(self, u, D=None):
        D = self.D if D is None else D
        return (torch.einsum("il,ekjl->ekji", D, u), torch.einsum("jl,ekli->ekji", D, u),
                torch.einsum("kl,elji->ekji", D, u))

    def rdiv(self, r, s, t, D=None):
        D = self.D if D is None else D
        return (torch.einsum("li,ekjl->ekji", D, r) + torch.einsum("lj,ekli->ekji", D, s)
                + torch.einsum("lk,elji->ekji", D, t))

    def gs(self, u):
        acc = torch.zeros(self.m.nu, dtype=torch.float64, device=DEV)
        acc.index_add_(0, self.m.gid, u.reshape(-1))
        return acc[self.m.gid].reshape(u.shape)

    def masked(self, u, dirichlet):
        if dirichlet:
            u.reshape(-1)[self.m.face] = 0.0
        return u

    def ax(self, u, h1=1.0, h2=None):
        g = self.rgrad(u)
        # fluxes of the physical gradient
        p = [sum(self.cof[d][c] * g[d] for d in range(3)) for c in range(3)]
        s = h1 * self.w3 / self.jac
        w = self.rdiv(*[s * sum(self.cof[d][c] * p[c] for c in range(3)) for d in range(3)])
        return w if h2 is None else w + h2 * self.B * u

    def diag(self, h1=1.0, h2=None):
        s = h1 * self.w3 / self.jac
        G = lambda a, b: s * sum(self.cof[a][c] * self.cof[b][c] for c in range(3))  # noqa: E731
        D, d = self.D, torch.diagonal(self.D)
        q = self.rdiv(G(0, 0), G(1, 1), G(2, 2), D * D)
        di, dj, dk = d.reshape(1, 1, 1, -1), d.reshape(1, 1, -1, 1), d.reshape(1, -1, 1, 1)
        q = q + 2 * (di * dj * G(0, 1) + di * dk * G(0, 2) + dj * dk * G(1, 2))
        return q if h2 is None else q + h2 * self.B

    def solve(self, b, dirichlet, h1=1.0, h2=None, x=None, rtol=1e-13, cap=6000):
        A = lambda v: self.masked(self.gs(self.ax(v, h1, h2)), dirichlet)  # noqa: E731
        dot = lambda a, c: (a * c * self.mult).sum()  # noqa: E731
        di = 1.0 / self.gs(self.diag(h1, h2))
        x = torch.zeros_like(b) if x is None else x.clone()
        r = b - A(x)
        z = di * r
        p, rz, stop = z.clone(), dot(r, z), rtol * dot(b, b).sqrt()
        for k in range(cap):
            if k % 8 == 0 and float(dot(r, r).sqrt()) <= float(stop):
                break
            w = A(p)
            a = rz / dot(p, w)
            x += a * p
            r -= a * w
            z = di * r
            rz, old = dot(r, z), rz
            p = z + (rz / old) * p
        return x

    def opgrad(self, u):
        g = self.rgrad(u)
        return [self.w3 * sum(self.cof[d][c] * g[d] for d in range(3)) for c in range(3)]

    def cdtp(self, a):
        """sum_c of the transposed weak derivative in direction c of a[c]."""
        return self.rdiv(*[self.w3 * sum(self.cof[d][c] * a[c] for c in range(3)) for d in range(3)])

    def curl(self, u):
        g = [self.opgrad(v) for v in u]
        b = 1.0 / self.gs(self.B)
        return [b * self.gs(g[2][1] - g[1][2]), b * self.gs(g[0][2] - g[2][0]), b * self.gs(g[1][0] - g[0][1])]


# ---------------------------------------------------------------------------
# kind: solve
# ---------------------------------------------------------------------------
def _solve_inputs(case, seed):
    mesh = Mesh(case, seed)
    h2 = _permeability(_density(mesh, seed, 5)) if case["op"] == "brinkman" else None
    return mesh, h2, _field(mesh, seed, 6, 16)


def _solver(coef, case):
    pkg = load_package()
    ksp = pkg.krylov_solver_factory(coef, case["method"], 20000, RTOL)
    if case["method"] == "cg_mixed":
        ksp.set_inner(2.2e-4, 1)
        ksp.set_schwarz(pkg.schwarz_t(coef, coarse=True))
    return ksp


def _prepare_solve(case, seed):
    mesh, h2, f = _solve_inputs(case, seed)
    coef = mesh.coef()
    coef.set_mask(mesh.mask(), base=1)
    coef.set_coefs(h1c=1.0, h2=h2, ifh2=h2 is not None)
    return {"coef": coef, "ksp": _solver(coef, case), "f": coef.rhs_assemble(f), "x": torch.zeros_like(f)}


def _run_solve(s):
    s["x"].zero_()
    s["ksp"].solve(s["x"], s["f"])
    return s["x"]


def _exact_solve(case, seed):
    n, side = case["ex"] * case["ey"] * case["ez"] * case["lx"] ** 3, max(case["ex"], case["ey"], case["ez"])
    if n > 9e6 or (case["op"] == "poisson" and (n > 1.5e6 or side > 24)):
        return None  # thousands of iterations: minutes in plain torch
    mesh, h2, f = _solve_inputs(case, seed)
    P = Plain(mesh)
    b = P.masked(P.gs(P.B * P.e(f)), True)
    return P.solve(b, True, 1.0, None if h2 is None else P.e(h2)).reshape(-1)


# ---------------------------------------------------------------------------
# kind: sequence
# ---------------------------------------------------------------------------
SEQ_HISTORY, SEQ_LENGTH = 5, 24


def _seq_sources(mesh, seed, steps):
    """Sources of 32 modes whose amplitudes drift (AR(1), 0.98) between solves."""
    r = _rng(seed, 7)
    k, ph = r.integers(1, 5, (32, 3)), r.uniform(0, 2 * math.pi, 32)
    c = r.standard_normal(32)
    for _ in range(steps):
        f = torch.zeros(mesh.n, dtype=torch.float64, device=DEV)
        for m in range(32):
            arg = 2 * math.pi * (k[m, 0] * mesh.xyz[0] + k[m, 1] * mesh.xyz[1] + k[m, 2] * mesh.xyz[2]) + ph[m]
            f.add_(arg.cos_(), alpha=c[m] / float((k[m] ** 2).sum()))
        yield f
        c = 0.98 * c + math.sqrt(1 - 0.98 ** 2) * r.standard_normal(32)


def _prepare_sequence(case, seed):
    pkg = load_package()
    mesh = Mesh(case, seed)
    coef = mesh.coef()
    coef.set_mask(mesh.mask(), base=1)
    coef.set_coefs(h1c=1.0, h2=_permeability(_density(mesh, seed, 5)), ifh2=True)
    seq = pkg.SolveSequence(coef, "cg_mixed", "learned_only", rtol=RTOL, L=20, train_steps=20, seed=3, lr=5e-4,
                            pc="schwarz2", delta=2.2e-4)
    f = [coef.rhs_assemble(g) for g in _seq_sources(mesh, seed, SEQ_HISTORY + SEQ_LENGTH)]
    for b in f[:SEQ_HISTORY]:  # the solves before this one: the network has its history
        seq.solve(b)
    return {"seq": seq, "f": f, "t": SEQ_HISTORY}


def _run_sequence(s):
    x = s["seq"].solve(s["f"][s["t"]])[0]
    s["t"] = s["t"] + 1 if s["t"] + 1 < len(s["f"]) else 0
    return x


def _exact_sequence(case, seed):
    mesh = Mesh(case, seed)
    P = Plain(mesh)
    for f in _seq_sources(mesh, seed, SEQ_HISTORY + 1):
        pass
    b = P.masked(P.gs(P.B * P.e(f)), True)
    return P.solve(b, True, 1.0, P.e(_permeability(_density(mesh, seed, 5))), rtol=1e-12).reshape(-1)


# ---------------------------------------------------------------------------
# kind: filter
# ---------------------------------------------------------------------------
def _prepare_filter(case, seed):
    pkg = load_package()
    mesh = Mesh(case, seed)
    coef = mesh.coef()
    x, g = _density(mesh, seed, 5), _field(mesh, seed, 6)
    return {"filter": pkg.PDE_filter_t(coef, r=case["radius"], abstol=1e-10, max_iter=2000), "x": x, "g": g,
            "y": torch.empty_like(x), "dy": torch.empty_like(x)}


def _run_filter(s):
    s["filter"].apply_forward(s["y"], s["x"])
    s["filter"].apply_backward(s["dy"], s["g"])
    return {"filtered": s["y"], "sensitivity": s["dy"]}


def _exact_filter(case, seed):
    mesh = Mesh(case, seed)
    P, r2 = Plain(mesh), case["radius"] ** 2
    one = torch.ones_like(P.B)
    out = {}
    for name, f in (("filtered", _density(mesh, seed, 5)), ("sensitivity", _field(mesh, seed, 6))):
        out[name] = P.solve(P.gs(P.B * P.e(f)), False, r2, one, x=P.e(f)).reshape(-1)
    return out


# ---------------------------------------------------------------------------
# kind: operator (FP64) and inner (FP32)
# ---------------------------------------------------------------------------
def _operator_inputs(case, seed):
    mesh = Mesh(case, seed)
    return mesh, _permeability(_density(mesh, seed, 5)), _field(mesh, seed, 6, 8, noise=1e-3)


def _prepare_operator(case, seed):
    mesh, h2, u = _operator_inputs(case, seed)
    coef = mesh.coef()
    coef.set_mask(mesh.mask(), base=1)
    coef.set_coefs(h1c=1.0, h2=h2, ifh2=True)
    s = {"coef": coef, "u": u, "w": torch.empty_like(u)}
    if case["kind"] == "inner":
        s["u"], s["w"] = u.float(), torch.empty_like(u, dtype=torch.float32)
        s["sw"], s["z"] = load_package().schwarz_t(coef, coarse=True), torch.empty_like(s["w"])
    return s


def _run_operator(s):
    pkg = load_package()
    pkg.ax_helm_t().compute(s["w"], s["u"], s["coef"])
    pkg.gs_t(s["coef"]).op(s["w"])
    pkg.api.bc_list_apply_scalar(s["coef"], s["w"])
    return s["w"]


def _run_inner(s):
    _run_operator(s)
    s["sw"].apply(s["z"], s["w"])
    return {"w": s["w"], "z": s["z"]}


def _exact_operator(case, seed):
    mesh, h2, u = _operator_inputs(case, seed)
    u = u.float().double() if case["kind"] == "inner" else u
    P = Plain(mesh)
    w = P.masked(P.gs(P.ax(P.e(u), 1.0, P.e(h2))), True).reshape(-1)
    return w if case["kind"] == "operator" else {"w": w, "z": None}


# ---------------------------------------------------------------------------
# kind: residuals
# ---------------------------------------------------------------------------
BD, DT, MU = 11.0 / 6.0, 1e-3, 0.01


def _flow(mesh, seed, stream, count):
    return [_field(mesh, seed, stream + q, 6, noise=1e-4) for q in range(count)]


def _forces(mesh, seed):
    """A right-hand side in weak form: weighted by the mass of a node, as the source terms leave it."""
    volume = math.prod(b - a for a, b in zip(mesh.lo, mesh.hi))
    return [f * (volume / mesh.n) for f in _flow(mesh, seed, 18, 3)]


def _prepare_residuals(case, seed):
    mesh = Mesh(case, seed)
    s = torch.zeros(3, mesh.face.numel(), dtype=torch.float64, device=DEV)
    s[0] = 1.0 / (case["ey"] * case["ez"] * (case["lx"] - 1) ** 2)
    z = torch.zeros(4, mesh.n, dtype=torch.float64, device=DEV)
    return {"coef": mesh.coef().metrics(), "u": _flow(mesh, seed, 10, 3), "ue": _flow(mesh, seed, 14, 3),
            "f": _forces(mesh, seed), "p": _field(mesh, seed, 22), "face": (mesh.mask(), s),
            "p_res": z[0], "res": [z[1], z[2], z[3]]}


def _run_residuals(s):
    pkg = load_package()
    pkg.pnpn_prs_res_t().compute(s["p"], s["p_res"], *s["u"], *s["ue"], *s["f"], s["coef"], s["face"], None, bd=BD,
                                 dt=DT, mu=MU, rho=1.0)
    pkg.pnpn_vel_res_t().compute(*s["u"], *s["res"], s["p"], *s["f"], s["coef"], mu=MU, rho=1.0, bd=BD, dt=DT)
    return {"p_res": s["p_res"], "res": s["res"]}


def _exact_residuals(case, seed):
    mesh = Mesh(case, seed)
    P = Plain(mesh)
    u, ue = ([P.e(v) for v in _flow(mesh, seed, q, 3)] for q in (10, 14))
    f = [P.e(v) for v in _forces(mesh, seed)]
    p = P.e(_field(mesh, seed, 22))
    wa = P.curl(P.curl(ue))
    b = 1.0 / P.gs(P.B)
    ta = [b * P.gs(f[c] - MU * P.B * wa[c]) for c in range(3)]
    pres = (P.cdtp(ta) - P.ax(p)).reshape(-1)
    pres[mesh.face] -= BD / DT * u[0].reshape(-1)[mesh.face] / (case["ey"] * case["ez"] * (case["lx"] - 1) ** 2)
    g = P.opgrad(p)
    res = [(f[c] - P.ax(u[c], MU) - BD / DT * P.B * u[c] - g[c]).reshape(-1) for c in range(3)]
    return {"p_res": pres, "res": res}


# ---------------------------------------------------------------------------
# kinds: dealias, advect
# ---------------------------------------------------------------------------
def _prepare_dealias(case, seed):
    pkg = load_package()
    mesh = Mesh(case, seed)
    adv = pkg.adv_lin_dealias_t(mesh.coef())
    f = _forces(mesh, seed)
    return {"run": adv.compute_adjoint if case["mode"] == "adjoint" else adv.compute_linear, "adv": adv,
            "u": _flow(mesh, seed, 10, 3), "ub": _flow(mesh, seed, 14, 3), "f0": f, "f": [g.clone() for g in f]}


def _run_dealias(s):
    for a, b in zip(s["f"], s["f0"]):  # this step's right-hand side
        a.copy_(b)
    s["run"](*s["u"], *s["ub"], *s["f"])
    return s["f"]


def _exact_dealias(case, seed):
    mesh = Mesh(case, seed)
    P = Plain(mesh)
    lxd = 3 * mesh.lx // 2
    xi = _gll(mesh.lx)[0]
    xg, wg = np.polynomial.legendre.leggauss(lxd)

    def lagrange(src, dst):
        L = np.ones((len(dst), len(src)))
        for a in range(len(src)):
            for k in range(len(src)):
                if k != a:
                    L[:, a] *= (dst - src[k]) / (src[a] - src[k])
        return L

    J = torch.as_tensor(lagrange(xi, xg), device=DEV)
    lam = np.array([1.0 / np.prod([xg[j] - xg[k] for k in range(lxd) if k != j]) for j in range(lxd)])
    Dg = np.array([[0.0 if i == j else lam[j] / lam[i] / (xg[i] - xg[j]) for j in range(lxd)] for i in range(lxd)])
    Dg = torch.as_tensor(Dg - np.diag(Dg.sum(1)), device=DEV)
    wt = torch.as_tensor(wg, device=DEV)
    w3 = wt.reshape(1, -1, 1, 1) * wt.reshape(1, 1, -1, 1) * wt.reshape(1, 1, 1, -1)
    u, ub = ([P.e(v) for v in _flow(mesh, seed, q, 3)] for q in (10, 14))
    f = [P.e(v) for v in _forces(mesh, seed)]
    out = [torch.empty_like(v) for v in f]
    up = lambda v: torch.einsum("Ck,Bj,Ai,ekji->eCBA", J, J, J, v)  # noqa: E731
    down = lambda v: torch.einsum("Ck,Bj,Ai,eCBA->ekji", J, J, J, v)  # noqa: E731
    for a in range(0, mesh.nelv, 1024):
        z = slice(a, min(a + 1024, mesh.nelv))
        U, V = [up(v[z]) for v in u], [up(v[z]) for v in ub]
        cof = [[up(P.cof[d][c][z]) for c in range(3)] for d in range(3)]

        def grad(v):
            g = P.rgrad(v, Dg)
            return [w3 * sum(cof[d][c] * g[d] for d in range(3)) for c in range(3)]

        gV = [grad(v) for v in V]
        if case["mode"] == "adjoint":
            flux = [w3 * sum(cof[d][c] * V[c] for c in range(3)) for d in range(3)]
            t = [sum(U[j] * gV[j][i] for j in range(3)) + P.rdiv(*[U[i] * q for q in flux], Dg) for i in range(3)]
        else:
            gU = [grad(v) for v in U]
            t = [sum(U[d] * gV[i][d] + V[d] * gU[i][d] for d in range(3)) for i in range(3)]
        for i in range(3):
            out[i][z] = f[i][z] - down(t[i])
    return [v.reshape(-1) for v in out]


def _prepare_advect(case, seed):
    pkg = load_package()
    mesh = Mesh(case, seed)
    coef = mesh.coef()
    f, u = _forces(mesh, seed), _flow(mesh, seed, 10, 3)
    fa, fl, fm = ([g.clone() for g in f] for _ in range(3))
    return {"adv": pkg.adv_lin_no_dealias_t(coef), "u": u, "ub": _flow(mesh, seed, 14, 3), "f0": f, "fa": fa, "fl": fl,
            "fm": fm, "forcing": pkg.adjoint_minimum_dissipation_source_term_t(fm, *u, coef, obj_scale=0.5)}


def _run_advect(s):
    for k in ("fa", "fl", "fm"):
        for a, b in zip(s[k], s["f0"]):
            a.copy_(b)
    s["adv"].compute_adjoint(*s["u"], *s["ub"], *s["fa"])
    s["adv"].compute_linear(*s["u"], *s["ub"], *s["fl"])
    s["forcing"].compute()
    return {"adjoint": s["fa"], "linear": s["fl"], "forcing": s["fm"]}


def _exact_advect(case, seed):
    mesh = Mesh(case, seed)
    P = Plain(mesh)
    u, ub = ([P.e(v) for v in _flow(mesh, seed, q, 3)] for q in (10, 14))
    f = [P.e(v) for v in _forces(mesh, seed)]
    gV, gU = [P.opgrad(v) for v in ub], [P.opgrad(v) for v in u]
    w = P.curl(P.curl(u))
    out = {"adjoint": [f[i] - sum(u[j] * gV[j][i] for j in range(3)) - P.cdtp([u[i] * ub[c] for c in range(3)])
                       for i in range(3)],
           "linear": [f[i] - sum(u[d] * gV[i][d] + ub[d] * gU[i][d] for d in range(3)) for i in range(3)],
           "forcing": [f[i] + 0.5 * w[i] for i in range(3)]}
    return {k: [x.reshape(-1) for x in v] for k, v in out.items()}


# ---------------------------------------------------------------------------
# kind: mma
# ---------------------------------------------------------------------------
def _mma_inputs(case, seed):
    """A compliance-like objective and m volume limits over parts of the design."""
    n, m = int(case["n"]), int(case["m"])
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    w = 0.5 + 1.5 * torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    x = 0.2 + 0.4 * torch.rand(n, dtype=torch.float64, device=DEV, generator=g)
    part = torch.rand(n, m, dtype=torch.float64, device=DEV, generator=g)
    return w, x, part / n


def _mma_problem(w, x, part):
    return -w / (x * x) / x.numel(), [float(v) - 0.18 for v in (x @ part)]


def _prepare_mma(case, seed):
    w, x, part = _mma_inputs(case, seed)
    n, m = part.shape
    return {"opt": load_package().mma_t(x, n, m, 1.0, 0.0, 1000.0, 1.0, 1e-3, 1.0), "w": w, "x0": x, "x": x.clone(),
            "part": part}


def _run_mma(s):
    x = s["x"].copy_(s["x0"])
    df0, f = _mma_problem(s["w"], x, s["part"])
    s["opt"].update(1, x, df0, f, s["part"])
    return x


def _exact_mma(case, seed):
    """Svanberg's subproblem by its primal-dual interior-point method (2007)."""
    w, x0, part = _mma_inputs(case, seed)
    n, m = part.shape
    df0, f = _mma_problem(w, x0, part)
    G = part.T
    c01, c09, c101 = (float(np.float32(v)) for v in (0.1, 0.9, 1.01))
    a0, a, c, d = 1.0, np.zeros(m), np.full(m, 1000.0), np.ones(m)
    xr = 1.0 - 1e-3
    lo, up = x0 - 0.5 * xr, x0 + 0.5 * xr
    al = torch.maximum((lo + 0.1 * (x0 - lo)).clamp(min=1e-3), x0 - 0.5 * xr)
    be = torch.minimum((up - c01 * (up - x0)).clamp(max=1.0), x0 + 0.5 * xr)
    r = 1e-5 / max(1e-5, xr)
    pos, neg = (lambda v: v.clamp(min=0)), (lambda v: (-v).clamp(min=0))
    ux2, xl2 = (up - x0) ** 2, (x0 - lo) ** 2
    p0, q0 = ux2 * (1.001 * pos(df0) + 0.001 * neg(df0) + r), xl2 * (0.001 * pos(df0) + 1.001 * neg(df0) + r)
    Pm, Qm = ux2 * (1.001 * pos(G) + 0.001 * neg(G) + r), xl2 * (0.001 * pos(G) + 1.001 * neg(G) + r)
    host = lambda v: v.cpu().numpy()  # noqa: E731
    b = host((Pm / (up - x0) + Qm / (x0 - lo)).sum(1)) - np.array(f)
    dev = lambda v: torch.as_tensor(v, device=DEV)  # noqa: E731

    def resid(x, xsi, eta, y, z, lam, s, mu, zeta, eps):
        ux, xl, L = up - x, x - lo, dev(lam)
        big = [(p0 + L @ Pm) / ux ** 2 - (q0 + L @ Qm) / xl ** 2 - xsi + eta, xsi * (x - al) - eps,
               eta * (be - x) - eps]
        g = host((Pm / ux + Qm / xl).sum(1))
        small = np.concatenate([c + d * y - lam - mu, [a0 - zeta - lam @ a], g - a * z - y + s - b, mu * y - eps,
                                [zeta * z - eps], lam * s - eps])
        return (math.sqrt((small ** 2).sum() + sum(float((v * v).sum()) for v in big)),
                max(np.abs(small).max(), max(float(v.abs().max()) for v in big)))

    x = 0.5 * (al + be)
    xsi, eta = (1.0 / (x - al)).clamp(min=1.0), (1.0 / (be - x)).clamp(min=1.0)
    y, z, zeta, lam, s, mu = np.ones(m), 1.0, 1.0, np.ones(m), np.ones(m), np.maximum(1.0, 0.5 * c)
    eps, last = 1.0, c09 * 1e-9 * math.sqrt(m + n)
    while eps > last:
        norm, top = resid(x, xsi, eta, y, z, lam, s, mu, zeta, eps)
        for _ in range(100):
            if top < eps:
                break
            ux, xl, L = up - x, x - lo, dev(lam)
            pl, ql = p0 + L @ Pm, q0 + L @ Qm
            delx = pl / ux ** 2 - ql / xl ** 2 - eps / (x - al) + eps / (be - x)
            diag = 2 * (pl / ux ** 3 + ql / xl ** 3) + xsi / (x - al) + eta / (be - x)
            GG = Pm / ux ** 2 - Qm / xl ** 2
            dely, delz = c + d * y - lam - eps / y, a0 - lam @ a - eps / z
            dellam = host((Pm / ux + Qm / xl).sum(1)) - a * z - y - b + eps / lam
            A = np.zeros((m + 1, m + 1))
            A[:m, :m] = host((GG / diag) @ GG.T) + np.diag(s / lam + 1.0 / (d + mu / y))
            A[:m, m] = A[m, :m] = a
            A[m, m] = -zeta / z
            sol = np.linalg.solve(A, np.append(dellam + dely / (d + mu / y) - host(GG @ (delx / diag)), delz))
            dl, dz = sol[:m], sol[m]
            dx = -(delx + dev(dl) @ GG) / diag
            dy = (dl - dely) / (d + mu / y)
            dxsi, deta = -xsi + (eps - dx * xsi) / (x - al), -eta + (eps + dx * eta) / (be - x)
            dmu, dzeta, ds = -mu + (eps - mu * dy) / y, -zeta + (eps - zeta * dz) / z, -s + (eps - dl * s) / lam
            ratios = [float((-c101 * u / v).max()) for u, v in ((dxsi, xsi), (deta, eta), (dx, x - al), (-dx, be - x))]
            ratios += list(-c101 * np.concatenate([dy / y, dl / lam, dmu / mu, ds / s, [dz / z, dzeta / zeta]]))
            step = 1.0 / max(1.0, max(ratios))
            old, new = (x, xsi, eta, y, z, lam, s, mu, zeta), 2 * norm
            for _ in range(50):
                x, xsi, eta, y, z, lam, s, mu, zeta = (
                    o + step * v for o, v in zip(old, (dx, dxsi, deta, dy, dz, dl, ds, dmu, dzeta)))
                new, top = resid(x, xsi, eta, y, z, lam, s, mu, zeta, eps)
                step /= 2
                if new <= norm:
                    break
            norm = new
        eps *= 0.1
    return x


# ---------------------------------------------------------------------------
_KINDS = {
    "solve": (_prepare_solve, _run_solve, _exact_solve),
    "sequence": (_prepare_sequence, _run_sequence, _exact_sequence),
    "filter": (_prepare_filter, _run_filter, _exact_filter),
    "operator": (_prepare_operator, _run_operator, _exact_operator),
    "inner": (_prepare_operator, _run_inner, _exact_operator),
    "residuals": (_prepare_residuals, _run_residuals, _exact_residuals),
    "dealias": (_prepare_dealias, _run_dealias, _exact_dealias),
    "advect": (_prepare_advect, _run_advect, _exact_advect),
    "mma": (_prepare_mma, _run_mma, _exact_mma),
}


def prepare(case, seed):
    return {"kind": case["kind"], **_KINDS[case["kind"]][0](case, seed)}


def run(state):
    return _KINDS[state["kind"]][1](state)


def exact(case, seed):
    return _KINDS[case["kind"]][2](case, seed)


def work(case):
    """Doubles (or floats) per node that a pass reads and writes at the least,
    and the operations of one application of its operators."""
    if case["kind"] == "mma":
        # the problem's data (w, x, m constraint rows) in, the design out
        return {"bytes": 8.0 * case["n"] * (3 + case["m"]), "flops": 60.0 * case["n"] * (1 + case["m"])}
    lx, lxd = case["lx"], 3 * case["lx"] // 2
    n = case["ex"] * case["ey"] * case["ez"] * lx ** 3
    ax = 12 * lx + 20  # operations per node of one operator application
    grad = 6 * lx
    ratio = (lxd / lx) ** 3
    interp = 2 * (lxd / lx) * (lx + lx * (lxd / lx) + lx * (lxd / lx) ** 2)  # one field to the GL points
    words, flops = {
        # right-hand side in, solution out, six geometric factors and the mass term
        "solve": (9, ax), "sequence": (9, ax), "filter": (2 * 3 + 7, 2 * ax), "operator": (9, ax),
        "inner": (10, 2 * ax),
        # p, u, u_e, f (10), the 9 cofactors, 6 factors, B; four residuals out
        "residuals": (30, 4 * ax + 3 * 2 * 3 * grad),
        # u, Ub, f in, f out, the 9 cofactors at the GL points
        "dealias": (12 + 9 * ratio, 9 * interp + ratio * ((3 + 3) * 6 * lxd + 90)),
        # u, Ub, f in, three results out, the 9 cofactors
        "advect": (9 + 9 + 9 + 1, 2 * 6 * grad + 150 + 2 * 3 * grad),
    }[case["kind"]]
    size = 4 if case["kind"] == "inner" else 8
    return {"bytes": float(size * words * n), "flops": float(flops * n)}
