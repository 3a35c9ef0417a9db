"""Performance cases of the fermion hot path, through its public entry points.

A case is one call (or the short sequence of calls) that a program built on this
library makes again and again: an operator application, a solve, a multi-shift
solve, a force of a molecular-dynamics step.  Links and fields are made on the
GPU from the seed and handed over as CLGBin-ordered device arrays, the way a
program with its own field storage does (``clg_gauge_import`` /
``clg_field_import`` with on_device = 1); results come back the same way
(``clg_field_export`` / ``clg_gauge_export``), so a pass ends with its whole
result in a device array.

Lattices, couplings and solver settings are those of this repository's
benchmark and tests: kappa = 0.1355, 2am = 0.02, boundary (+,+,+,-), Haar or
exp(i 0.25 H) links, true relative residual 1e-10 for every solve.
"""
import ctypes as C
import math

import torch

import cudalatticegauge_b200 as clg

KAPPA, MASS, EPS, TOL = 0.1355, 0.02, 0.25, 1e-10
BC = (1, 1, 1, -1)
DIMS = ("lx", "ly", "lz", "lt")
DEV = "cuda"
OPS = {"D": clg.EFO_F_D, "Ddagger": clg.EFO_F_Ddagger, "DDdagger": clg.EFO_F_DDdagger}
PREC = {"double": clg.DOUBLE, "single": clg.SINGLE, "half": clg.HALF}
SOLVERS = {"gmres": clg.CSLASolverGMRES, "bicgstab": clg.CSLASolverBiCGStab, "cg": clg.CSLASolverCG}
# the five lattices of uneven volume that one clg_solve_lattices call takes
UNEVEN = ((8, 8, 8, 8), (12, 12, 12, 12), (16, 16, 16, 16), (16, 16, 16, 32), (24, 24, 24, 16))


def _case(kind, dims, **more):
    return dict(kind=kind, **dict(zip(DIMS, dims)), **more)


def listed():
    return [
        # the smallest call: one D on the 8^4 lattice of the reference's own tests; latency and launches
        dict(_case("apply", (8, 8, 8, 8), fermion="wilson", op="D", prec="double", in_place=False, nrhs=1),
             name="wilson_d_8x8x8x8"),
        # D D^+ in place, as CField::ApplyOperator is called (action and heat bath of an HMC step)
        dict(_case("apply", (16, 16, 16, 32), fermion="wilson", op="DDdagger", prec="double", in_place=True, nrhs=1),
             name="wilson_dddag_16x16x16x32"),
        # D^+ in single precision on the largest lattice of the benchmark
        dict(_case("apply", (48, 48, 48, 24), fermion="wilson", op="Ddagger", prec="single", in_place=False, nrhs=1),
             name="wilson_ddag_single_48x48x48x24"),
        # staggered D D^+ in place on ragged extents (finite-temperature studies take any even extents)
        dict(_case("apply", (28, 22, 26, 18), fermion="staggered", op="DDdagger", prec="double", in_place=True, nrhs=1),
             name="staggered_dddag_28x22x26x18"),
        # the small solve: GMRES(12) with the default single-precision inner iterations on Haar links
        dict(_case("solve", (8, 8, 8, 8), solver="gmres", inner="single", op="D", nrhs=1, links="haar"),
             name="wilson_gmres_8x8x8x8"),
        # one source on an HMC-sized lattice, half-precision inner CG on the normal equations
        dict(_case("solve", (32, 32, 32, 16), solver="cg", inner="half", op="D", nrhs=1, links="exph"),
             name="wilson_cg_half_32x32x32x16"),
        # the headline: 28 sources (propagators and noise) in one batched solve
        dict(_case("solve", (32, 32, 32, 32), solver="cg", inner="half", op="D", nrhs=28, links="exph"),
             name="wilson_cg_half_28rhs_32x32x32x32"),
        # five lattices of uneven volume, four sources each, in one call
        dict(kind="lattices", largest=5, nrhs=4, inner="half", name="wilson_lattices_uneven"),
        # rational approximation: 12 shifts of the staggered even-site operator, mixed precision
        dict(_case("cgm", (32, 32, 32, 16), shifts=12, inner="single"), name="staggered_cgm_12_32x32x32x16"),
        # the reference's multi-shift FOM(30) with complex shifts of D
        dict(_case("fom", (8, 8, 8, 16), shifts=6, max_dim=30), name="wilson_fom_6_8x8x8x16"),
        # the Wilson force of one molecular-dynamics step: new links in, force out
        dict(_case("wilson_force", (32, 32, 32, 16), nrhs=1), name="wilson_force_32x32x32x16"),
        # the staggered rational force of one step: 12 poles, force out
        dict(_case("ks_force", (32, 32, 32, 16), poles=12), name="staggered_force_12_32x32x32x16"),
    ]


def _even(rng, lo, hi):
    return 2 * int(round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2)))))


def _dims(rng, lo, hi, vmax):
    while True:
        d = tuple(_even(rng, lo, hi) for _ in range(4))
        if math.prod(d) <= vmax:
            return d


def draw(rng):
    kind = rng.choice(("apply", "apply", "apply", "solve", "solve", "solve", "lattices", "cgm", "fom", "wilson_force",
                       "ks_force"))
    if kind == "apply":
        return _case(kind, _dims(rng, 6, 48, 48 ** 3 * 24), fermion=rng.choice(("wilson", "staggered")),
                     op=rng.choice(tuple(OPS)), prec=rng.choice(("double", "double", "single")),
                     in_place=rng.random() < 0.5, nrhs=rng.choice((1, 1, 1, 2, 3)))
    if kind == "solve":
        if rng.random() < 0.4:  # Haar links: every solver family, small to ordinary
            return _case(kind, _dims(rng, 6, 24, 1 << 17), solver=rng.choice(("gmres", "bicgstab", "cg")),
                         inner=rng.choice(("double", "single", "half")), op=rng.choice(("D", "Ddagger")),
                         nrhs=rng.choice((1, 1, 2, 4)), links="haar")
        return _case(kind, _dims(rng, 8, 32, 1 << 19), solver="cg", inner=rng.choice(("single", "half", "half")),
                     op=rng.choice(("D", "Ddagger")), nrhs=rng.choice((1, 1, 4, 12, 15)), links="exph")
    if kind == "lattices":
        return dict(kind=kind, largest=rng.randint(2, 5), nrhs=rng.randint(1, 6), inner=rng.choice(("single", "half")))
    if kind == "cgm":
        return _case(kind, _dims(rng, 8, 32, 1 << 19), shifts=rng.randint(6, 16), inner=rng.choice(("double", "single")))
    if kind == "fom":
        return _case(kind, _dims(rng, 6, 16, 1 << 14), shifts=rng.randint(3, 8), max_dim=rng.choice((20, 30)))
    if kind == "wilson_force":
        return _case(kind, _dims(rng, 6, 32, 1 << 19), nrhs=rng.choice((1, 1, 2)))
    return _case(kind, _dims(rng, 6, 32, 1 << 19), poles=rng.randint(6, 16))


# ------------------------------------------------------------------ inputs (torch, from the seed alone)
def _dims_of(c):
    return tuple(c[k] for k in DIMS)


def _gen(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + stream) & 0x7FFFFFFFFFFF)
    return g


def _gauss(g, shape):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=g, device=DEV, dtype=torch.float64)).mul_(math.sqrt(0.5))


def _mm(a, b):
    """product of 3x3 matrices stored row-major in the last two axes"""
    out = torch.empty_like(a)
    for i in range(3):
        out[..., i, :] = a[..., i, 0:1] * b[..., 0, :] + a[..., i, 1:2] * b[..., 1, :] + a[..., i, 2:3] * b[..., 2, :]
    return out


def _unitarise(m):
    """rows 0 and 1 orthonormal, row 2 = conj(row 0 x row 1): SU(3)"""
    for _ in range(2):
        a = m[..., 0, :]
        a /= a.abs().square().sum(-1, keepdim=True).sqrt()
        b = m[..., 1, :]
        b -= (a.conj() * b).sum(-1, keepdim=True) * a
        b /= b.abs().square().sum(-1, keepdim=True).sqrt()
    a, b = m[..., 0, :], m[..., 1, :]
    m[..., 2, 0] = (a[..., 1] * b[..., 2] - a[..., 2] * b[..., 1]).conj()
    m[..., 2, 1] = (a[..., 2] * b[..., 0] - a[..., 0] * b[..., 2]).conj()
    m[..., 2, 2] = (a[..., 0] * b[..., 1] - a[..., 1] * b[..., 0]).conj()
    return m


def _links(dims, seed, kind):
    """[V, 4, 3, 3] complex128 links, site-major (CLGBin order)"""
    g = _gen(seed, 1)
    m = _gauss(g, (math.prod(dims), 4, 3, 3))
    if kind == "haar":  # QR of a complex Gaussian matrix, determinant 1
        return _unitarise(m)
    # exp(i eps H), H traceless Hermitian with unit-normal Gell-Mann coefficients
    # (sum_a h_a lambda_a / 2): off-diagonal entries (h - i h') / 2
    h = torch.zeros_like(m)
    for i, j in ((0, 1), (0, 2), (1, 2)):
        z = m[..., i, j] * (math.sqrt(2.0) * 0.5)
        h[..., i, j] = z
        h[..., j, i] = z.conj()
    d3 = m[..., 0, 0].real * math.sqrt(2.0) * 0.5
    d8 = m[..., 1, 1].real * math.sqrt(2.0) * 0.5 / math.sqrt(3.0)
    h[..., 0, 0] = d3 + d8
    h[..., 1, 1] = d8 - d3
    h[..., 2, 2] = -2.0 * d8
    del m, d3, d8
    h *= 1j * EPS
    eye = torch.eye(3, device=DEV, dtype=torch.complex128)
    e = eye + h / 16.0
    for n in range(15, 0, -1):
        e = eye + _mm(h, e) / n
    return _unitarise(e)


def _field(dims, seed, stream, nc):
    return _gauss(_gen(seed, stream), (math.prod(dims), *nc))


# ------------------------------------------------------------------ handles
_ctx = None


def _context():
    """one context per program, as the library is meant to be used"""
    global _ctx
    if _ctx is None:
        _ctx = clg.Context(0)
    return _ctx


def _ptr(t):
    return C.c_void_p(t.data_ptr())


class _State:
    """What the program holds between calls; destroyed with it."""

    def __init__(self, case):
        self.case, self.ctx, self.owned = case, _context(), []

    def own(self, obj):
        self.owned.append(obj)
        return obj

    def lattice(self, dims):
        return self.own(clg.Lattice(self.ctx, dims, BC))

    def gauge(self, lat, links=None):
        u = self.own(clg.CFieldGaugeSU3(lat))
        if links is not None:
            self.import_gauge(u, links)
        return u

    def import_gauge(self, u, links):
        self.ctx.check(self.ctx.lib.clg_gauge_import(u.h, _ptr(links), clg.LAYOUT_CLGBIN, 1), "clg_gauge_import")

    def export_gauge(self, u, out):
        self.ctx.check(self.ctx.lib.clg_gauge_export(u.h, _ptr(out), 1), "clg_gauge_export")

    def import_field(self, f, t, rhs=0):
        self.ctx.check(self.ctx.lib.clg_field_import(f.h, rhs, _ptr(t), 1), "clg_field_import")

    def export_field(self, f, out, rhs=0):
        self.ctx.check(self.ctx.lib.clg_field_export(f.h, rhs, _ptr(out), 1), "clg_field_export")

    def __del__(self):
        for obj in reversed(self.owned):
            obj.close()
        self.owned = []


def _wilson(s, lat, **kw):
    return s.own(clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, **kw))


def _staggered(s, lat, mass=MASS, **kw):
    return s.own(clg.CFieldFermionKSSU3(lat, mass, **kw))


def _cgm_shifts(n):
    return [10.0 ** (-4 + 5 * k / (n - 1)) for k in range(n)]


def _fom_shifts(n):
    """the reference test's complex shifts first"""
    return [2.0, 1.0, 0.5, 1j, 0.5 + 0.5j, 1 - 1j, 3.0, 1.5 - 0.5j][:n]


def _poles(n):
    return [0.05 + 0.9 ** k for k in range(n)]


def _out(*shape):
    return torch.zeros(*shape, device=DEV, dtype=torch.complex128)


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind == "lattices":
        s.xs, s.bs, s.us, s.out = [], [], [], []
        for i, dims in enumerate(UNEVEN[: case["largest"]]):
            lat = s.lattice(dims)
            links = _links(dims, seed + 31 * i, "exph")
            b = _wilson(s, lat, nrhs=case["nrhs"])
            src = [_field(dims, seed + 31 * i, 2 + r, (4, 3)) for r in range(case["nrhs"])]
            torch.cuda.synchronize()
            s.us.append(s.gauge(lat, links))
            for r, t in enumerate(src):
                s.import_field(b, t, r)
            s.bs.append(b)
            s.xs.append(_wilson(s, lat, nrhs=case["nrhs"]))
            s.out.append(_out(case["nrhs"], lat.volume, 4, 3))
        s.solver = s.own(clg.CSLASolverCG(s.ctx, inner_precision=PREC[case["inner"]], tol_true_rel=TOL))
        torch.cuda.synchronize()
        return s
    dims = _dims_of(case)
    lat = s.lattice(dims)
    V = lat.volume
    links = _links(dims, seed, case.get("links", "exph"))
    torch.cuda.synchronize()
    if kind == "apply":
        prec, n = PREC[case["prec"]], case["nrhs"]
        make, nc = (_wilson, (4, 3)) if case["fermion"] == "wilson" else (_staggered, (3,))
        s.u = s.gauge(lat, links)
        s.src, s.dst = make(s, lat, precision=prec, nrhs=n), make(s, lat, precision=prec, nrhs=n)
        for r in range(n):
            t = _field(dims, seed, 2 + r, nc)
            torch.cuda.synchronize()
            s.import_field(s.src, t, r)
        s.out = _out(n, V, *nc)
    elif kind == "solve":
        n = case["nrhs"]
        s.u = s.gauge(lat, links)
        del links
        s.b, s.x = _wilson(s, lat, nrhs=n), _wilson(s, lat, nrhs=n)
        for r in range(n):
            t = _field(dims, seed, 2 + r, (4, 3))
            torch.cuda.synchronize()
            s.import_field(s.b, t, r)
        s.out = _out(n, V, 4, 3)
        more = {"MaxDim": 12} if case["solver"] == "gmres" else {}
        s.solver = s.own(SOLVERS[case["solver"]](s.ctx, inner_precision=PREC[case["inner"]], tol_true_rel=TOL, **more))
    elif kind == "cgm":
        s.u = s.gauge(lat, links)
        s.b = _staggered(s, lat, subset=clg.EVEN)
        t = _field(dims, seed, 2, (3,))
        torch.cuda.synchronize()
        s.import_field(s.b, t)
        s.shifts = _cgm_shifts(case["shifts"])
        s.xs = [_staggered(s, lat, subset=clg.EVEN) for _ in s.shifts]
        s.out = _out(len(s.shifts), V, 3)
        s.solver = s.own(clg.CMultiShiftCG(s.ctx, inner_precision=PREC[case["inner"]], tol_true_rel=TOL))
    elif kind == "fom":
        s.u = s.gauge(lat, links)
        s.b = _wilson(s, lat)
        t = _field(dims, seed, 2, (4, 3))
        torch.cuda.synchronize()
        s.import_field(s.b, t)
        s.shifts = _fom_shifts(case["shifts"])
        s.xs = [_wilson(s, lat) for _ in s.shifts]
        s.out = _out(len(s.shifts), V, 4, 3)
        s.solver = s.own(clg.CMultiShiftFOM(s.ctx, MaxDim=case["max_dim"], tol_true_rel=TOL))
    elif kind == "wilson_force":
        s.links, s.u, s.f = links, s.gauge(lat, links), s.gauge(lat)
        s.x, s.y = _wilson(s, lat, nrhs=case["nrhs"]), _wilson(s, lat, nrhs=case["nrhs"])
        for r in range(case["nrhs"]):
            for k, fld in enumerate((s.x, s.y)):
                t = _field(dims, seed, 2 + 2 * r + k, (4, 3))
                torch.cuda.synchronize()
                s.import_field(fld, t, r)
        s.out = _out(V, 4, 3, 3)
    else:
        s.u, s.f = s.gauge(lat, links), s.gauge(lat)
        s.num = _poles(case["poles"])
        s.phi, s.phid = [], []
        for k in range(case["poles"]):
            for j, lst in enumerate((s.phi, s.phid)):
                f = _staggered(s, lat, mass=0.0)
                t = _field(dims, seed, 2 + 2 * k + j, (3,))
                torch.cuda.synchronize()
                s.import_field(f, t)
                lst.append(f)
        s.out = _out(V, 4, 3, 3)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "apply":
        if case["in_place"]:
            s.src.CopyTo(s.dst)
            s.dst.ApplyOperator(OPS[case["op"]], s.u)
        elif case["op"] == "DDdagger":
            s.src.apply_to(clg.EFO_F_DDdagger, s.dst, s.u)
        else:
            s.src.apply_to(OPS[case["op"]], s.dst, s.u)
        for r in range(case["nrhs"]):
            s.export_field(s.dst, s.out[r], r)
    elif kind == "solve":
        s.solver.Solve(s.x, s.b, s.u, OPS[case["op"]])
        for r in range(case["nrhs"]):
            s.export_field(s.x, s.out[r], r)
    elif kind == "lattices":
        s.solver.SolveLattices(s.xs, s.bs, s.us, clg.EFO_F_D)
        for x, out in zip(s.xs, s.out):
            for r in range(case["nrhs"]):
                s.export_field(x, out[r], r)
    elif kind == "cgm":
        s.solver.Solve(s.xs, s.shifts, s.b, s.u, clg.OP_DDDAG_EE)
        for k, x in enumerate(s.xs):
            s.export_field(x, s.out[k])
    elif kind == "fom":
        s.solver.Solve(s.xs, s.shifts, s.b, s.u, clg.EFO_F_D)
        for k, x in enumerate(s.xs):
            s.export_field(x, s.out[k])
    elif kind == "wilson_force":
        s.import_gauge(s.u, s.links)
        s.f.InitialField(clg.GAUGE_ZERO)
        clg.CFieldFermionWilsonSquareSU3.DerivateDOperator(s.f, s.y, s.x, s.u)
        s.export_gauge(s.f, s.out)
    else:
        s.f.InitialField(clg.GAUGE_ZERO)
        clg.CFieldFermionKSSU3.DerivateD0(s.f, s.u, s.phi, s.phid, s.num)
        s.export_gauge(s.f, s.out)
    return s.out


# ------------------------------------------------------------------ what a pass cannot do without
def _site_bytes(prec, nc):
    return {"double": 16, "single": 8, "half": 4}[prec] * nc + (4 if prec == "half" else 0)


def _link_bytes(prec):
    """four links of a site: 18 reals FP64, 12 reals below"""
    return {"double": 576, "single": 192, "half": 96}[prec]


def _solve_work(V, nrhs, solver, inner, links):
    """CG on the normal equations: per iteration four half-lattice hops and the
    CG vectors (x, r, p read, x, r, p written; q and the odd vectors once each
    way), about 115 iterations (exp(i eps H) links); Haar links: about 20
    operator applications of two hops.  Links once per hop pair for all rhs."""
    v = _site_bytes(inner, 12)
    if links == "haar":
        its, hops, vec = (20, 2, 8) if solver != "cg" else (14, 4, 14)
    else:
        its, hops, vec = 115, 4, 14
    b = its * (hops / 2 * V * _link_bytes(inner) + vec * V / 2 * v * nrhs) + 6 * V * 192 * nrhs + V * 576
    return {"bytes": b, "flops": its * (hops * V / 2 * 1320 + V / 2 * 24 * 8) * nrhs}


def work(case):
    kind = case["kind"]
    if kind == "lattices":
        w = [_solve_work(math.prod(d), case["nrhs"], "cg", case["inner"], "exph") for d in UNEVEN[: case["largest"]]]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    V = math.prod(_dims_of(case))
    if kind == "apply":
        # the source and the links read once, the exported FP64 result written once
        nc, flops = (12, 1320 + 48) if case["fermion"] == "wilson" else (3, 570 + 12)
        n = case["nrhs"]
        return {"bytes": V * ((_site_bytes(case["prec"], nc) + 16 * nc) * n + _link_bytes(case["prec"])),
                "flops": V * flops * n * (2 if case["op"] == "DDdagger" else 1)}
    if kind == "solve":
        return _solve_work(V, case["nrhs"], case["solver"], case["inner"], case["links"])
    if kind == "cgm":
        # about 130 iterations, a third of them FP64: links once per iteration, r, p, q; x_k once
        n, its = case["shifts"], 130
        lo = _link_bytes(case["inner"]) / 4 * 4
        return {"bytes": V * (its / 3 * 576 + its * 2 / 3 * lo) + its * V / 2 * 5 * 36 + n * V * 72,
                "flops": its * V * 570}
    if kind == "fom":
        # two to three cycles of max_dim applications of D with their Gram-Schmidt (basis once per step)
        m, its = case["max_dim"], 40
        return {"bytes": its * V * (576 + 2 * 192) + its * m / 2 * V * 192 + case["shifts"] * V * 192 * 3,
                "flops": its * V * (1368 + m / 2 * 192)}
    n = case["nrhs"] if kind == "wilson_force" else case["poles"]
    if kind == "wilson_force":
        # X, Y and the new links read once, the exported force written once
        return {"bytes": V * (2 * 192 * n + 576 + 576), "flops": V * 4 * (36 * 8 * n + 27 * 8 + 60)}
    return {"bytes": V * (2 * 48 * n + 576 + 576), "flops": V * 4 * (18 * 8 * n + 54 * 8 + 60)}


def tolerance(case):
    kind = case["kind"]
    if kind == "apply":
        return {"rel": 1e-15, "max": 2e-14} if case["prec"] == "double" else {"rel": 3e-7, "max": 6e-6}
    if kind in ("wilson_force", "ks_force"):
        return {"rel": 1e-15, "max": 2e-14}
    # solves to a true relative residual of 1e-10: solutions within the condition number of that
    return {"rel": 5e-9, "max": 5e-7}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
def _gammas():
    out = []
    z = ((3, 3, 1, 1), (2, 0, 0, 2), (3, 1, 1, 3), (0, 0, 0, 0))
    for mu in range(4):
        g = torch.zeros(4, 4, dtype=torch.complex128, device=DEV)
        for r in range(4):
            g[r, 3 - r if mu < 2 else (r + 2) % 4] = 1j ** z[mu][r]
        out.append(g)
    return out


def _shift(v, mu, step, dims):
    """v(x + step mu) with the boundary sign; v: [n, Lx, Ly, Lz, Lt, ...]"""
    w = torch.roll(v, -step, mu + 1)
    if BC[mu] < 0:
        w.select(mu + 1, dims[mu] - 1 if step > 0 else 0).mul_(-1)
    return w


def _eta(mu, dims):
    x = [torch.arange(d, device=DEV).view([-1 if i == k else 1 for i in range(4)]) for k, d in enumerate(dims)]
    s = torch.zeros((1, 1, 1, 1), device=DEV, dtype=torch.int64)
    for k in range(mu):
        s = s + x[k]
    return 1.0 - 2.0 * (s % 2).double()


class _Exact:
    """D = 1 - kappa H (Wilson) and D = 2am + H (staggered) on [n, V, ...] fields"""

    def __init__(self, dims, links, fermion, param):
        self.dims, self.fermion, self.param = dims, fermion, param
        self.u = links.view(*dims, 4, 3, 3)
        self.g = _gammas() if fermion == "wilson" else None

    def hop(self, v, dagger=False):
        dims = self.dims
        v = v.reshape(v.shape[0], *dims, *v.shape[2:])
        out = torch.zeros_like(v)
        for mu in range(4):
            u = self.u[..., mu, :, :]
            if self.fermion == "wilson":
                sg = -1.0 if dagger else 1.0
                w = _shift(v, mu, 1, dims)
                w = w - sg * torch.einsum("rs,...sc->...rc", self.g[mu], w)
                out += torch.einsum("...ab,...sb->...sa", u, w)
                w = v + sg * torch.einsum("rs,...sc->...rc", self.g[mu], v)
                out += _shift(torch.einsum("...ba,...sb->...sa", u.conj(), w), mu, -1, dims)
            else:
                eta = _eta(mu, dims)[..., None]
                w = torch.einsum("...ab,...b->...a", u, _shift(v, mu, 1, dims))
                w = w - _shift(torch.einsum("...ba,...b->...a", u.conj(), v), mu, -1, dims)
                out += eta * w
        return out.reshape(v.shape[0], -1, *v.shape[5:])

    def D(self, v, dagger=False):
        if self.fermion == "wilson":
            return v - self.param * self.hop(v, dagger)
        return self.param * v + (-1.0 if dagger else 1.0) * self.hop(v)

    def op(self, name, v):
        if name == "DDdagger":
            return self.D(self.D(v, True))
        return self.D(v, name == "Ddagger")


def _cg(a, b, its=4000):
    """CG on a Hermitian positive operator, each right-hand side on its own, to 64-bit rounding"""
    shape = (-1, *([1] * (b.dim() - 1)))
    dot = lambda p, q: (p.conj() * q).real.flatten(1).sum(1)  # noqa: E731
    x, r, p = torch.zeros_like(b), b.clone(), b.clone()
    rr = dot(r, r)
    goal = rr * 1e-28
    for k in range(its):
        q = a(p)
        al = torch.where(rr > goal, rr / dot(p, q).clamp_min(1e-300), torch.zeros_like(rr))
        x += al.view(shape) * p
        r -= al.view(shape) * q
        new = dot(r, r)
        be = torch.where(rr > goal, new / rr.clamp_min(1e-300), torch.zeros_like(rr))
        rr = torch.where(rr > goal, new, rr)
        if k % 16 == 15 and bool((rr <= goal).all()):
            break
        p = r + be.view(shape) * p
    return x


def _ta(m):
    a = 0.5 * (m - m.mH)
    tr = a.diagonal(dim1=-2, dim2=-1).sum(-1) / 3.0
    return a - tr[..., None, None] * torch.eye(3, device=DEV, dtype=m.dtype)


def exact(case, seed):
    kind = case["kind"]
    if kind == "lattices":
        return None
    dims = _dims_of(case)
    V = math.prod(dims)
    if kind == "solve" and V * case["nrhs"] > 1 << 16 or kind == "cgm" and V * case["shifts"] > 1 << 18:
        return None
    links = _links(dims, seed, case.get("links", "exph"))
    if kind == "apply":
        nc = (4, 3) if case["fermion"] == "wilson" else (3,)
        e = _Exact(dims, links, case["fermion"], KAPPA if case["fermion"] == "wilson" else MASS)
        return torch.cat([e.op(case["op"], _field(dims, seed, 2 + r, nc)[None]) for r in range(case["nrhs"])])
    if kind == "solve":
        e = _Exact(dims, links, "wilson", KAPPA)
        b = torch.stack([_field(dims, seed, 2 + r, (4, 3)) for r in range(case["nrhs"])])
        dag = case["op"] == "Ddagger"
        return e.D(_cg(lambda v: e.D(e.D(v, not dag), dag), b), not dag)
    if kind == "cgm":
        e = _Exact(dims, links, "staggered", MASS)
        b = _field(dims, seed, 2, (3,)).view(*dims, 3).clone()
        par = sum(torch.arange(d, device=DEV).view([-1 if i == k else 1 for i in range(4)]) for k, d in enumerate(dims))
        b[(par % 2) == 1] = 0
        sh = torch.tensor(_cgm_shifts(case["shifts"]), device=DEV, dtype=torch.float64).view(-1, 1, 1)
        b = b.view(1, V, 3).expand(case["shifts"], V, 3).clone()
        return _cg(lambda v: e.op("DDdagger", v) + sh * v, b)
    if kind == "fom":
        e = _Exact(dims, links, "wilson", KAPPA)
        c = torch.tensor(_fom_shifts(case["shifts"]), device=DEV, dtype=torch.complex128).view(-1, 1, 1, 1)
        b = _field(dims, seed, 2, (4, 3))[None].expand(case["shifts"], V, 4, 3).clone()
        a, ah = lambda v: e.D(v) + c * v, lambda v: e.D(v, True) + c.conj() * v
        return ah(_cg(lambda v: a(ah(v)), b))
    u = links.view(*dims, 4, 3, 3)
    out = torch.zeros_like(u)
    if kind == "wilson_force":
        g = _gammas()
        for r in range(case["nrhs"]):
            x, y = (_field(dims, seed, 2 + 2 * r + k, (4, 3)).view(1, *dims, 4, 3) for k in (0, 1))
            for mu in range(4):
                xp, yp = _shift(x, mu, 1, dims)[0], _shift(y, mu, 1, dims)[0]
                l1 = yp - torch.einsum("rs,...sc->...rc", g[mu], yp)
                r2 = y[0] + torch.einsum("rs,...sc->...rc", g[mu], y[0])
                mid = torch.einsum("...sa,...sb->...ab", l1, x[0].conj()) + torch.einsum("...sa,...sb->...ab", xp, r2.conj())
                out[..., mu, :, :] += KAPPA * _ta(u[..., mu, :, :] @ mid)
        return out.view(V, 4, 3, 3)
    for k, a in enumerate(_poles(case["poles"])):
        p, pd = (_field(dims, seed, 2 + 2 * k + j, (3,)).view(1, *dims, 3) for j in (0, 1))
        for mu in range(4):
            t1 = torch.einsum("...ab,...b->...a", u[..., mu, :, :], _shift(p, mu, 1, dims)[0])
            t2 = torch.einsum("...ab,...b->...a", u[..., mu, :, :], _shift(pd, mu, 1, dims)[0])
            m = t1[..., :, None] * pd[0][..., None, :].conj() + p[0][..., :, None] * t2[..., None, :].conj()
            out[..., mu, :, :] -= _ta(a * _eta(mu, dims)[..., None, None] * m)
    return out.view(V, 4, 3, 3)
