"""What is measured when the speed of this library is measured: a dozen calls
of its public entry points over the range its users work in.

A case is a dict of plain values: ``op`` names the call, ``p`` the degree (one
for all directions), ``nu, nv, nw`` the elements per direction, and the rest the
call's options.  ``prepare`` makes what a program has in hand before the call
(geometry, operator, right-hand side), ``run`` is the call, ``work`` the bytes
and operations that it cannot do without, and ``exact`` what it should return,
from a restatement of the mathematics in 64 bits.

The solids are blocks with perturbed interior control points and random NURBS
weights (0.8 .. 1.2), clamped at one face: the patches of the benchmark, of the
serving stream and of the tests.
"""
import math
import time

import numpy as np
import torch

from yeti_b200 import _lib
from yeti_b200.gradient import grad_from_system_args
from yeti_b200.massmtrx import build_cmassmatrix
from yeti_b200.patches import u1_system_args
from yeti_b200.serve import Server
from yeti_b200.stiffmtrx_elemstorage import SYSTEM_ARG_NAMES, sys_linmat_lindef_static
from yeti_b200.wq import WQElasticity

E, NU, RHO = 1.0, 0.3, 7.8
CLAMP = {"w0": (0, 1, 2)}
GRAVITY = (0.0, 0.0, -1.0)
RTOL = 1e-10          # of the solves: the solutions agree to about 1e-11
SERVE_RTOL = 1e-11    # of the served solves, whose Gaussian loads are rougher


def _case(op, p, nel, **more):
    return dict({"op": op, "p": p, "nu": nel[0], "nv": nel[1], "nw": nel[2]}, **more)


def listed():
    return [
        # one operator product on a small patch: launch latency
        dict(_case("apply", 2, (8, 8, 8), prec="f64"), name="apply f64 p2 8x8x8"),
        # the product inside every FP32 Krylov iteration of the benchmark
        dict(_case("apply", 3, (64, 64, 64), prec="f32"), name="apply f32 p3 64x64x64"),
        # a ragged mesh of a higher degree in FP64, as residual checks run it
        dict(_case("apply", 4, (61, 47, 29), prec="f64"), name="apply f64 p4 61x47x29"),
        # a new operator with its diagonal and load: each step of a design loop
        dict(_case("setup", 3, (32, 24, 28)), name="setup p3 32x24x28"),
        # the benchmark's solve: mixed precision, Jacobi
        dict(_case("solve", 3, (64, 64, 64), precond="jacobi"), name="solve jacobi p3 64x64x64"),
        # the large block, mixed precision, fast diagonalisation
        dict(_case("solve", 4, (128, 128, 32), precond="fd"), name="solve fd p4 128x128x32"),
        # one request of the serving stream: set up, solve, return on the host
        dict(_case("serve", 3, (21, 17, 25), nrhs=4), name="serve p3 21x17x25"),
        # the cantilever as the drop-in is called: host arrays in and out
        dict(_case("assemble", 2, (16, 4, 4), kernel="pairs", device=False),
             name="assemble p2 16x4x4"),
        # larger solids, the COO arrays left on the device
        dict(_case("assemble", 3, (16, 16, 16), kernel="pairs", device=True),
             name="assemble p3 16x16x16"),
        dict(_case("assemble", 4, (12, 12, 12), kernel="sumfact", device=True),
             name="assemble sumfact p4 12^3"),
        # shape optimisation: the adjoint gradient of a thin solid
        dict(_case("gradient", 2, (32, 32, 2)), name="gradient p2 32x32x2"),
        # the mass matrix of a mid-size ragged mesh
        dict(_case("mass", 3, (13, 9, 11)), name="mass p3 13x9x11"),
    ]


def _between(rng, lo, hi):
    """lo .. hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["apply", "apply", "setup", "solve", "solve", "serve", "assemble",
                     "assemble", "assemble", "gradient", "mass"])

    def nel(lo, hi):
        return tuple(_between(rng, lo, hi) for _ in range(3))
    if op == "apply":
        return _case(op, rng.choice([2, 3, 4]), nel(8, 64), prec=rng.choice(["f32", "f64"]))
    if op == "setup":
        return _case(op, rng.choice([2, 3]), nel(8, 40))
    if op == "solve":
        if rng.random() < 0.4:
            return _case(op, rng.choice([2, 3]), nel(16, 48), precond="jacobi")
        return _case(op, rng.choice([2, 3, 4]),
                     (_between(rng, 16, 128), _between(rng, 16, 128), _between(rng, 8, 32)),
                     precond="fd")
    if op == "serve":
        return _case(op, rng.choice([2, 3]), nel(4, 32), nrhs=rng.randint(1, 8))
    if op == "assemble":
        kind = rng.choice(["host", "pairs", "sumfact"])
        if kind == "host":
            return _case(op, 2, (_between(rng, 4, 24), _between(rng, 2, 8), _between(rng, 2, 8)),
                         kernel="pairs", device=False)
        if kind == "pairs":
            return _case(op, rng.choice([2, 3]), nel(4, 16), kernel="pairs", device=True)
        return _case(op, rng.choice([3, 4]), nel(4, 12), kernel="sumfact", device=True)
    if op == "gradient":
        return _case(op, 2, (_between(rng, 6, 32), _between(rng, 6, 32), rng.randint(1, 4)))
    return _case(op, rng.choice([2, 3]), nel(4, 16))


# ------------------------------------------------------------------- inputs
def _patch(case, seed):
    """A block of unit elements' aspect: Greville control points, the interior
    ones moved by up to a tenth of an element, weights U(0.8, 1.2)."""
    rng = np.random.default_rng([seed, 17])
    p, nel = case["p"], (case["nu"], case["nv"], case["nw"])
    size = [n / max(nel) for n in nel]
    g = []
    for d in range(3):
        kv = _knots(p, nel[d])
        g.append(size[d] * np.array([kv[i + 1:i + p + 1].mean() for i in range(p + nel[d])]))
    W, V, U = np.meshgrid(g[2], g[1], g[0], indexing="ij")
    cps = np.stack([U, V, W])
    for d in range(3):
        h = size[d] / nel[d]
        cps[d][1:-1, 1:-1, 1:-1] += rng.uniform(-0.1 * h, 0.1 * h, cps[d][1:-1, 1:-1, 1:-1].shape)
    return {"p": (p, p, p), "nel": nel, "cps": np.ascontiguousarray(cps.reshape(3, -1)),
            "weights": rng.uniform(0.8, 1.2, cps[0].size)}


def _rhs(case, seed):
    """Gaussian right-hand sides of a serving request (host)."""
    n = 3 * math.prod(case["p"] + case[k] for k in ("nu", "nv", "nw"))
    return np.random.default_rng([seed, 23]).standard_normal((case["nrhs"], n))


def _field(case, seed, dtype):
    """A Krylov vector (component-major): Gaussian."""
    n = 3 * math.prod(case["p"] + case[k] for k in ("nu", "nv", "nw"))
    u = np.random.default_rng([seed, 29]).standard_normal(n)
    return torch.from_numpy(u.astype(dtype))


def _bending(patch, seed):
    """A displacement state of the gradient's solid: bending and stretching of
    a tenth of its size, with 1 % noise; (3, nb_cp)."""
    x, y, z = patch["cps"]
    rng = np.random.default_rng([seed, 31])
    a, b, c = rng.uniform(0.5, 1.0, 3)
    u = np.stack([0.1 * a * x - 0.2 * c * x * z, -0.03 * a * y + 0.05 * b * x * y,
                  0.1 * c * x * x + 0.02 * b * y])
    return u + 0.001 * rng.standard_normal(u.shape)


def _system(case, patch):
    """The 38 arguments of the assembly: one end clamped, a load on the other."""
    return u1_system_args(patch, E=E, nu=NU, rho=RHO, clamp_u0=True, load_u1=(3, -1.0))


def _mass_args(case, patch):
    d = dict(zip(SYSTEM_ARG_NAMES, _system(case, patch)))
    return [d[k] for k in ("activeElement", "nb_data", "COORDS3D", "IEN", "nb_elem_patch", "Nkv",
                           "Ukv", "Nijk", "weight", "Jpqr", "ELT_TYPE", "PROPS", "JPROPS", "RHO",
                           "TENSOR", "ind_dof_free", "nb_dof_free", "MCRD", "NBINT", "NNODE")]


_kept = {}


def _server():
    """The program's one server."""
    if "server" not in _kept:
        _kept["server"] = Server(max_active=64)
    return _kept["server"]


def prepare(case, seed):
    ctx = _lib.default_context()
    ctx.set_stream(torch.cuda.current_stream())
    patch = _patch(case, seed)
    op = case["op"]
    s = {"case": case, "patch": patch}
    if op == "apply":
        s["op"] = WQElasticity(patch, E, NU, CLAMP, precisions=case["prec"])
        s["u"] = _field(case, seed, np.float32 if case["prec"] == "f32" else np.float64).cuda()
    elif op == "solve":
        s["op"] = WQElasticity(patch, E, NU, CLAMP, precisions="both")
        s["b"] = torch.from_numpy(s["op"].eval_bodyforce_vector(GRAVITY)).cuda()
    elif op == "serve":
        s["rhs"] = _rhs(case, seed)
        _server()
    elif op == "assemble":
        s["args"] = _system(case, patch)
    elif op == "gradient":
        s["args"] = _system(case, patch)
        s["sol"] = _bending(patch, seed)
        s["adj"] = 0.5 * s["sol"][None]
    elif op == "mass":
        s["args"] = _mass_args(case, patch)
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "apply":
        return s["op"].eval_Ku(s["u"], precision=case["prec"])
    if op == "setup":
        w = WQElasticity(s["patch"], E, NU, CLAMP, precisions="both")
        return w.diag(), w.eval_bodyforce_vector(GRAVITY)
    if op == "solve":
        return s["op"].pcg(s["b"], rtol=RTOL, mixed=True, precond=case["precond"])[0]
    if op == "serve":
        srv = _server()
        t = srv.submit(s["patch"], E, NU, CLAMP, s["rhs"], rtol=SERVE_RTOL, precond="fd",
                       method="bicgstab")
        return srv.wait(t)[0]
    if op == "assemble":
        return sys_linmat_lindef_static(*s["args"], device_out=case["device"],
                                        element_kernel=case["kernel"])
    if op == "gradient":
        return grad_from_system_args(s["args"], s["sol"], s["adj"], include_surface=True)
    return build_cmassmatrix(*s["args"], device_out=True)


# --------------------------------------------------------------------- work
def _sizes(case):
    p = case["p"]
    nel = [case[k] for k in ("nu", "nv", "nw")]
    ndof = 3 * math.prod(p + n for n in nel)
    nqp = math.prod(2 * p + 2 * n - 1 for n in nel)
    return p, nel, ndof, nqp


def _product_flops(p, nqp):
    # per point: 9 derivatives and 27 channels through one-dimensional sums of
    # p+1 terms along u (the sums along v and w are shared by the points of a
    # row), and the 9x9 coefficient
    return 2.0 * nqp * (81 + (p + 1) * (9 + 27))


def work(case):
    p, nel, ndof, nqp = _sizes(case)
    op = case["op"]
    nelem, nn = math.prod(nel), (p + 1) ** 3
    slots = nelem * (9 * nn * (nn - 1) // 2 + 6 * nn)
    if op == "apply":
        es = 4 if case["prec"] == "f32" else 8
        return {"bytes": es * (45.0 * nqp + 2 * ndof), "flops": _product_flops(p, nqp)}
    if op == "setup":
        # both precisions of the coefficients written; geometry, diagonal, load
        return {"bytes": 12.0 * 45 * nqp + 8.0 * (ndof + 4 * ndof // 3 + 2 * ndof),
                "flops": 2.0 * nqp * (16 * (p + 1) + 300)}
    if op == "solve":
        # iterations of the method on these blocks to the tolerance: Jacobi
        # grows with the mesh, fast diagonalisation does not
        its = 16 * max(nel) if case["precond"] == "jacobi" else 50
        vectors = 14 if case["precond"] == "jacobi" else 12
        fd = 0.0 if case["precond"] == "jacobi" else 4.0 * ndof * sum(p + n for n in nel)
        return {"bytes": its * 4.0 * (45.0 * nqp + (2 + vectors) * ndof),
                "flops": its * (_product_flops(p, nqp) + fd)}
    if op == "serve":
        its = 30 * case["nrhs"]
        return {"bytes": 8.0 * (45.0 * nqp + 2 * case["nrhs"] * ndof) +
                its * 2 * 8.0 * (45.0 * nqp + 10 * ndof),
                "flops": its * 2 * (_product_flops(p, nqp) + 4.0 * ndof * sum(p + n for n in nel))}
    if op == "assemble":
        # value, row and column of every slot; the isotropic 3x3 blocks
        flops = (nelem * nn * (nn + 1) / 2.0 * nn * 48 if case["kernel"] == "pairs" else
                 nelem * 9.0 * (p + 1) ** 6 * (p + 1) * 4)
        return {"bytes": 16.0 * slots + 8.0 * (2 * ndof + 2 * nelem * nn), "flops": flops}
    if op == "gradient":
        return {"bytes": 8.0 * 5 * ndof + 12.0 * nelem * nn, "flops": nelem * nn * nn * 3.0 * 200}
    return {"bytes": 16.0 * slots + 8.0 * (ndof + 2 * nelem * nn),
            "flops": nelem * nn * (nn + 1) / 2.0 * nn * 3}


# -------------------------------------------------- the same, in 64 bits
def _knots(p, nel):
    return np.concatenate([np.zeros(p + 1), np.arange(1, nel) / nel, np.ones(p + 1)])


def _splines(p, nel, x):
    """All B-splines of degree p on nel uniform elements at x, and their first
    derivatives: (p + nel, len(x)) each (Cox-de Boor)."""
    U = _knots(p, nel)
    span = np.minimum((x * nel).astype(int), nel - 1) + p
    N = np.zeros((len(U) - 1, len(x)))
    N[span, np.arange(len(x))] = 1.0
    dN = None
    for q in range(1, p + 1):
        def over(i, q=q):
            d = U[i + q] - U[i]
            return 1.0 / d if d > 0 else 0.0
        M = np.zeros((len(U) - 1 - q, len(x)))
        D = np.zeros_like(M)
        for i in range(len(M)):
            a, b = over(i), over(i + 1)
            M[i] = (x - U[i]) * a * N[i] + (U[i + q + 1] - x) * b * N[i + 1]
            D[i] = q * (a * N[i] - b * N[i + 1])
        N, dN = M, D
    return N, dN


def _wq_rule(p, nel):
    """The weighted-quadrature rule of one direction: p+2 points in the first
    and last element, the ends and the middle of the others; per test function
    the least-norm weights at the points of its support that integrate it (or
    its derivative) exactly against the trial space (of degree p, or p-1 for
    derivatives of trial functions)."""
    parts = []
    for e in range(nel):
        m = p + 2 if e in (0, nel - 1) else 3
        parts.append((e + np.arange(m) / (m - 1)) / nel)
    x = np.concatenate([parts[0]] + [q[1:] for q in parts[1:]])
    xg, wg = np.polynomial.legendre.leggauss(p + 1)
    xc = np.concatenate([(e + 0.5 * (xg + 1)) / nel for e in range(nel)])
    wc = np.tile(0.5 * wg / nel, nel)
    B0, B1 = _splines(p, nel, x)
    C0, C1 = _splines(p, nel, xc)
    L0, LC = _splines(p - 1, nel, x)[0], _splines(p - 1, nel, xc)[0]
    R = {"B0": B0, "B1": B1}
    for trial, (at, on) in enumerate(((B0, C0), (L0, LC))):
        meet = (np.abs(on) > 1e-15).astype(float) @ (np.abs(C0) > 1e-15).T > 0
        for test, T in enumerate((C0, C1)):
            target = (on * wc) @ T.T
            W = np.zeros_like(B0)
            for i in range(len(B0)):
                cols, rows = np.flatnonzero(B0[i] > 1e-13), np.flatnonzero(meet[:, i])
                W[i, cols] = np.linalg.lstsq(at[np.ix_(rows, cols)], target[rows, i], rcond=None)[0]
            R["W%d%d" % (test, trial)] = W
    return R


class _Operator:
    """The weighted-quadrature elastic operator of a patch in 64 bits: B-spline
    trial and test functions, the exact NURBS geometry, one full tensor of
    points; fields are (3, w, v, u)."""

    def __init__(self, case, patch):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        nel = patch["nel"]
        p = patch["p"][0]
        self.n = [p + nel[d] for d in range(3)]
        rules = {n: {k: self._t(v) for k, v in _wq_rule(p, n).items()} for n in set(nel)}
        self.R = [rules[n] for n in nel]
        shape = self.n[::-1]
        w = self._t(patch["weights"]).reshape(shape)
        X = self._t(patch["cps"]).reshape([3] + shape)
        fields = [w * X[0], w * X[1], w * X[2], w]
        V = [self.fwd(f, None) for f in fields]
        D = [[self.fwd(f, l) for l in range(3)] for f in fields]
        J = torch.stack([torch.stack([(D[c][l] - V[c] / V[3] * D[3][l]) / V[3] for l in range(3)])
                         for c in range(3)])
        del V, D
        J = J.permute(2, 3, 4, 0, 1).contiguous()
        inv = torch.linalg.inv(J).permute(3, 4, 0, 1, 2).contiguous()     # dxi_k / dx_d
        self.det = torch.linalg.det(J).abs()
        self.inv = inv
        self.lam = E * NU / ((1 + NU) * (1 - 2 * NU))
        self.mu = E / (2 * (1 + NU))
        self.metric = [[(inv[k] * inv[l]).sum(0) for l in range(3)] for k in range(3)]
        self.free = torch.ones([3] + shape, dtype=torch.float64, device=self.dev)
        self.free[:, 0] = 0.0                                             # the face w = 0

    def _t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(self.dev)

    def _along(self, f, mats):
        """f (a, b, c) contracted with mats (u, v, w): rows of each are new."""
        t = f @ mats[0].T
        t = torch.matmul(mats[1], t)
        return (mats[2] @ t.reshape(t.shape[0], -1)).reshape(-1, t.shape[1], t.shape[2])

    def fwd(self, f, l):
        return self._along(f, [self.R[d]["B1" if d == l else "B0"].T for d in range(3)])

    def bwd(self, h, k, l):
        return self._along(h, [self.R[d]["W%d%d" % (d == k, d == l)] for d in range(3)])

    def apply(self, u):
        u = u.reshape(self.free.shape) * self.free
        out = torch.zeros_like(u)
        for l in range(3):
            F = [self.fwd(u[j], l) for j in range(3)]
            div = sum(self.inv[l][j] * F[j] for j in range(3))
            for k in range(3):
                cross = sum(self.inv[k][j] * F[j] for j in range(3))
                for i in range(3):
                    h = self.det * (self.lam * self.inv[k][i] * div + self.mu *
                                    (self.metric[k][l] * F[i] + self.inv[l][i] * cross))
                    out[i] += self.bwd(h, k, l)
        return (out * self.free).reshape(-1)

    def diag(self):
        out = torch.zeros_like(self.free)
        for i in range(3):
            for k in range(3):
                for l in range(3):
                    s = self.det * ((self.lam + self.mu) * self.inv[k][i] * self.inv[l][i] +
                                    self.mu * self.metric[k][l])
                    out[i] += self._along(s, [self.R[d]["W%d%d" % (d == k, d == l)] *
                                              self.R[d]["B1" if d == l else "B0"]
                                              for d in range(3)])
        return torch.where(self.free > 0, out, torch.ones_like(out)).reshape(-1)

    def force(self, f):
        out = torch.stack([self.bwd(f[i] * self.det, None, None) for i in range(3)])
        return (out * self.free).reshape(-1)

    def solve(self, b, until):
        """Jacobi-preconditioned BiCGSTAB, restarted with the true residual,
        to 1e-12; None when it is not there by the time `until`."""
        b = b * self.free.reshape(-1)
        dinv = 1.0 / self.diag()
        x = torch.zeros_like(b)
        for _ in range(40):
            r = b - self.apply(x)
            start = r.norm()
            if start <= 1e-12 * b.norm():
                return x
            hat, q, rho = r.clone(), r.clone(), r @ r
            for it in range(3000):
                y = dinv * q
                v = self.apply(y)
                alpha = rho / (hat @ v)
                s = r - alpha * v
                z = dinv * s
                t = self.apply(z)
                omega = (t @ s) / (t @ t)
                x = x + alpha * y + omega * z
                r = s - omega * t
                new = hat @ r
                q = r + (new / rho) * (alpha / omega) * (q - omega * v)
                rho = new
                if it % 10 == 9:
                    if time.perf_counter() > until:
                        return None
                    if not r.norm() > 1e-4 * start:
                        break
        return None


class _Elements:
    """Rational basis of every element of a patch at its (p+1)^3 Gauss points,
    in the connectivity's order of nodes (each index descending)."""

    def __init__(self, case, patch):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        p, nel = patch["p"][0], patch["nel"]
        self.p, self.nel, self.nn = p, nel, (p + 1) ** 3
        self.g, self.gw = np.polynomial.legendre.leggauss(p + 1)
        self.w = self._t(patch["weights"])
        self.n = [p + m for m in nel]
        e = np.stack(np.meshgrid(*(np.arange(m) for m in nel[::-1]), indexing="ij")[::-1])
        e = e.reshape(3, -1)                                   # u fastest
        a = np.arange(self.nn)
        loc = [a % (p + 1), a // (p + 1) % (p + 1), a // (p + 1) ** 2]
        f = [e[d][:, None] + p - loc[d][None, :] for d in range(3)]
        self.cp = f[0] + self.n[0] * (f[1] + self.n[1] * f[2])   # (elements, nodes)
        self.e, self.f = e, f
        self.cpt = torch.from_numpy(self.cp).to(self.dev)

    def _t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(self.dev)

    def basis(self, at, which):
        """R (elements, points, nodes) and dR/dparent (.., 3) at the parent
        points `at` ((points, 3)) of the elements `which`."""
        N = []
        for d in range(3):
            m = self.nel[d]
            x = ((np.arange(m)[:, None] + 0.5 * (at[:, d][None, :] + 1)) / m)
            x = np.minimum(x, 1.0)
            v, dv = _splines(self.p, m, x.ravel())
            cols = np.arange(m * len(at)).reshape(m, -1)[self.e[d][which]]   # (elements, points)
            rows = self.f[d][which]
            take = (rows[:, None, :], cols[:, :, None])
            N.append((self._t(v[take]), self._t(dv[take] / (2.0 * m))))
        w = self.w[self.cpt[which]][:, None, :]
        (a, da), (b, db), (c, dc) = N
        num = a * b * c * w
        S = num.sum(-1, keepdim=True)
        R = num / S
        dR = []
        for t in (da * b * c * w, a * db * c * w, a * b * dc * w):
            dR.append((t - R * t.sum(-1, keepdim=True)) / S)
        return R, torch.stack(dR, -1)

    def volume(self):
        i, j, k = np.meshgrid(*[np.arange(self.p + 1)] * 3, indexing="ij")
        at = np.stack([self.g[i.ravel()], self.g[j.ravel()], self.g[k.ravel()]], 1)
        wq = self._t(self.gw[i.ravel()] * self.gw[j.ravel()] * self.gw[k.ravel()])
        R, dR = self.basis(at, np.arange(len(self.cp)))
        return R, dR, wq

    def gradients(self, X, dR):
        """dR/dx and the Jacobian determinant for control points X (ncp, 3)."""
        J = torch.einsum("eac,eqad->eqcd", X[self.cpt], dR)
        return dR @ torch.linalg.inv(J), torch.linalg.det(J)

    def load(self, X):
        """The load vector of a unit traction -e_z on the face u = 1: (ncp, 3)."""
        p = self.p
        which = np.flatnonzero(self.e[0] == self.nel[0] - 1)
        j, k = (m.ravel() for m in np.meshgrid(np.arange(p + 1), np.arange(p + 1), indexing="ij"))
        at = np.stack([np.ones(len(j)), self.g[j], self.g[k]], 1)
        R, dR = self.basis(at, which)
        cp = self.cpt[which]
        T = torch.einsum("eac,eqad->eqcd", X[cp], dR)
        area = torch.linalg.cross(T[..., 1], T[..., 2]).norm(dim=-1) * self._t(self.gw[j] * self.gw[k])
        f = -(R * area[..., None]).sum(1)
        F = torch.zeros_like(X)
        z = torch.zeros(len(X), dtype=X.dtype, device=X.device).index_add(0, cp.reshape(-1), f.reshape(-1))
        return F + z[:, None] * torch.tensor([0.0, 0.0, 1.0], dtype=X.dtype, device=X.device)

    def slots(self, blocks):
        """The COO arrays from blocks(rows i, rows j) -> (elements, pairs, 3, 3)
        of the upper-triangle pairs, in the reference's order of slots."""
        nn = self.nn
        j = np.repeat(np.arange(nn), np.arange(1, nn + 1))
        i = np.concatenate([np.arange(m + 1) for m in range(nn)])
        r = np.tile([0, 1, 2], 3)                   # row component fastest
        c = np.repeat([0, 1, 2], 3)
        keep = ((i[:, None] < j[:, None]) | (r[None, :] <= c[None, :])).ravel()
        half = np.where((i[:, None] == j[:, None]) & (r[None, :] == c[None, :]), 0.5, 1.0)
        keep_t = torch.from_numpy(keep).to(self.dev)
        val = blocks(i, j).transpose(-1, -2).reshape(len(self.cp), -1, 9) * self._t(half)
        val = val.reshape(len(self.cp), -1)[:, keep_t].reshape(-1)
        row = (3 * self.cpt[:, i][:, :, None] + torch.from_numpy(r).to(self.dev)).to(torch.int32)
        col = (3 * self.cpt[:, j][:, :, None] + torch.from_numpy(c).to(self.dev)).to(torch.int32)
        n = len(self.cp)
        return (val, row.reshape(n, -1)[:, keep_t].reshape(-1),
                col.reshape(n, -1)[:, keep_t].reshape(-1))


def _stiffness_blocks(el, X, dR, wq):
    lam, mu = E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))
    G, det = el.gradients(X, dR)
    ne, nq, nn = G.shape[:3]
    A = G.permute(0, 2, 3, 1).reshape(ne, 3 * nn, nq)
    I = torch.matmul(A * (wq * det.abs())[:, None, :], A.transpose(1, 2))
    I = I.reshape(ne, nn, 3, nn, 3)                # integral of d_r R_a d_s R_b

    def blocks(i, j):
        P = I[:, i, :, j, :].movedim(0, 1)         # (elements, pairs, r, s)
        tr = P.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
        return lam * P + mu * P.transpose(-1, -2) + mu * tr * torch.eye(3, dtype=P.dtype, device=P.device)
    return blocks


def exact(case, seed):
    began = time.perf_counter()
    patch = _patch(case, seed)
    op = case["op"]
    if op in ("apply", "setup", "solve", "serve"):
        W = _Operator(case, patch)
        if op == "apply":
            u = _field(case, seed, np.float32 if case["prec"] == "f32" else np.float64)
            return W.apply(u.double().to(W.dev))
        if op == "setup":
            return W.diag(), W.force(GRAVITY)
        if op == "solve":
            return W.solve(W.force(GRAVITY), began + 18.0)
        got = []
        for b in _rhs(case, seed):
            got.append(W.solve(torch.from_numpy(b).to(W.dev), began + 18.0))
            if got[-1] is None:
                return None
        return torch.stack(got)
    el = _Elements(case, patch)
    X = el._t(patch["cps"].T)
    R, dR, wq = el.volume()
    if op == "assemble":
        val, row, col = el.slots(_stiffness_blocks(el, X, dR, wq))
        return val, row, col, el.load(X).reshape(-1)
    if op == "mass":
        det = el.gradients(X, dR)[1]
        M = torch.matmul((R * (RHO * wq * det)[..., None]).transpose(1, 2), R)
        eye = torch.eye(3, dtype=X.dtype, device=X.device)
        return el.slots(lambda i, j: M[:, i, j][..., None, None] * eye)
    # the adjoint gradient: derivatives of -u*.K(P) u and u*.F(P) with the
    # displacements u and u* = u/2 held
    lam, mu = E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))
    u = el._t(_bending(patch, seed).T)
    X.requires_grad_(True)
    G, det = el.gradients(X, dR)
    H = torch.einsum("eac,eqad->eqcd", u[el.cpt], G)
    eps = 0.5 * (H + H.transpose(-1, -2))
    tr = eps.diagonal(dim1=-2, dim2=-1).sum(-1)
    energy = ((lam * tr * tr + 2 * mu * (eps * eps).sum((-1, -2))) * wq * det.abs()).sum()
    inner, = torch.autograd.grad(-0.5 * energy, X)
    outer, = torch.autograd.grad((0.5 * u * el.load(X)).sum(), X)
    return inner.T[None], outer.T[None]
