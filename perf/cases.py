"""The solver's work, as programs that use it call it: sizes, entry points, inputs, exact results.

Every case is one call of a public entry point of ``hprmat_b200`` (or, for the gradient, the
forward and backward of one loss): a single collision matrix over the range of orders N =
channels x mesh points, from two channels to the production size, both precisions, one and
several intervals, with wave functions and with a non-local potential; an energy scan by
either method; the potential gradient at several energies; a dense solve.

The systems are ``workloads``' coupled-channel potentials with seeded couplings.  Channel
thresholds lie on a grid of 3 MeV (levels of a rotational band) and energies 1.0 to 2.8 MeV
above a grid point, so that no channel is so close above its threshold that the Coulomb
functions fail.  A context is shared by the states of one case, as a program keeps one solver
for many potentials.
"""
from __future__ import annotations

import math
import weakref

import numpy as np
import torch

from hprmat_b200 import api, autograd, workloads

HM = workloads.HBAR2_2MU
LEVEL = 3.0  # MeV between the levels that set the channel thresholds

_contexts: "weakref.WeakValueDictionary" = weakref.WeakValueDictionary()


def listed():
    return [
        # two channels (NN scattering, tensor coupling): the smallest call, all latency
        {"name": "two_channels", "kind": "solve", "nch": 2, "nr": 60, "ns": 1, "rmax": 10.0, "charge": 0.0,
         "precision": "mixed", "device": False, "waves": 0, "nonlocal": False},
        # an ordinary small problem, all channels through the host interface
        {"name": "eight_channels", "kind": "solve", "nch": 8, "nr": 50, "ns": 1, "rmax": 10.0, "charge": 0.0,
         "precision": "mixed", "device": False, "waves": 0, "nonlocal": False},
        # R-matrix propagation over four intervals (12C + alpha's mesh)
        {"name": "propagation", "kind": "solve", "nch": 8, "nr": 25, "ns": 4, "rmax": 10.0, "charge": 6.0,
         "precision": "mixed", "device": False, "waves": 0, "nonlocal": False},
        # wave functions of two entrance channels, odd sizes
        {"name": "wave_functions", "kind": "solve", "nch": 21, "nr": 83, "ns": 1, "rmax": 15.0, "charge": 6.0,
         "precision": "mixed", "device": False, "waves": 2, "nonlocal": False},
        # a non-local potential (dense channel blocks)
        {"name": "nonlocal", "kind": "solve", "nch": 12, "nr": 60, "ns": 1, "rmax": 12.0, "charge": 6.0,
         "precision": "mixed", "device": False, "waves": 0, "nonlocal": True},
        # FP64 throughout, for a check of the mixed solver or an ill-conditioned potential
        {"name": "fp64", "kind": "solve", "nch": 20, "nr": 200, "ns": 1, "rmax": 20.0, "charge": 6.0,
         "precision": "fp64", "device": False, "waves": 0, "nonlocal": False},
        # a large problem on the production mesh, potential and result on the host
        {"name": "large", "kind": "solve", "nch": 32, "nr": 200, "ns": 1, "rmax": 20.0, "charge": 6.0,
         "precision": "mixed", "device": False, "waves": 0, "nonlocal": False},
        # the production size, potential and result on the device
        {"name": "production", "kind": "solve", "nch": 128, "nr": 200, "ns": 1, "rmax": 20.0, "charge": 6.0,
         "precision": "mixed", "device": True, "waves": 0, "nonlocal": False},
        # an energy scan of three J-pi blocks by the shifted method
        {"name": "scan_shifted", "kind": "scan", "method": "shifted", "blocks": "12,33,64", "nr": 60, "rmax": 20.0,
         "energies": 64},
        # an energy scan by one LU per energy (the default method)
        {"name": "scan_lu", "kind": "scan", "method": "lu", "blocks": "4,9,17,24", "nr": 60, "rmax": 20.0,
         "energies": 16},
        # the gradient of a fit to collision matrices at eight energies (forward and backward)
        {"name": "gradient", "kind": "gradient", "nch": 32, "nr": 100, "rmax": 20.0, "energies": 8},
        # the dense solve under the R-matrix path, called by itself on device arrays
        {"name": "dense", "kind": "dense", "n": 3000, "nrhs": 48, "precision": "mixed"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "solve", "scan", "gradient", "dense"])
    if kind == "scan":
        method = rng.choice(["shifted", "lu"])
        if method == "shifted":
            sizes, ne = [_log(rng, 4, 64) for _ in range(rng.randint(2, 4))], _log(rng, 24, 64)
        else:
            sizes, ne = [_log(rng, 4, 28) for _ in range(rng.randint(2, 4))], _log(rng, 6, 20)
        return {"kind": "scan", "method": method, "blocks": ",".join(map(str, sizes)), "nr": rng.randint(40, 64),
                "rmax": rng.choice([15.0, 20.0]), "energies": ne}
    if kind == "gradient":
        return {"kind": "gradient", "nch": _log(rng, 8, 36), "nr": rng.randint(50, 101), "rmax": rng.choice([15.0, 20.0]),
                "energies": rng.randint(3, 10)}
    if kind == "dense":
        return {"kind": "dense", "n": _log(rng, 200, 6000), "nrhs": _log(rng, 4, 130),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    case = {"kind": "solve", "ns": 1, "rmax": rng.choice([10.0, 12.0, 15.0, 20.0]), "charge": rng.choice([0.0, 6.0]),
            "precision": rng.choice(["mixed", "mixed", "fp64"]), "device": False, "waves": 0, "nonlocal": False}
    form = rng.choice(["plain", "plain", "plain", "propagation", "waves", "nonlocal"])
    if form == "propagation":
        return dict(case, nch=_log(rng, 2, 24), nr=rng.randint(20, 60), ns=rng.randint(2, 5))
    if form == "waves":
        return dict(case, nch=_log(rng, 2, 40), nr=rng.randint(40, 100), waves=rng.randint(1, 2))
    if form == "nonlocal":
        return dict(case, nch=_log(rng, 1, 16), nr=rng.randint(20, 60)) | {"nonlocal": True}
    n = _log(rng, 100, 6500 if case["precision"] == "fp64" else 13000)
    nr = rng.randint(50, 60) if n < 2000 else rng.randint(60, 200)
    return dict(case, nch=max(2, n // nr), nr=nr, device=rng.random() < 0.3)


# -- inputs ---------------------------------------------------------------------------------


def _system(rng, nch, nr, ns, rmax, charge):
    """One J-pi block: a ``Workload`` with seeded couplings and thresholds on the level grid."""
    re = rng.uniform(-5.0, 5.0, (nch, nch))
    c = np.triu(re + 1j * rng.uniform(-1.0, 0.0, (nch, nch)), 1)
    thr = LEVEL * ((np.arange(nch) * 5 + np.arange(nch) // 7) % 7)  # the entrance channel lowest
    p = workloads.PotentialParams(z1z2=charge, v0=rng.uniform(-55.0, -45.0), w0=rng.uniform(-12.0, -8.0))
    lval = (np.arange(nch) % 10).astype(np.int32)
    w = workloads.Workload("case", nch, nr, ns, rmax, 0.0, HM, lval, thr, c + c.T, p)
    r = np.concatenate([(s + workloads.lagrange_radii(nr, 1.0)) * (rmax / ns) for s in range(ns)])
    w.cpot = workloads.potential_matrix(r, nch, w.coupling, p, HM)
    return w


def _energies(rng, n, lo, hi):
    """n energies rising through the levels lo..hi-1 of the grid (so that the numbers of open
    channels do not depend on the seed)."""
    return np.sort(LEVEL * (lo + np.arange(n) * (hi - lo) // n) + rng.uniform(1.0, 2.8, n))


def _kinematics(w, energies):
    ks = [workloads.channel_kinematics(e, w.thresholds, w.hm, w.params.z1z2) for e in energies]
    return np.array([k[0] for k in ks]), np.array([k[1] for k in ks])


def _nonlocal(rng, nch, r):
    """Separable Gaussian couplings, complex strengths, symmetric in the channels."""
    s = rng.uniform(-2.0, 2.0, (nch, nch)) + 1j * rng.uniform(-0.3, 0.0, (nch, nch))
    s = np.triu(s) + np.triu(s, 1).T
    g = np.exp(-((r[:, None] - 1.5) ** 2 + (r[None, :] - 1.5) ** 2) / 2.0).reshape(-1)
    return np.asfortranarray(g[:, None, None] * s[None, :, :])


def _inputs(case, seed):
    """The host inputs of a case, from the seed alone."""
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "solve":
        w = _system(rng, case["nch"], case["nr"], case["ns"], case["rmax"], case["charge"])
        qk, eta = _kinematics(w, _energies(rng, 1, 3, 4))
        cpnl = _nonlocal(rng, w.nch, workloads.lagrange_radii(w.nr, w.rmax)) if case["nonlocal"] else None
        return {"w": w, "qk": qk[0], "eta": eta[0], "cpnl": cpnl}
    if case["kind"] == "scan":
        ws = [_system(rng, int(n), case["nr"], 1, case["rmax"], 6.0) for n in case["blocks"].split(",")]
        kin = [_kinematics(w, _energies(rng, case["energies"], 0, 10)) for w in ws]
        return {"blocks": [(w.lval, w.cpot, qk, eta) for w, (qk, eta) in zip(ws, kin)]}
    if case["kind"] == "gradient":
        w = _system(rng, case["nch"], case["nr"], 1, case["rmax"], 6.0)
        qk, eta = _kinematics(w, _energies(rng, case["energies"], 1, 8))
        targets = []
        for k in qk:  # collision matrices to fit: unit modulus on the diagonal, small couplings
            no = int((k > 0).sum())
            t = 0.02 * (rng.standard_normal((no, no)) + 1j * rng.standard_normal((no, no)))
            targets.append(np.diag(np.exp(2j * rng.uniform(0.0, math.pi, no))) + t + t.T)
        return {"w": w, "qk": qk, "eta": eta, "targets": targets}
    n = case["n"]
    gen = torch.Generator("cuda").manual_seed(seed * 7 + 5)
    a = torch.complex(*(torch.rand((n, n), dtype=torch.float64, device="cuda", generator=gen) - 0.5 for _ in range(2)))
    a += torch.diag(torch.full((n,), 2.0 * math.sqrt(n), dtype=torch.float64, device="cuda"))
    b = torch.complex(*(torch.rand((n, case["nrhs"]), dtype=torch.float64, device="cuda", generator=gen) for _ in range(2)))
    return {"a": a, "b": b}


def _context(precision, *mesh, copy=0):
    key = (precision, mesh, copy)
    ctx = _contexts.get(key)
    if ctx is None:
        ctx = api.Context(device=0, precision=precision, max_refine=6)  # room for a hard potential
        if mesh:
            ctx.rmat_ini(*mesh)
        _contexts[key] = ctx
    return ctx


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    if case["kind"] == "solve":
        s["ctx"] = _context(case["precision"], case["nr"], case["ns"], case["rmax"])
        if case["device"]:
            s["cpot"] = torch.from_numpy(np.ascontiguousarray(s["w"].cpot.T)).cuda()  # Fortran order
            s["cu"] = torch.zeros((case["nch"], case["nch"]), dtype=torch.complex128, device="cuda")
    elif case["kind"] == "scan":
        s["ctx"] = _context("mixed", case["nr"], 1, case["rmax"])
    elif case["kind"] == "gradient":
        s["pool"] = [_context("mixed", case["nr"], 1, case["rmax"], copy=k) for k in range(4)]
        s["cpot"] = torch.from_numpy(s["w"].cpot).cuda().requires_grad_(True)
        s["kin"] = list(zip(s["qk"], s["eta"]))
        s["targets"] = [torch.from_numpy(t).cuda() for t in s["targets"]]
    else:
        s["ctx"] = _context(case["precision"])
        s["a"] = s["a"].T.contiguous()  # column-major
        s["b"] = s["b"].T.contiguous()
    torch.cuda.synchronize()
    return s


# -- one pass -------------------------------------------------------------------------------


def run(s):
    case = s["case"]
    if case["kind"] == "solve":
        w, ctx = s["w"], s["ctx"]
        head = (w.nch, w.lval, s["qk"], s["eta"], w.rmax, w.nr, w.ns)
        if case["device"]:
            ctx.rmatrix_device(*head, s["cpot"].data_ptr(), w.nr * w.ns, w.nch, s["cu"].data_ptr())
            return {"u": s["cu"].T}
        if case["waves"]:
            cu, _, cf = ctx.rmatrix_wf(*head, w.cpot, list(range(1, case["waves"] + 1)), cpnl=s["cpnl"])
            return {"u": cu, "cf": cf}
        return {"u": ctx.rmatrix(*head, w.cpot, cpnl=s["cpnl"])[0]}
    if case["kind"] == "scan":
        out = s["ctx"].rmatrix_scan(s["blocks"], case["rmax"], case["nr"], method=case["method"])
        return [cu for cu, _, _ in out]
    if case["kind"] == "gradient":
        w = s["w"]
        us = autograd.collision_matrices(s["cpot"], s["pool"], w.lval, s["kin"], w.rmax, w.nr)
        loss = sum((u - t).abs().square().sum() for u, t in zip(us, s["targets"]))
        (grad,) = torch.autograd.grad(loss, s["cpot"])
        return {"u": [u.detach() for u in us], "grad": grad}
    x = s["b"].clone()
    torch.cuda.current_stream().synchronize()  # the context orders its work on its own stream
    n, nrhs = case["n"], case["nrhs"]
    s["ctx"].solve_linear_device(s["a"].data_ptr(), x.data_ptr(), n, nrhs)
    return {"x": x.T}


def work(case):
    """Each input read and each output written once (16 bytes a complex number); the arithmetic of
    an LU and its solves, or of one Hessenberg reduction and a solve per energy."""
    def lu(n, m):
        return 8.0 * n ** 3 / 3.0 + 8.0 * n * n * m

    if case["kind"] == "solve":
        nch, nr, ns = case["nch"], case["nr"], case["ns"]
        n = nch * nr
        size = nch * nch * (nr * ns + 1) + (nr * nr * nch * nch if case["nonlocal"] else 0) + case["waves"] * n * ns
        return {"bytes": 16.0 * size, "flops": ns * lu(n, nch if ns == 1 else 2 * nch)}
    if case["kind"] == "scan":
        size, flops = 0.0, 0.0
        for c in map(int, case["blocks"].split(",")):
            n, ne = c * case["nr"], case["energies"]
            size += 16.0 * c * c * (case["nr"] + ne)
            shifted = 40.0 * n ** 3 / 3.0 + ne * (4.0 * n * n + 4.0 * n * n * c)
            flops += min(shifted, ne * lu(n, c))
        return {"bytes": size, "flops": flops}
    if case["kind"] == "gradient":
        nch, n, ne = case["nch"], case["nch"] * case["nr"], case["energies"]
        return {"bytes": 16.0 * nch * nch * (2 * case["nr"] + ne), "flops": ne * (lu(n, nch) + 16.0 * n * nch * nch)}
    n, m = case["n"], case["nrhs"]
    return {"bytes": 16.0 * (n * n + 2 * n * m), "flops": lu(n, m)}


# -- exact results, in 64 bits --------------------------------------------------------------


def _sigma(l, eta):
    """arg Gamma(l + 1 + i eta): Stirling's series 30 above, and the recurrence down."""
    z = l + 1.0 + 1j * eta
    down = sum(np.angle(z + k) for k in range(30))
    z = z + 30.0
    s = (z - 0.5) * np.log(z) - z + 1.0 / (12 * z) - 1.0 / (360 * z ** 3) + 1.0 / (1260 * z ** 5)
    return s.imag - down


def _outgoing(l, eta, rho, closed):
    """H+ = G + iF (open) or the Whittaker function W_{-eta,l+1/2}(2 rho) (closed) and its
    derivative in rho: the asymptotic series far out, Taylor steps of the radial equation
    u'' = (l(l+1)/rho^2 + 2 eta/rho -+ 1) u inwards."""
    l = l.astype(np.float64)
    p = np.maximum(rho, 60.0 + l * (l + 1) + 2.0 * eta * eta)
    f = np.where(closed, -1.0, 1j)  # u ~ exp(f rho) (2 rho)^(-eta or -i eta) sum t_n
    e = np.where(closed, -eta, -1j * eta)
    t, u, du = np.ones_like(f), np.zeros_like(f), np.zeros_like(f)
    for n in range(60):
        u, du = u + t, du + t * (f + (e - n) / p)
        t = t * (e - n + l) * (e - n - l - 1) / (2.0 * f * (n + 1) * p)
    scale = np.exp(np.where(closed, -p - eta * np.log(2 * p),
                            1j * (p - eta * np.log(2 * p) - 0.5 * math.pi * l + _sigma(l, eta))))
    u, du = u * scale, du * scale
    s = np.where(closed, 1.0, -1.0)
    steps = max(1, int(np.ceil(np.max((p - rho) / 0.25))))
    h = (rho - p) / steps
    for _ in range(steps):
        a0, b0, c0 = l * (l + 1) + 2 * eta * p + s * p * p, 2 * eta + 2 * s * p, s
        a = [u, du]
        for n in range(28):
            v = (a0 - n * (n - 1)) * a[n] - 2 * p * (n + 1) * n * a[n + 1]
            if n > 0:
                v = v + b0 * a[n - 1]
            if n > 1:
                v = v + c0 * a[n - 2]
            a.append(v / (p * p * (n + 2) * (n + 1)))
        u, du = np.zeros_like(u), np.zeros_like(u)
        for n in range(len(a) - 1, -1, -1):
            u = u * h + a[n]
        for n in range(len(a) - 1, 0, -1):
            du = du * h + n * a[n]
        p = p + h
    return u, du


def _mesh(nr, ns, rmax):
    """Abscissas and weights on (0, 1), and per interval the kinetic + Bloch matrix, the Bloch
    products of the closed channels (times rmax/ns) and the boundary values q1, q2."""
    x, w = np.polynomial.legendre.leggauss(nr)
    order = np.argsort(x)
    x, w = (x[order] + 1) / 2, w[order] / 2
    a, m = rmax / ns, nr * (nr + 1.0)
    i = np.arange(1, nr + 1)
    sign = np.where((i[:, None] + i[None, :]) % 2 == 1, -1.0, 1.0)
    flip = np.where(i % 2 == 1, -1.0, 1.0)
    y = 1 - x
    dx = x[:, None] - x[None, :] + np.eye(nr)
    out = []
    for s in range(ns):
        if s == 0:
            t = (m + 1 + (x[:, None] + x[None, :] - 2 * np.outer(x, x)) / dx ** 2 - 1 / y[:, None] - 1 / y[None, :])
            t = t / np.sqrt(np.outer(x * y, x * y))
            np.fill_diagonal(t, (4 * m + 3 + (1 - 6 * x) / (x * y)) / (3 * x * y))
            q2 = 1 / np.sqrt(x * y) * flip * (-1.0 if nr % 2 else 1.0)
            q1 = np.zeros(nr)
            b = 1 / np.sqrt(np.outer(x * y, x * y)) * sign ** ns
        else:
            lo = np.tril(np.ones((nr, nr)), -1)
            q = x * y
            yy = (np.sqrt(q[None, :] / q[:, None] ** 3)
                  * (2 * np.outer(x, x) + 3 * x[:, None] - x[None, :] - 4 * x[:, None] ** 2) / dx ** 2)
            lb = np.sqrt(np.outer(x / y, x / y)) * (m - 1 / y[None, :])
            la = np.sqrt(np.outer(y / x, y / x)) * (-m + 1 / x[None, :])
            t = (yy + lb - la) * lo
            t = t + t.T + np.diag((m + 6 - 2 / q) / (3 * q) + x / y * (m - 1 / y) - y / x * (-m + 1 / x))
            q2 = np.sqrt(x / y) * flip * (-1.0 if nr % 2 else 1.0)
            q1 = -np.sqrt(y / x) * flip
            b = sign * (np.sqrt(np.outer(x / y, x / y)) / (s + 1) - np.sqrt(np.outer(y / x, y / x)) / s)
        out.append((t * sign / a ** 2, b / a, q1 / math.sqrt(a), q2 / math.sqrt(a)))
    return x, w, out


class _Block:
    """A channel block in 64 bits on the GPU: C(E) per interval, its solution, R and U."""

    def __init__(self, lval, nr, ns, rmax, qk, eta):
        self.nch, self.nr, self.ns, self.rmax = len(lval), nr, ns, rmax
        self.x, self.w, self.mesh = _mesh(nr, ns, rmax)
        self.lval = lval
        qk, eta = np.atleast_2d(qk), np.atleast_2d(eta)
        k = np.abs(qk)
        h, dh = _outgoing(np.broadcast_to(lval, qk.shape).ravel(), eta.ravel(), (k * rmax).ravel(), (qk < 0).ravel())
        self.h, self.rho_dh = h.reshape(qk.shape), dh.reshape(qk.shape) * k * rmax
        self.qk = qk

    def matrix(self, s, e, cpot, cpnl=None):
        """C(E) of interval s: a (nch, nr, nch, nr) tensor.  cpot: (nr, nch, nch) tensor."""
        nch, nr, qk = self.nch, self.nr, self.qk[e]
        t, b, _, _ = self.mesh[s]
        r = (s + self.x) * self.rmax / self.ns
        c = torch.zeros((nch, nr, nch, nr), dtype=torch.complex128, device="cuda")
        ts, bs = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (t, b))
        diag = self.lval[:, None] * (self.lval[:, None] + 1.0) / r ** 2 - (qk * np.abs(qk))[:, None]
        diag = torch.from_numpy(diag).cuda()
        shift = np.where(qk < 0, (self.rho_dh[e] / self.h[e]).real, 0.0) / (self.rmax / self.ns)
        for i in range(nch):
            c[i, :, i, :] = ts - float(shift[i]) * bs + torch.diag(diag[i])
        if cpnl is not None:
            f = np.sqrt(np.outer(self.w, self.w)) * self.rmax
            f = torch.from_numpy(np.ascontiguousarray(f)).cuda()
            c += cpnl.reshape(nr, nr, nch, nch).permute(2, 0, 3, 1) * f[None, :, None, :]
        return c + torch.einsum("icd,ij->cidj", cpot, torch.eye(nr, dtype=torch.complex128, device="cuda"))

    def solve(self, s, e, cpot, cpnl=None):
        """C^-1 [q1 | q2] of interval s (q2 alone when there is one interval)."""
        n = self.nch * self.nr
        _, _, q1, q2 = self.mesh[s]
        eye = np.eye(self.nch)
        q = np.concatenate([np.kron(eye, v[:, None]) for v in ((q1, q2) if self.ns > 1 else (q2,))], axis=1)
        b = torch.from_numpy(q).to(torch.complex128).cuda()
        return torch.linalg.solve(self.matrix(s, e, cpot, cpnl).reshape(n, n), b)

    def project(self, q, x):
        return torch.einsum("i,cim->cm", torch.from_numpy(np.ascontiguousarray(q)).to(x), x.reshape(self.nch, self.nr, -1))

    def forward(self, e, cpot, cpnl=None):
        """(U, R per interval, (R00, R01) per interval, X per interval)."""
        nch, nr, a = self.nch, self.nr, self.rmax / self.ns
        rs, parts, xs, r = [], [], [], None
        for s in range(self.ns):
            _, _, q1, q2 = self.mesh[s]
            x = self.solve(s, e, cpot[s * nr:(s + 1) * nr], cpnl)
            x1, x2 = (x[:, :nch], x[:, nch:]) if self.ns > 1 else (None, x)
            r11 = self.project(q2, x2)
            r00 = r01 = None
            if self.ns > 1:
                r00, r01 = self.project(q1, x1), self.project(q1, x2)
            if s == 0:
                r = r11 / a
            else:
                r = (r11 - r01.T @ torch.linalg.solve(r00 + s * a * r, r01)) / ((s + 1) * a)
            rs.append(r)
            parts.append((r00, r01))
            xs.append((x1, x2))
        op = np.flatnonzero(self.qk[e] > 0)
        h, d = (torch.from_numpy(v[e][op]).cuda() for v in (self.h, self.rho_dh))
        k = torch.from_numpy(self.qk[e][op]).cuda()
        at = torch.from_numpy(op).cuda()
        rt = r[at][:, at] * torch.sqrt(k[:, None] / k[None, :])
        u = torch.linalg.solve(torch.diag(h) - rt * d[None, :], torch.diag(h.conj()) - rt * d.conj()[None, :])
        return u, rs, parts, xs

    def waves(self, e, nw, u, rs, parts, xs):
        """(closed-channel amplitudes, internal wave functions) of the first nw open channels."""
        nch, nr, ns, a = self.nch, self.nr, self.ns, self.rmax / self.ns
        op, cl = np.flatnonzero(self.qk[e] > 0), np.flatnonzero(self.qk[e] < 0)
        d = torch.from_numpy(self.rho_dh[e][op]).cuda()
        k = torch.from_numpy(self.qk[e][op]).cuda()
        amp = (torch.diag(d.conj()) - u * d[:, None] * torch.sqrt(k[None, :] / k[:, None]))[:, :nw] / self.rmax
        v = torch.zeros((nch, nw), dtype=torch.complex128, device="cuda")
        v[torch.from_numpy(op).cuda()] = amp
        cf = torch.zeros((nr * ns, nch, nw), dtype=torch.complex128, device="cuda")
        closed = None
        for s in range(ns - 1, -1, -1):
            x1, x2 = xs[s]
            f = x2 @ v
            if s > 0:
                v = torch.linalg.solve(parts[s][0] + s * a * rs[s - 1], parts[s][1]) @ v
                f = f - x1 @ v
            if s == ns - 1:
                closed = self.project(self.mesh[s][3], f)[torch.from_numpy(cl).cuda()]
                closed = closed / torch.from_numpy(self.h[e][cl].real).cuda()[:, None]
            norm = torch.from_numpy(1 / np.sqrt(a * self.w)).cuda()
            cf[s * nr:(s + 1) * nr] = f.reshape(nch, nr, nw).permute(1, 0, 2) * norm[:, None, None]
        return closed, cf


def _padded(u, n):
    out = torch.zeros((n, n), dtype=torch.complex128, device=u.device)
    out[:u.shape[0], :u.shape[1]] = u
    return out


def exact(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "dense":
        return {"x": torch.linalg.solve(s["a"], s["b"])}
    if case["kind"] == "scan":
        out = []
        for lval, cpot, qk, eta in s["blocks"]:
            blk, cp = _Block(lval, case["nr"], 1, case["rmax"], qk, eta), torch.from_numpy(cpot).cuda()
            out.append(torch.stack([_padded(blk.forward(e, cp)[0], len(lval)) for e in range(len(qk))]))
        return out
    w = s["w"]
    blk = _Block(w.lval, w.nr, w.ns, w.rmax, s["qk"], s["eta"])
    cp = torch.from_numpy(w.cpot).cuda()
    if case["kind"] == "gradient":
        us, grad = [], torch.zeros_like(cp)
        for e, t in enumerate(s["targets"]):
            leaf = cp.clone().requires_grad_(True)
            u = blk.forward(e, leaf)[0]
            (g,) = torch.autograd.grad((u - torch.from_numpy(t).cuda()).abs().square().sum(), leaf)
            us.append(u.detach())
            grad += g
        return {"u": us, "grad": grad}
    cpnl = torch.from_numpy(s["cpnl"]).cuda() if s["cpnl"] is not None else None
    u, rs, parts, xs = blk.forward(0, cp, cpnl)
    cu = _padded(u, w.nch)
    if not case["waves"]:
        return {"u": cu}
    closed, cf = blk.waves(0, case["waves"], u, rs, parts, xs)
    no = u.shape[0]
    cu[no:no + closed.shape[0], :case["waves"]] = closed
    return {"u": cu, "cf": cf}
