"""The work that a program using this framework has it do, as cases to be timed.

A case is a dict of plain values.  Its ``kind`` names the path:

* ``mg``      one pressure solve through ``solver.New`` / ``GPUMG.solve`` on
              device arrays: the closed cavity, the tanh channel, a box with
              Dirichlet ends, the two-phase sphere (variable coefficient), the
              seven-brick mesh and boxes split into bricks; FP64 and mixed
              precision, with and without flexible CG, V and F cycles
* ``fft``     one direct solve of the FFT Poisson solver
* ``project`` one projection step of a staggered solver: explicit predictor,
              pressure right-hand side, FFT solve, velocity correction
* ``split``   one solve of the split Poisson solver (FFT corrections)
* ``unet``    one forward pass of the U-Net, or one training step

Sizes are those of the benchmark's and the tests' configurations, and others
of the same ranges.  Right-hand sides have the benchmark's distributions
(divergence of seeded N(0, 1) face velocities, N(0, 1) cell sources).
"""
from __future__ import annotations

import math

import numpy as np
import torch

V22 = {"cycle": "V", "pre": 2, "post": 2, "coarse": 1}


def _mg(name, mesh, n, precision, krylov, relTol, cycle=None):
    c = {"kind": "mg", "mesh": mesh, "n0": n[0], "n1": n[1], "n2": n[2], "precision": precision, "krylov": krylov,
         "relTol": relTol}
    c.update(cycle or V22)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        _mg("mg cavity 16 fp64", "cavity", (16, 16, 16), "fp64", "none", 1e-10),
        _mg("mg cavity 64 fp64", "cavity", (64, 64, 64), "fp64", "none", 1e-10),
        _mg("mg walls 96x192x24 F", "walls", (96, 192, 24), "fp64", "none", 1e-9,
            {"cycle": "F", "pre": 0, "post": 2, "coarse": 0}),
        _mg("mg seven bricks mixed", "bricks7", (1, 1, 1), "mixed", "fcg", 1e-8,
            {"cycle": "V", "pre": 2, "post": 2, "coarse": 0}),
        _mg("mg sphere 128 mixed", "sphere", (128, 128, 128), "mixed", "fcg", 1e-8),
        _mg("mg channel 256 mixed", "channel", (256, 256, 256), "mixed", "fcg", 1e-8),
        _mg("mg channel 256 fp64", "channel", (256, 256, 256), "fp64", "none", 1e-8),
        {"name": "fft channel 256", "kind": "fft", "bc": "PNP", "n0": 256, "n1": 256, "n2": 256},
        {"name": "project 128x96x64", "kind": "project", "bc": "NNN", "n0": 128, "n1": 96, "n2": 64},
        {"name": "split sphere 128", "kind": "split", "n0": 128, "n1": 128, "n2": 128, "ncorr": 3},
        {"name": "unet forward 256", "kind": "unet", "what": "forward", "n0": 256, "n1": 256, "n2": 256},
        {"name": "unet train 128", "kind": "unet", "what": "train", "n0": 128, "n1": 128, "n2": 128},
    ]


def draw(rng):
    kind = rng.choice(["mg", "mg", "mg", "mg", "mg", "fft", "fft", "project", "split", "unet"])
    if kind == "mg":
        mesh = rng.choice(["cavity", "channel", "channel", "walls", "sphere", "bricks"])
        precision, krylov = rng.choice([("fp64", "none"), ("mixed", "fcg"), ("mixed", "none"), ("fp64", "fcg")])
        if mesh == "bricks":
            # a box split into bricks along its first axis
            while True:
                n = [16 * rng.randint(2, 10), 16 * rng.randint(1, 8), 16 * rng.randint(1, 8)]
                if n[0] * n[1] * n[2] <= 1 << 19:
                    break
            c = _mg(None, mesh, n, precision, krylov, 1e-8, {"cycle": "V", "pre": 2, "post": 2, "coarse": 0})
            c["cut"] = 16 * rng.randint(1, n[0] // 16 - 1)
            return c
        # single bricks halve down to extents of 2 and 3 (2 along periodic axes)
        most = 1 << (21 if mesh == "sphere" else 24)
        base = 2 ** rng.uniform(4, 7 if mesh == "sphere" else 8)
        while True:
            n = []
            for d in range(3):
                sizes = (16, 32, 64, 128, 256) if mesh == "channel" and d != 1 else (16, 24, 32, 48, 64, 96, 128, 192, 256)
                t = math.log(base * 2 ** rng.uniform(-1, 1))
                n.append(min(sizes, key=lambda v: abs(math.log(v) - t)))
            if n[0] * n[1] * n[2] <= most:
                break
        cyc = None
        if mesh in ("cavity", "walls") and rng.random() < 0.3:
            cyc = {"cycle": "F", "pre": 0, "post": 2, "coarse": 0}
        return _mg(None, mesh, n, precision, krylov, rng.choice([1e-6, 1e-8]), cyc)
    if kind in ("fft", "project"):
        while True:
            n = [2 ** rng.randint(5, 9), int(round(2 ** rng.uniform(4.6, 8.6))), 2 ** rng.randint(5, 9)]
            if kind == "project":  # the step's solver context halves the extents down to 2 or 3
                n[1] = rng.choice([24, 32, 48, 64, 96, 128, 192, 256])
            if n[0] * n[1] * n[2] <= 1 << 24:
                break
        bc = "".join(rng.choice(s) for s in ("PNDM", "ND", "PNDM")) if kind == "fft" else rng.choice(["PNP", "NNN", "PNN"])
        return {"kind": kind, "bc": bc, "n0": n[0], "n1": n[1], "n2": n[2]}
    if kind == "split":
        n = [2 ** rng.randint(5, 7) for _ in range(3)]
        return {"kind": "split", "n0": n[0], "n1": n[1], "n2": n[2], "ncorr": rng.randint(1, 6)}
    what = rng.choice(["forward", "forward", "train"])
    most = 1 << (23 if what == "forward" else 20)
    while True:
        n = [8 * int(round(2 ** rng.uniform(1, 4.6))) for _ in range(3)]
        if n[0] * n[1] * n[2] <= most:
            break
    return {"kind": "unet", "what": what, "n0": n[0], "n1": n[1], "n2": n[2]}


# ---------------------------------------------------------------------------
# meshes (host arrays of vertex coordinates; no code of the package)
# ---------------------------------------------------------------------------
def _uniform(n, length=1.0):
    return length * np.arange(n + 1, dtype=np.float64) / n


def _tanh(n, gamma=2.0, length=1.0):
    y = 0.5 * (1.0 + np.tanh(gamma * (2.0 * np.arange(n + 1, dtype=np.float64) / n - 1.0)) / np.tanh(gamma))
    y[0], y[-1] = 0.0, 1.0
    return length * y


def _shape(c):
    return c["n0"], c["n1"], c["n2"]


def _points_bc(c):
    """vertex coordinates per axis and one letter per axis: P periodic, N
    zero-gradient walls, D zero-value walls, M a zero-value lower and a
    zero-gradient upper wall"""
    n = _shape(c)
    # cells of one size along the uniform axes, the longest axis of length 1
    pts = [_uniform(m, m / max(n)) for m in n]
    if c["kind"] == "mg":
        if c["mesh"] == "channel":
            pts[1] = _tanh(n[1], 2.0, n[1] / max(n))
            return pts, "PNP"
        return pts, {"walls": "DNN"}.get(c["mesh"], "NNN")
    if c["kind"] in ("fft", "project"):
        pts[1] = _tanh(n[1], 1.5, n[1] / max(n))
        return pts, c["bc"]
    return pts, "NNN"


_PAIR = {"P": ("periodic", "periodic"), "N": ("Neumann", "Neumann"), "D": ("Dirichlet", "Dirichlet"),
         "M": ("Dirichlet", "Neumann")}


def _faces(bc):
    return tuple(f for letter in bc for f in _PAIR[letter])


_LAYOUT7 = [((128, 64, 64), (0, 0, 0)), ((96, 96, 96), (128, 0, 0)), ((64, 128, 32), (0, 64, 0)),
            ((128, 32, 64), (0, 192, 0)), ((64, 64, 64), (224, 0, 0)), ((48, 96, 48), (64, 64, 0)),
            ((32, 32, 128), (0, 0, 64))]


def _layout(c):
    """(cells, origin) of every brick and the cell size"""
    if c["mesh"] == "bricks7":
        return _LAYOUT7, 1.0 / 128
    n, cut = _shape(c), c["cut"]
    return [((cut, n[1], n[2]), (0, 0, 0)), ((n[0] - cut, n[1], n[2]), (cut, 0, 0))], 1.0 / max(n)


def _mesh(c):
    from briscola_b200.mesh import Brick, Mesh

    if c["kind"] == "mg" and c["mesh"].startswith("bricks"):
        lay, h = _layout(c)
        return Mesh([Brick([o[d] * h + h * np.arange(n[d] + 1, dtype=np.float64) for d in range(3)],
                           _faces("NNN"), o) for n, o in lay])
    pts, bc = _points_bc(c)
    return Mesh([Brick(pts, _faces(bc))])


def _cells(c):
    if c["kind"] == "mg" and c["mesh"].startswith("bricks"):
        return sum(int(np.prod(n)) for n, _ in _layout(c)[0])
    return int(np.prod(_shape(c)))


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    return torch.Generator(device=_dev()).manual_seed(int(seed))


def _randn(shape, g):
    return torch.randn(shape, generator=g, dtype=torch.float64, device=_dev())


def _sizes(pts):
    return [torch.from_numpy(np.diff(p)).to(_dev()) for p in pts]


def _along(v, d):
    s = [1, 1, 1]
    s[d] = -1
    return v.view(s)


def _volumes(h):
    return _along(h[0], 0) * _along(h[1], 1) * _along(h[2], 2)


def _velocity(n, bc, g):
    """seeded N(0, 1) face velocities: one face where an axis is periodic,
    nothing through the walls"""
    u = []
    for d in range(3):
        s = list(n)
        s[d] += 1
        a = _randn(s, g)
        if bc[d] == "P":
            a.select(d, n[d]).copy_(a.select(d, 0))
        else:
            a.select(d, 0).zero_()
            a.select(d, n[d]).zero_()
        u.append(a)
    return u


def _divergence(u, h, n):
    div = torch.zeros(n, dtype=torch.float64, device=u[0].device)
    for d in range(3):
        div += torch.diff(u[d], dim=d) / _along(h[d], d)
    return div


def _source(c, seed):
    """a cell source f, of zero volume-weighted mean where every wall is
    zero-gradient"""
    n = _shape(c)
    pts, bc = _points_bc(c)
    h = _sizes(pts)
    g = _gen(seed)
    if c["kind"] == "mg" and c["mesh"] in ("cavity", "channel"):
        f = _divergence(_velocity(n, bc, g), h, n)
        if c["mesh"] == "channel":
            cc = [torch.from_numpy(0.5 * (p[1:] + p[:-1])).to(f.device) for p in pts]
            f += torch.sin(2 * math.pi * _along(cc[0], 0) / pts[0][-1]) * torch.cos(
                math.pi * _along(cc[1], 1) / pts[1][-1])
    else:
        f = _randn(n, g)
    if not set(bc) & set("DM"):
        V = _volumes(h)
        f -= (f * V).sum() / V.sum()
    return f


def _bricks_rhs(c, seed):
    lay, h = _layout(c)
    b = _randn((_cells(c),), _gen(seed))
    return (b - b.mean()) * -h ** 3


def _sphere_lambda(c):
    """face coefficients of the two-phase sphere: 1/rho with rho 1 outside and
    1000 inside radius 0.2 (of the longest axis), ramped over two cells"""
    n = _shape(c)
    pts, _ = _points_bc(c)
    cc = [torch.from_numpy(0.5 * (p[1:] + p[:-1])).to(_dev()) for p in pts]
    ctr = [p[-1] * q for p, q in zip(pts, (0.45, 0.55, 0.6))]
    dist = torch.sqrt(sum((_along(cc[d], d) - ctr[d]) ** 2 for d in range(3))) - 0.2 * min(p[-1] for p in pts)
    alpha = torch.clamp(0.5 - dist / (2.0 / max(n)), 0.0, 1.0)
    inv = 1.0 / (alpha * 1000.0 + (1.0 - alpha))
    lam = []
    for d in range(3):
        lo = torch.cat([inv.narrow(d, 0, 1), inv], d)
        hi = torch.cat([inv, inv.narrow(d, n[d] - 1, 1)], d)
        lam.append((0.5 * (lo + hi)).contiguous())
    return lam


def _options(c):
    return {"type": "GPUMG", "relTol": c["relTol"], "tolerance": 0, "cycleType": c["cycle"], "nSweepsPre": c["pre"],
            "nSweepsPost": c["post"], "coarseLevel": c["coarse"], "smoother": "rbgs", "precision": c["precision"],
            "krylov": c["krylov"]}


def _unet_pair(c, seed):
    """a source of unit rms and the (periodic, spectral) solution of its
    Poisson problem, of unit rms: the training pairs' kind of field"""
    n = _shape(c)
    f = torch.randn(n, generator=_gen(seed), dtype=torch.float32, device=_dev())
    f -= f.mean()
    k = [torch.fft.fftfreq(m, device=f.device) * m for m in n]
    k2 = sum(_along(q, d) ** 2 for d, q in enumerate(k))
    k2[0, 0, 0] = 1.0
    F = torch.fft.fftn(f) / k2
    F[0, 0, 0] = 0.0
    t = torch.fft.ifftn(F).real
    return (f / f.square().mean().sqrt()).reshape(-1).contiguous(), (t / t.square().mean().sqrt()).reshape(-1).contiguous()


LR = 1e-4
C_DT = 1e-3


# ---------------------------------------------------------------------------
# the path
# ---------------------------------------------------------------------------
def prepare(case, seed):
    import briscola_b200 as bb
    from briscola_b200 import fft, split, unet
    from briscola_b200.mesh import Mesh

    kind = case["kind"]
    s = {"case": dict(case)}
    if kind == "mg":
        mesh = _mesh(case)
        sol = bb.solver.New(bb.Dictionary(_options(case)), mesh)
        lam = None
        if case["mesh"].startswith("bricks"):
            b = _bricks_rhs(case, seed)
        else:
            b = (_source(case, seed) * -_volumes(_sizes(_points_bc(case)[0]))).reshape(-1).contiguous()
            if case["mesh"] == "sphere":
                # the coefficients are given with a first solve and kept (constMatrix) after it
                lam = [a.cpu().numpy() for a in _sphere_lambda(case)]
        s.update(solver=sol, sys=bb.LinearSystem(mesh, torch.zeros_like(b), b, lam, zero_guess=True), x=None)
        if lam is not None:
            sol.solve(s["sys"], constMatrix=False)
    elif kind == "fft":
        f = _source(case, seed)
        s.update(solver=fft.FFTPoissonSolver(_mesh(case)), f=f, x=torch.empty_like(f))
    elif kind == "project":
        mesh = _mesh(case)
        n, g, bc = _shape(case), _gen(seed), _points_bc(case)[1]
        p = torch.zeros(n, dtype=torch.float64, device=_dev())
        s.update(solver=fft.FFTPoissonSolver(mesh),
                 context=bb.Context(mesh, bb.make_options({"relTol": 1e-8, "tolerance": 0, "autotune": "off"})),
                 u=_velocity(n, bc, g), acc=_velocity(n, bc, g), p=p, rhs=torch.empty_like(p))
        s["us"] = [torch.empty_like(a) for a in s["u"]]
    elif kind == "split":
        f = _source(case, seed)
        s.update(solver=split.SplitPoissonSolver(_mesh(case), {"solver": {"type": "FFT"}, "prediction": "off",
                                                               "nCorr": case["ncorr"]}),
                 f=f, lam=_sphere_lambda(case), x=torch.zeros_like(f))
    else:
        net = unet.UNet(_shape(case), seed=int(seed) % 1000)
        x, t = _unet_pair(case, seed)
        s.update(net=net, x=x, t=t)
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "mg":
        state["solver"].solve(state["sys"], constMatrix=True)
        return state["sys"].x
    if kind == "fft":
        return state["solver"].solve(state["x"], state["f"])
    if kind == "project":
        us, ctx = state["us"], state["context"]
        for a, u, acc in zip(us, state["u"], state["acc"]):
            torch.add(u, acc, alpha=0.1, out=a)  # the explicit predictor
        ctx.project_rhs(us, C_DT, state["rhs"], per_volume=True)
        state["solver"].solve(state["p"], state["rhs"])
        ctx.project_correct(us, state["p"], C_DT)
        return [state["p"], *us]
    if kind == "split":
        state["x"].zero_()
        return state["solver"].solve(state["x"], state["f"], state["lam"], constMatrix=True)
    net = state["net"]
    if c["what"] == "forward":
        return net.forward(state["x"])
    loss = net.train_step(state["x"], state["t"], lr=LR)
    return {"loss": loss, "gradients": net.g, "parameters": net.p}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far two correct ones may differ
# ---------------------------------------------------------------------------
_CONVS = ((0, 16, 16), (1, 16, 32), (1, 32, 32), (2, 32, 64), (2, 64, 64), (3, 64, 64), (3, 64, 64), (2, 128, 64),
          (2, 64, 64), (1, 96, 32), (1, 32, 32), (0, 48, 16), (0, 16, 16))  # level, channels in, out


def work(case):
    n = _cells(case)
    kind = case["kind"]
    if kind == "mg":
        # right-hand side in, solution out; with face coefficients also those
        lam = 24 * n if case["mesh"] == "sphere" else 0
        return {"bytes": 16 * n + lam, "flops": 0}
    if kind == "fft":
        m = case["n0"] * case["n2"]
        return {"bytes": 16 * n, "flops": n * (10 * math.log2(m) / 2 + 6)}
    if kind == "project":
        # velocity and accelerations in, corrected velocity and pressure out
        return {"bytes": 8 * n * (6 + 3 + 1), "flops": n * (10 * math.log2(case["n0"] * case["n2"]) / 2 + 30)}
    if kind == "split":
        return {"bytes": 8 * n * 5, "flops": case["ncorr"] * n * (10 * math.log2(n) / 3 + 40)}
    f = 2.0 * 28 * 16 * n + sum(2.0 * 27 * ci * co * (n >> (3 * lev)) for lev, ci, co in _CONVS)
    if case["what"] == "forward":
        return {"bytes": 8 * n, "flops": f}
    return {"bytes": 8 * n + 28 * 700_000, "flops": 3 * f}


def tolerance(case):
    kind = case["kind"]
    if kind == "mg":
        # two solves that stop at the same relative residual
        return {"rel": TOL_MG * case["relTol"], "max": 40 * TOL_MG * case["relTol"]}
    if kind in ("fft", "project", "split"):
        return {"rel": 5e-11, "max": 5e-9}
    if case["what"] == "forward":
        return {"rel": 2.5e-2, "max": 0.5}
    return {"rel": 2.5e-2, "max": 0.9}


TOL_MG = 60.0


# ---------------------------------------------------------------------------
# the same results in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _axis(points, letter):
    """eigenvectors Q and eigenvalues of the 1-D cell-centred Laplacian K
    scaled by the cell sizes, H^-1/2 K H^-1/2 = Q diag(e) Q^T, and H"""
    h = torch.from_numpy(np.diff(points)).to(_dev())
    n = h.numel()
    K = torch.zeros((n, n), dtype=torch.float64, device=h.device)
    for a in range(n - 1):
        w = 2.0 / (h[a] + h[a + 1])
        K[a, a] -= w
        K[a + 1, a + 1] -= w
        K[a, a + 1] += w
        K[a + 1, a] += w
    if letter == "P":
        w = 2.0 / (h[0] + h[-1])
        K[0, 0] -= w
        K[-1, -1] -= w
        K[0, -1] += w
        K[-1, 0] += w
    if letter in "DM":
        K[0, 0] -= 2.0 / h[0]
    if letter == "D":
        K[-1, -1] -= 2.0 / h[-1]
    r = h.rsqrt()
    e, Q = torch.linalg.eigh(r[:, None] * K * r[None, :])
    return h, e, Q


def _apply(Q, x, d):
    return torch.movedim(torch.tensordot(Q, x, dims=([1], [d])), 0, d)


class _Direct:
    """A x = b for the constant-coefficient operator of a box, by its
    eigenvectors along the three axes; the null-space part is dropped (zero
    volume-weighted mean)"""

    def __init__(self, pts, bc):
        self.ax = [_axis(p, q) for p, q in zip(pts, bc)]
        L = sum(_along(a[1], d) for d, a in enumerate(self.ax))
        self.singular = not set(bc) & set("DM")
        self.inv = 1.0 / L
        if self.singular:
            self.inv.view(-1)[L.abs().argmin()] = 0.0

    def solve(self, b):
        for d, (h, e, Q) in enumerate(self.ax):
            b = _apply(Q.T.contiguous(), b * _along(h.rsqrt(), d), d)
        b = b * self.inv
        for d, (h, e, Q) in enumerate(self.ax):
            b = _apply(Q, b, d) * _along(h.rsqrt(), d)
        return b


def _flux_div(x, lam, h):
    """V div(lam grad x) of a box with walls all round (interior faces only)"""
    out = torch.zeros_like(x)
    area = [_along(h[1], 1) * _along(h[2], 2), _along(h[0], 0) * _along(h[2], 2), _along(h[0], 0) * _along(h[1], 1)]
    for d in range(3):
        n = x.shape[d]
        w = area[d] * 2.0 / _along(h[d][1:] + h[d][:-1], d)
        q = lam[d].narrow(d, 1, n - 1) * w * torch.diff(x, dim=d)
        out.narrow(d, 0, n - 1).add_(q)
        out.narrow(d, 1, n - 1).sub_(q)
    return out


def _pcg(A, M, b, tol=1e-13, most=3000):
    x = torch.zeros_like(b)
    r = b.clone()
    z = M(r)
    p = z.clone()
    rz = (r * z).sum()
    stop = tol * b.norm()
    for _ in range(most):
        q = A(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        if r.norm() <= stop:
            break
        z = M(r)
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _bricks_exact(c, b):
    """the union of the bricks by conjugate gradients on its lattice box"""
    lay, h = _layout(c)
    hi = [max(o[d] + n[d] for n, o in lay) for d in range(3)]
    on = torch.zeros(hi, dtype=torch.float64, device=b.device)
    full = torch.zeros_like(on)
    at = 0
    cut = []
    for n, o in lay:
        sl = tuple(slice(o[d], o[d] + n[d]) for d in range(3))
        m = int(np.prod(n))
        on[sl] = 1.0
        full[sl] = b[at:at + m].view(n)
        cut.append(sl)
        at += m
    w = [on.narrow(d, 1, hi[d] - 1) * on.narrow(d, 0, hi[d] - 1) * h for d in range(3)]
    diag = torch.zeros_like(on)

    def A(x):
        out = torch.zeros_like(x)
        for d in range(3):
            q = w[d] * torch.diff(x, dim=d)
            out.narrow(d, 0, hi[d] - 1).sub_(q)
            out.narrow(d, 1, hi[d] - 1).add_(q)
        return out

    for d in range(3):
        diag.narrow(d, 0, hi[d] - 1).add_(w[d])
        diag.narrow(d, 1, hi[d] - 1).add_(w[d])
    inv = torch.where(diag > 0, 1.0 / diag.clamp(min=1e-300), torch.zeros_like(diag))
    x = _pcg(A, lambda r: r * inv, -full, 1e-12)
    x = torch.cat([x[sl].reshape(-1) for sl in cut])
    return x - x.mean()


def _conv(x, w):
    """x: (channels, n0, n1, n2), w: (27, channels in, out); zero padding"""
    n = x.shape[1:]
    xp = torch.nn.functional.pad(x, (1,) * 6)
    out = torch.zeros((w.shape[2], n[0] * n[1] * n[2]), dtype=x.dtype, device=x.device)
    for t in range(27):
        a, b, c = t // 9, (t // 3) % 3, t % 3
        out.addmm_(w[t].T, xp[:, a:a + n[0], b:b + n[1], c:c + n[2]].reshape(x.shape[0], -1))
    return out.view(w.shape[2], *n)


class _Conv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        return _conv(x, w)

    @staticmethod
    def backward(ctx, dz):
        x, w = ctx.saved_tensors
        n = x.shape[1:]
        flat = dz.reshape(dz.shape[0], -1)
        xp = torch.nn.functional.pad(x, (1,) * 6)
        dw = torch.stack([xp[:, t // 9:t // 9 + n[0], (t // 3) % 3:(t // 3) % 3 + n[1], t % 3:t % 3 + n[2]].reshape(
            x.shape[0], -1) @ flat.T for t in range(27)])
        dx = _conv(dz, w.flip(0).transpose(1, 2)) if ctx.needs_input_grad[0] else None
        return dx, dw


_NAMES = ("e0b", "e1a", "e1b", "e2a", "e2b", "e3a", "e3b", "d2a", "d2b", "d1a", "d1b", "d0a", "d0b")


def _net_params(seed):
    """the network's He-normal initial weights, laid out as its parameter
    vector: input layer and bias, the convolutions, the head and its bias"""
    rng = np.random.default_rng(seed)
    shapes = [("in.w", (27, 1, 16), 27), ("in.b", (16,), 0)]
    shapes += [(k, (27, ci, co), 27 * ci) for k, (_, ci, co) in zip(_NAMES, _CONVS)]
    shapes += [("head.w", (16,), 16), ("head.b", (1,), 0)]
    out = {}
    for name, shape, fan in shapes:
        a = np.zeros(shape, dtype=np.float32)
        if fan:
            a = (rng.standard_normal(int(np.prod(shape))) * math.sqrt(2.0 / fan)).astype(np.float32).reshape(shape)
        out[name] = torch.from_numpy(a.astype(np.float64)).to(_dev())
    return out


def _net(P, x):
    conv, relu = _Conv.apply, torch.relu
    pool = lambda a: torch.nn.functional.avg_pool3d(a[None], 2)[0]  # noqa: E731

    def up(a):
        return a.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    def two(a, k):
        return relu(conv(relu(conv(a, P[k + "a"])), P[k + "b"]))

    a0 = relu(conv(x[None], P["in.w"]) + P["in.b"].view(-1, 1, 1, 1))
    s0 = relu(conv(a0, P["e0b"]))
    s1 = two(pool(s0), "e1")
    s2 = two(pool(s1), "e2")
    b3 = two(pool(s2), "e3")
    d2 = two(torch.cat([up(b3), s2]), "d2")
    d1 = two(torch.cat([up(d2), s1]), "d1")
    d0 = two(torch.cat([up(d1), s0]), "d0")
    return torch.tensordot(P["head.w"], d0, dims=([0], [0])) + P["head.b"]


def exact(case, seed):
    kind = case["kind"]
    cells = _cells(case)
    if not torch.cuda.is_available() and cells > 1 << 18:
        return None
    if kind == "mg":
        if case["mesh"].startswith("bricks"):
            return _bricks_exact(case, _bricks_rhs(case, seed))
        pts, bc = _points_bc(case)
        h = _sizes(pts)
        b = _source(case, seed) * -_volumes(h)
        D = _Direct(pts, bc)
        if case["mesh"] != "sphere":
            return D.solve(b).reshape(-1)
        lam = _sphere_lambda(case)
        # scaled by the diagonal, then corrected by the constant-coefficient inverse
        mean = sum(l.mean() for l in lam) / 3
        x = _pcg(lambda p: -_flux_div(p, lam, h), lambda r: -D.solve(r) / mean, -b)
        V = _volumes(h)
        return (x - (x * V).sum() / V.sum()).reshape(-1)
    if kind == "fft":
        pts, bc = _points_bc(case)
        x = _Direct(pts, bc).solve(_source(case, seed) * -_volumes(_sizes(pts)))
        if not set(bc) & set("DM"):
            x -= x[:, :1].mean()  # the free constant: zero mean in the first plane of the solve axis
        return x
    if kind == "project":
        pts, bc = _points_bc(case)
        n, g, h = _shape(case), _gen(seed), _sizes(pts)
        u, acc = _velocity(n, bc, g), _velocity(n, bc, g)
        us = [a + 0.1 * b for a, b in zip(u, acc)]
        V = _volumes(h)
        # Laplacian(p) = -rhs, rhs = div(u) / (-C_DT)
        p = _Direct(pts, bc).solve(_divergence(us, h, n) / C_DT * V)
        p -= p[:, :1].mean()
        for d in range(3):
            q = torch.diff(p, dim=d) * 2.0 / _along(h[d][1:] + h[d][:-1], d)
            us[d].narrow(d, 1, n[d] - 1).sub_(C_DT * q)
            if bc[d] == "P":
                e = (p.narrow(d, 0, 1) - p.narrow(d, n[d] - 1, 1)) * 2.0 / (h[d][0] + h[d][-1])
                us[d].narrow(d, 0, 1).sub_(C_DT * e)
                us[d].narrow(d, n[d], 1).sub_(C_DT * e)
        return [p, *us]
    if kind == "split":
        pts, bc = _points_bc(case)
        h = _sizes(pts)
        V = _volumes(h)
        f, lam = _source(case, seed), _sphere_lambda(case)
        top = max(float(l.max()) for l in lam)
        D = _Direct(pts, bc)
        x = torch.zeros_like(f)
        for _ in range(case["ncorr"]):
            src = f / top + _flux_div(x, [l / top - 1.0 for l in lam], h) / V
            x = D.solve(-src * V)
            x -= x[:1].mean()
        return x
    P = _net_params(int(seed) % 1000)
    x, t = _unet_pair(case, seed)
    x, t = x.double().view(_shape(case)), t.double()
    if case["what"] == "forward":
        with torch.no_grad():
            return _net(P, x).reshape(-1)
    for p in P.values():
        p.requires_grad_(True)
    loss = (_net(P, x).reshape(-1) - t).square().mean()
    loss.backward()
    g = torch.cat([p.grad.reshape(-1) for p in P.values()])
    # the first Adam step moves every weight by lr * g / (|g| + eps)
    w = torch.cat([p.detach().reshape(-1) for p in P.values()])
    w = w - LR * g / (g.abs() + 1e-8)
    return {"loss": loss.detach().reshape(1), "gradients": g, "parameters": w}
