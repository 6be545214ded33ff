"""Performance cases: the work that users of ves3d_b200 have it do, over the range of sizes,
orders, options and precisions that it is used at, each through the public entry points.

Every listed case says beside it what it stands for; draw() gives further cases of the same
ranges. A case's "kind" selects the entry point:

  eval         StokesVelocity: SetSrcCoord + SetDensitySL (+ SetDensityDL) + operator(), the
               evaluation of a time step on moved surfaces (self matrices rebuilt)
  poly         PolydisperseStokesVelocity: the same over vesicles of several SH orders
  matvec       the implicit step's operator [u; sigma] -> [u - S f; -div S f] on fixed
               surfaces, what each BiCGStab iteration applies
  targets      velocities at off-surface targets with the near-singular correction
  interaction  the all-pairs VesInteraction handle on host arrays
  sht          SHTrans: analysis, synthesis and the low-pass filter of grid functions

exact() restates each in plain torch, in 64 bits.
"""
import ctypes
import math

import numpy as np
import torch

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
KAPPA, DT, RATE = 0.05, 0.01, 1.0  # implicit step: bending modulus, time step, shear rate
EDGE = 8  # interpolation nodes of the near-singular correction


def listed():
    return [
        # a pair of vesicles at a low order, from host arrays: the smallest call a program makes
        # (two-vesicle interaction studies), all launches and latency
        dict(name="pair_p6", kind="eval", nves=2, p=6, p_up=12, prec="fp64", dl=False, host=True),
        # the 8-vesicle p = 12 suspension, plain FP64, through host arrays
        dict(name="eval_8ves_p12", kind="eval", nves=8, p=12, p_up=24, prec="fp64", dl=False, host=True),
        # an ordinary suspension, plain FP64, device arrays
        dict(name="eval_64ves_p16", kind="eval", nves=64, p=16, p_up=32, prec="fp64", dl=False, host=False),
        # the headline suspension: 512 vesicles of p = 16, mixed precision
        dict(name="eval_512ves_p16_mixed", kind="eval", nves=512, p=16, p_up=32, prec="mixed", dl=False, host=False),
        # and in plain FP64, the form that parity is stated for
        dict(name="eval_512ves_p16", kind="eval", nves=512, p=16, p_up=32, prec="fp64", dl=False, host=False),
        # single and double layer together (a viscosity contrast's evaluation)
        dict(name="both_layers_48ves_p16", kind="eval", nves=48, p=16, p_up=32, prec="fp64", dl=True, host=False),
        # the upsampling order moved up by 2, as MonitorError adapts it
        dict(name="adapted_27ves_p12", kind="eval", nves=27, p=12, p_up=26, prec="fp64", dl=False, host=False),
        # vesicles of four orders in one suspension, mixed precision
        dict(name="poly_256ves_mixed", kind="poly", nves=256, orders="8,12,16,24", prec="mixed", dl=False),
        # one application of the implicit operator (a 4 x 4 x 2 suspension), plain FP64
        dict(name="matvec_32ves_p16", kind="matvec", nves=32, p=16, prec="fp64"),
        # flow field around a suspension, many of its targets close to a surface
        dict(name="targets_27ves_p12", kind="targets", nves=27, p=12, m=20000, dl=False),
        # the interaction handle of a program that keeps its own data on the host
        dict(name="interaction_19000", kind="interaction", n=19000),
        # transforms of the coordinates of 256 vesicles
        dict(name="sht_768fun_p16", kind="sht", nfun=768, p=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "poly", "matvec", "targets", "interaction", "sht"])
    if kind == "eval":
        p = rng.choice([4, 5, 6, 8, 8, 10, 12, 12, 15, 16, 16, 18, 24])
        up = 2 * p + rng.choice([0, 0, 0, 0, -2, 2])
        c = dict(kind="eval", nves=_log(rng, 1, 512), p=p, p_up=up, prec=rng.choice(["fp64", "fp64", "mixed"]),
                 dl=rng.random() < 0.25, host=rng.random() < 0.3)
    elif kind == "poly":
        o = sorted(rng.sample([4, 6, 8, 12, 16, 20, 24], rng.randint(2, 4)))
        c = dict(kind="poly", nves=_log(rng, 6, 256), orders=",".join(map(str, o)), prec=rng.choice(["fp64", "mixed"]),
                 dl=rng.random() < 0.25)
    elif kind == "matvec":
        c = dict(kind="matvec", nves=_log(rng, 1, 256), p=rng.choice([6, 8, 9, 12, 16, 16, 20]),
                 prec=rng.choice(["fp64", "mixed"]))
    elif kind == "targets":
        c = dict(kind="targets", nves=_log(rng, 1, 64), p=rng.choice([6, 8, 11, 12, 16]), m=_log(rng, 50, 20000),
                 dl=rng.random() < 0.3)
    elif kind == "interaction":
        return dict(kind="interaction", n=_log(rng, 100, 100000))
    else:
        return dict(kind="sht", nfun=_log(rng, 3, 3000), p=rng.choice([4, 6, 8, 11, 12, 16, 16, 17, 24, 32]))
    while _cost(c) > 0.5 * _cost(listed()[4]):  # (the dearest listed case is the 512-vesicle FP64 evaluation)
        c["nves"] = c["nves"] * 2 // 3
    return c


# ---- sizes and work --------------------------------------------------------------------------
def _orders(case):
    """The SH order of every vesicle, ascending."""
    if case["kind"] == "poly":
        o = [int(x) for x in case["orders"].split(",")]
        return sorted(o[v % len(o)] for v in range(case["nves"]))
    return [case["p"]] * case["nves"]


def _ng(p):
    return 2 * p * (p + 1)


def _nc(p):
    return p * (p + 2)


def _sht_flops(p, q):
    """One function between order-p coefficients and an order-q grid: Legendre sums and DFTs."""
    return 2.0 * _nc(p) * (q + 1) + 2.0 * (q + 1) * 2 * p * 2 * q


def _build_flops(p, q, layers):
    """Self matrices of one vesicle: every rotation of the surface and the adjoint of 12 kernel
    components per rotation, the kernel itself, and the analysis of the result."""
    rot, blocks = p * (p + 1), sum(min(2 * n + 1, 2 * p) ** 2 for n in range(p + 1))
    per = 2.0 * 3 * blocks + 3 * 3 * _sht_flops(p, q)
    per += layers * (2 * _ng(q) * 45.0 + 12 * _sht_flops(p, q) + 2.0 * 12 * blocks)
    return rot * per + layers * 9 * _nc(p) * _sht_flops(p, p)


def _far_flops(orders, layers):
    ng = np.array([_ng(p) for p in orders], dtype=np.float64)
    return float(ng.sum() ** 2 - (ng ** 2).sum()) * (28.0 + 30.0 * (layers - 1))


def _cost(case):
    """A rough cost for draw(): general orders run at a fraction of the rate of the usual ones."""
    orders = _orders(case)
    layers = 2 if case.get("dl") else 1
    build = 0.0
    if case["kind"] != "matvec":
        for p in orders:
            q = case.get("p_up", 2 * p)
            usual = p in (4, 8, 12, 16, 24) and q == 2 * p
            build += _build_flops(p, q, 1) * (1 if usual else 10) + (layers - 1) * 10 * _build_flops(p, q, 1)
    return build + 1.5 * _far_flops(orders, layers)


def work(case):
    kind = case["kind"]
    if kind == "interaction":
        return dict(bytes=72.0 * case["n"], flops=28.0 * case["n"] * (case["n"] - 1.0))
    if kind == "sht":
        p, n = case["p"], case["nfun"]
        # the grid and the coefficients are read, and both grids and the coefficients written
        return dict(bytes=8.0 * n * (4 * _ng(p) + 2 * _nc(p)), flops=4.0 * n * _sht_flops(p, p))
    orders = _orders(case)
    layers = 2 if case.get("dl") else 1
    N = float(sum(_ng(p) for p in orders))
    if kind == "matvec":
        p, nv = case["p"], case["nves"]
        # displacement, h, grad h, sigma, f, the velocity and its divergence each transformed once;
        # the self matrices are read once
        sht = nv * (3 * 4 + 1 * 3 + 3 * 3 + 1 * 3 + 3 * 2 + 3 * 3) * _sht_flops(p, p)
        gemv = nv * (3.0 * _nc(p)) ** 2
        return dict(bytes=8 * (8 * N + gemv), flops=sht + 2 * gemv + _far_flops(orders, 1))
    if kind == "targets":
        p, m = case["p"], case["m"]
        pairs = float(m) * case["nves"] * _ng(2 * p)
        gemv = layers * case["nves"] * (3.0 * _nc(p)) ** 2
        return dict(bytes=8 * (6.0 * m + 3 * layers * N + gemv), flops=pairs * (28 + 30 * (layers - 1)) + 2 * gemv)
    build = sum(_build_flops(p, case.get("p_up", 2 * p), layers) for p in orders)
    gemv = layers * sum((3.0 * _nc(p)) ** 2 for p in orders)
    return dict(bytes=8 * 3 * N * (2 + layers), flops=build + 2 * gemv + _far_flops(orders, layers))


# ---- inputs ------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _shapes(p, centers, radii, axes, amp, g):
    """Surfaces [n][3][ng]: ellipsoids of the given semi-axes with a smooth perturbation (degrees
    1 to 4) of relative size up to amp."""
    n = centers.shape[0]
    x, _ = _gauss(p + 1)
    s = torch.sqrt(1 - x * x)
    ph = torch.arange(2 * p, device=DEV, dtype=F64) * (math.pi / p)
    xx, ss = x.repeat_interleave(2 * p), s.repeat_interleave(2 * p)
    pp = ph.repeat(p + 1)
    e = torch.stack([ss * torch.cos(pp), ss * torch.sin(pp), xx])
    deg = min(4, p)
    Y = _basis(deg, xx, ss, pp)[1:]
    q = (torch.rand(n, Y.shape[0], generator=g, device=DEV, dtype=F64) * 2 - 1) @ Y
    q = q / q.abs().amax(1, keepdim=True)
    e = e * torch.tensor(axes, device=DEV, dtype=F64)[:, None]
    r = radii[:, None] * (1 + amp * q)
    return centers[:, :, None] + r[:, None, :] * e


def _centers(n, spacing, g):
    """The first n points of a cubic lattice, jittered."""
    k = 1
    while k ** 3 < n:
        k += 1
    i = torch.arange(n, device=DEV)
    c = torch.stack([i % k, (i // k) % k, i // (k * k)], 1).to(F64) * spacing
    return c + (torch.rand(n, 3, generator=g, device=DEV, dtype=F64) * 2 - 1) * 0.1


def _inputs(case, seed):
    """The case's arrays on DEV: surfaces and densities as flat per-vesicle [3][ng] blocks."""
    g = _gen(seed)
    kind = case["kind"]

    def randn(n):
        return torch.randn(n, generator=g, device=DEV, dtype=F64)

    if kind == "interaction":
        n = case["n"]
        box = (n / 100.0) ** (1.0 / 3.0)
        return dict(src=torch.rand(3 * n, generator=g, device=DEV, dtype=F64) * box, den=randn(3 * n))
    if kind == "sht":
        return dict(grid=randn(case["nfun"] * _ng(case["p"])))
    orders = _orders(case)
    n = len(orders)
    if kind == "poly":
        radii = 0.7 + 0.6 * torch.rand(n, generator=g, device=DEV, dtype=F64)
        cen = _centers(n, 3.3, g)[torch.randperm(n, generator=g, device=DEV)]
        X, at = [], 0
        for p in sorted(set(orders)):
            k = orders.count(p)
            X.append(_shapes(p, cen[at:at + k], radii[at:at + k], (1.0, 1.0, 0.8), 0.05, g).reshape(-1))
            at += k
        X = torch.cat(X)
    else:
        one = torch.ones(n, device=DEV, dtype=F64)
        X = _shapes(orders[0], _centers(n, 2.7, g), one, (1.0, 1.0, 0.9), 0.08, g).reshape(-1)
    d = dict(X=X, f=randn(X.numel()))
    if case.get("dl"):
        d["g"] = randn(X.numel())
    if kind == "matvec":
        # a velocity and tension of the sizes that a solve meets: smooth at the order's scale
        p = case["p"]
        lo = max(2, p // 2)
        x, s, ph = _grid(p)
        Y = _basis(lo, x, s, ph)
        d["z"] = (randn(4 * n * Y.shape[0]).reshape(-1, Y.shape[0]) @ Y).reshape(-1) / math.sqrt(Y.shape[0])
    if kind == "targets":
        # two thirds of the targets within 0.3 of a surface (outside and inside), the others
        # anywhere in the box
        m, Xv = case["m"], X.reshape(n, 3, -1)
        near = 2 * m // 3
        v = torch.randint(n, (near,), generator=g, device=DEV)
        k = torch.randint(Xv.shape[2], (near,), generator=g, device=DEV)
        P, C = Xv[v, :, k], Xv.mean(2)[v]
        t = 1 + 0.6 * (torch.rand(near, 1, generator=g, device=DEV, dtype=F64) - 0.5)
        lo, hi = Xv.amin((0, 2)) - 0.5, Xv.amax((0, 2)) + 0.5
        far = lo + (hi - lo) * torch.rand(m - near, 3, generator=g, device=DEV, dtype=F64)
        d["T"] = torch.cat([C + t * (P - C), far]).contiguous().reshape(-1)
    return d


def prepare(case, seed):
    from ves3d_b200 import stokes_velocity as sv_mod
    kind, d = case["kind"], _inputs(case, seed)
    st = dict(kind=kind, **d)
    if kind == "interaction":
        st["src"], st["den"] = d["src"].cpu().numpy(), d["den"].cpu().numpy()
        st["pot"] = np.empty_like(st["den"])
        st["handle"] = _Handle()
        return st
    if kind == "sht":
        st["trans"] = sv_mod.SHTrans(case["p"])
        st["shc"] = torch.empty(case["nfun"] * _nc(case["p"]), device=DEV, dtype=F64)
        st["back"], st["low"] = torch.empty_like(d["grid"]), torch.empty_like(d["grid"])
        return st
    if kind == "poly":
        st["op"] = sv_mod.PolydisperseStokesVelocity(case["prec"])
        st["orders"] = np.array(_orders(case), dtype=np.int32)
        st["out"] = torch.empty_like(d["X"])
        return st
    st["op"] = op = sv_mod.StokesVelocity(case["p"], case.get("p_up", -1), case.get("prec", "fp64"))
    if kind == "eval":
        st["out"] = torch.empty_like(d["X"])
        if case["host"]:
            for k in ("X", "f", "g"):
                if k in st:
                    st[k] = st[k].cpu().numpy()
            st["out"] = np.empty_like(st["X"])
    elif kind == "matvec":
        # the solver's surfaces are set once per step, its operator applied many times
        op.SetSrcCoord(d["X"])
        op.set_implicit_params(DT, KAPPA, RATE)
        op.setup()
        st["z"] = d["z"].cpu().numpy()
    else:
        # the surfaces and their self matrices are at hand after the step's own evaluation
        op.SetSrcCoord(d["X"])
        op.set_near_singular(True)
        op.setup()
        st["vel"] = torch.empty_like(d["T"])
    return st


class _Handle:
    """The workspace that ves3d_stokes_alltoall_f64 keeps between calls."""

    def __init__(self):
        self.ctx = ctypes.c_void_p()

    def __del__(self):
        from ves3d_b200 import _lib
        if self.ctx:
            _lib.lib().ves3d_interaction_free(ctypes.byref(self.ctx))


def run(st):
    kind = st["kind"]
    if kind in ("eval", "poly"):
        op = st["op"]
        if kind == "poly":
            op.SetSrcCoord(st["X"], st["orders"])
        else:
            op.SetSrcCoord(st["X"])
        op.SetDensitySL(st["f"])
        if "g" in st:
            op.SetDensityDL(st["g"])
        return op(st["out"])
    if kind == "matvec":
        return st["op"].surface_op("implicit_matvec", st["z"])
    if kind == "targets":
        op = st["op"]
        op.SetDensitySL(st["f"])
        if "g" in st:
            op.SetDensityDL(st["g"])
        op.SetTrgCoord(st["T"])
        return op.eval_targets(st["vel"])
    if kind == "interaction":
        from ves3d_b200 import _lib
        src, den, pot = st["src"], st["den"], st["pot"]
        _lib.lib().ves3d_stokes_alltoall_f64(src.ctypes.data, den.ctypes.data, src.size // 3, pot.ctypes.data,
                                             ctypes.byref(st["handle"].ctx))
        return pot
    t = st["trans"]
    t.forward(st["grid"], st["shc"])
    t.backward(st["shc"], st["back"])
    t.lowPassFilter(st["grid"], st["low"])
    return dict(shc=st["shc"], back=st["back"], low=st["low"])


# ---- the same in plain 64-bit torch --------------------------------------------------------------
def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return torch.tensor(x, device=DEV), torch.tensor(w, device=DEV)


def _grid(p):
    """cos(theta), sin(theta), phi of the (p + 1) x 2p grid, latitude-major, cos(theta) ascending."""
    x = _gauss(p + 1)[0]
    s = torch.sqrt(1 - x * x)
    ph = torch.arange(2 * p, device=DEV, dtype=F64) * (math.pi / p)
    return x.repeat_interleave(2 * p), s.repeat_interleave(2 * p), ph.repeat(p + 1)


def _legendre(p, x, s):
    """sqrt(2 pi) times the orthonormal associated Legendre functions (with the (-1)^m phase),
    [m][n][points], n <= p, and m up to p + 1 (zeros)."""
    P = torch.zeros(p + 2, p + 1, x.numel(), device=DEV, dtype=F64)
    d = torch.full_like(x, math.sqrt(2 * math.pi) / math.sqrt(4 * math.pi))
    for m in range(p + 1):
        if m:
            d = -d * s * math.sqrt((2 * m + 1) / (2 * m))
        P[m, m] = d
        for n in range(m + 1, p + 1):
            a = math.sqrt((2 * n - 1) * (2 * n + 1) / ((n - m) * (n + m)))
            P[m, n] = a * x * P[m, n - 1]
            if n > m + 1:
                b = math.sqrt((2 * n + 1) * (n + m - 1) * (n - m - 1) / ((n - m) * (n + m) * (2 * n - 3)))
                P[m, n] -= b * P[m, n - 2]
    return P


def _blocks(p):
    """(m, sine) of each Fourier block in coefficient order: cosines of 0..p, sines of 1..p-1."""
    return [(0, 0)] + [(m, k) for m in range(1, p) for k in (0, 1)] + [(p, 0)]


def _basis(p, x, s, ph, du=0, dv=0):
    """The basis functions of the order-p coefficients at points, [nc][points]: du derivatives in
    theta (off the poles), dv in phi."""
    P = _legendre(p, x, s)
    if du:
        m = torch.arange(p + 1, device=DEV, dtype=F64)[:, None, None]
        n = torch.arange(p + 1, device=DEV, dtype=F64)[None, :, None]
        c = torch.sqrt(torch.clamp((n + m + 1) * (n - m), min=0.0))
        D = (m * x * P[:-1] + c * s * P[1:]) / s
        P = D if du == 1 else -(x / s) * D - (n * (n + 1) - m * m / (s * s)) * P[:-1]
    out = []
    for m, sine in _blocks(p):
        a = m * ph + (0.5 * math.pi) * dv
        out.append(P[m, m:] * (float(m) ** dv * (torch.sin(a) if sine else torch.cos(a))))
    return torch.cat(out)


def _analysis(p, q=None):
    """Grid values at order q (default p) to order-p coefficients, [ng][nc]."""
    q = p if q is None else q
    x, s, ph = _grid(q)
    w = _gauss(q + 1)[1].repeat_interleave(2 * q) / (2 * q)
    scale = [(1.0 if m == 0 or (m == p and p == q) else 2.0) for m, _ in _blocks(p) for _ in range(p + 1 - m)]
    return (_basis(p, x, s, ph) * w).T * torch.tensor(scale, device=DEV, dtype=F64)


def _smooth_w(p):
    x, w = _gauss(p + 1)
    return (w * (math.pi / p) / torch.sqrt(1 - x * x)).repeat_interleave(2 * p)


def _cross(a, b, dim):
    return torch.linalg.cross(a, b, dim=dim)


class _Surface:
    """Vesicles of one order: X [n][3][ng]."""

    def __init__(self, X, p, p_up):
        self.p, self.q, self.X = p, p_up, X.reshape(-1, 3, _ng(p))
        self.A = _analysis(p)
        g = _grid(p)
        self.Y = _basis(p, *g)
        self.Yu, self.Yv = _basis(p, *g, du=1), _basis(p, *g, dv=1)
        self.S = self.X @ self.A
        n = _cross(self.S @ self.Yu, self.S @ self.Yv, 1)
        self.area = torch.sqrt((n * n).sum(1))
        self.nrm = n / self.area[:, None]

    def weighted(self, f):
        return f.reshape(self.X.shape) * (self.area * _smooth_w(self.p))[:, None]

    def own(self, f, g=None):
        """Coefficients of the vesicles' own velocity: the rotated pole quadrature at every point."""
        p, q = self.p, self.q
        nv, nc = self.X.shape[0], _nc(p)
        x, s, ph = _grid(q)
        Y, Yu, Yv = _basis(p, x, s, ph), _basis(p, x, s, ph, du=1), _basis(p, x, s, ph, dv=1)
        xq, wq = _gauss(q + 1)
        zero = torch.zeros(2, device=DEV, dtype=F64)
        poles = _basis(p, torch.tensor([-1.0, 1.0], device=DEV, dtype=F64), zero, zero)
        # pole-singular weights: sum_j 4 pi / (2 j + 1) P_j(1) P_j(x)
        L = _legendre(q, torch.cat([xq, torch.ones(1, device=DEV, dtype=F64)]), torch.zeros(q + 2, device=DEV, dtype=F64))[0]
        j = torch.arange(q + 1, device=DEV, dtype=F64)
        sw = (4 * math.pi / (2 * j + 1) * L[:, -1] / (2 * math.pi)) @ L[:, :-1]
        sw = wq * (math.pi / q) * sw / torch.cos(torch.arccos(xq) / 2)
        w = torch.stack([sw.flip(0), sw]).repeat_interleave(2 * q, dim=1)
        x0 = _gauss(p + 1)[0]
        xg, sg, pg = _grid(p)
        C0 = torch.stack([xg, sg * torch.sin(pg), sg * torch.cos(pg)])
        A = self.A
        fields = [self.S, f.reshape(self.X.shape) @ A] + ([g.reshape(self.X.shape) @ A] if g is not None else [])
        # longitude phases of each (cosine, sine) block pair
        jj = torch.arange(p, device=DEV, dtype=F64) * (math.pi / p)
        rot = []
        for Sf in fields:
            parts, at = [], 0
            blocks = _blocks(p)
            k = 0
            while k < len(blocks):
                m = blocks[k][0]
                ln = p + 1 - m
                a = Sf[..., at:at + ln]
                if 0 < m < p:
                    b = Sf[..., at + ln:at + 2 * ln]
                    c, d = torch.cos(m * jj)[:, None, None], torch.sin(m * jj)[:, None, None]
                    parts += [a[:, None] * c + b[:, None] * d, b[:, None] * c - a[:, None] * d]
                    k, at = k + 2, at + 2 * ln
                else:
                    parts.append(a[:, None].expand(-1, p, -1, -1))
                    k, at = k + 1, at + ln
            rot.append(torch.cat(parts, -1))  # [nv][j][3][nc]
        u = torch.zeros(nv, 3, p + 1, 2 * p, device=DEV, dtype=F64)
        per = max(1, int(2e7 // (p * _ng(q))))
        for t in range(p + 1):
            c, s_ = -x0[t], -torch.sqrt(1 - x0[t] ** 2)
            x1, y1, z1 = c * C0[0] - s_ * C0[2], C0[1], s_ * C0[0] + c * C0[2]
            D = _basis(p, x1, torch.hypot(y1, z1), torch.atan2(y1, z1)) @ A
            for v0 in range(0, nv, per):
                R = [r[v0:v0 + per] @ D for r in rot]
                Xr = R[0] @ Y
                n = _cross(R[0] @ Yu, R[0] @ Yv, 2)
                F = R[1] @ Y
                G = R[2] @ Y if g is not None else None
                area = torch.sqrt((n * n).sum(2))
                trg = R[0] @ poles
                for k in range(2):
                    r = trg[..., k:k + 1] - Xr
                    ri = torch.rsqrt((r * r).sum(2))
                    a = w[k] * area * ri
                    val = (F * a[:, :, None]).sum(3) + (r * (a * ri * ri * (r * F).sum(2))[:, :, None]).sum(3)
                    val = val / (8 * math.pi)
                    if G is not None:
                        b = w[k] * (n * r).sum(2) * (r * G).sum(2) * ri ** 5
                        val = val + 3 / (4 * math.pi) * (r * b[:, :, None]).sum(3)
                    val = val.transpose(1, 2)
                    if k == 0:
                        u[v0:v0 + per, :, t, :p] = val
                    else:
                        u[v0:v0 + per, :, p - t, p:] = val
        return u.reshape(nv, 3, -1) @ A


def _sum_pairs(T, idt, X, ids, D, N=None, G=None):
    """Velocities [m][3] at T [m][3] of the sources X [n][3] of other vesicles (ids differ): the
    single layer of D and, with N and G, the double layer; coincident points contribute nothing."""
    out = torch.empty_like(T)
    per = max(1, int(4e8 // X.shape[0]))
    for a in range(0, T.shape[0], per):
        t = T[a:a + per]
        r = [X[None, :, c] - t[:, None, c] for c in range(3)]
        ri = torch.addcmul(torch.addcmul(r[0] * r[0], r[1], r[1]), r[2], r[2]).rsqrt_()
        ri.masked_fill_(torch.isinf(ri), 0.0)
        if idt is not None:
            ri.masked_fill_(idt[a:a + per, None] == ids[None, :], 0.0)
        k = r[0] * D[:, 0]
        k.addcmul_(r[1], D[None, :, 1]).addcmul_(r[2], D[None, :, 2]).mul_(ri).mul_(ri).mul_(ri)
        u = torch.stack([(k * r[c]).sum(1) for c in range(3)], 1).add_(ri @ D).div_(8 * math.pi)
        if N is not None:
            k = sum(r[c] * N[:, c] for c in range(3))
            k *= sum(r[c] * G[:, c] for c in range(3))
            k *= ri ** 5
            u -= 3 / (4 * math.pi) * torch.stack([(k * r[c]).sum(1) for c in range(3)], 1)
        out[a:a + per] = u
    return out


def _points(A):
    """[n][3][ng] -> [n ng][3]."""
    return A.transpose(1, 2).reshape(-1, 3).contiguous()


def _evaluate(groups, fs, gs):
    """Velocities of a suspension of groups of vesicles: own parts plus every other vesicle's points."""
    own, X, D, N, G, ids, nv = [], [], [], [], [], [], 0
    for k, s in enumerate(groups):
        own.append(s.own(fs[k], gs[k] if gs else None) @ s.Y)
        X.append(_points(s.X))
        D.append(_points(s.weighted(fs[k])))
        if gs:
            N.append(_points(s.nrm))
            G.append(_points(s.weighted(gs[k])))
        n = s.X.shape[0]
        ids.append(torch.arange(nv, nv + n, device=DEV).repeat_interleave(s.X.shape[2]))
        nv += n
    X, D, ids = torch.cat(X), torch.cat(D), torch.cat(ids)
    far = _sum_pairs(X, ids, X, ids, D, torch.cat(N) if gs else None, torch.cat(G) if gs else None)
    out, at = [], 0
    for s, o in zip(groups, own):
        k = o.shape[0] * o.shape[2]
        out.append((o + far[at:at + k].reshape(o.shape[0], -1, 3).transpose(1, 2)).reshape(-1))
        at += k
    return torch.cat(out)


def _operator(s, z):
    """[u - S f; -div S f], f the linearised bending of dt u plus the tension sigma."""
    p, nv = s.p, s.X.shape[0]
    g = _grid(p)
    Yuu, Yuv, Yvv = _basis(p, *g, du=2), _basis(p, *g, du=1, dv=1), _basis(p, *g, dv=2)
    u = z[:3 * nv * _ng(p)].reshape(s.X.shape)
    sig = z[3 * nv * _ng(p):].reshape(nv, -1)
    xu, xv = s.S @ s.Yu, s.S @ s.Yv
    E, F, G = (xu * xu).sum(1), (xu * xv).sum(1), (xv * xv).sum(1)
    W2 = E * G - F * F
    E, F, G = E / W2, F / W2, G / W2
    cu, cv = G[:, None] * xu - F[:, None] * xv, E[:, None] * xv - F[:, None] * xu
    L, M, N = (((s.S @ Y) * s.nrm).sum(1) for Y in (Yuu, Yuv, Yvv))
    H, K = 0.5 * (G * L + E * N) - F * M, (L * N - M * M) / W2

    def grad(a):
        c = a @ s.A
        return (c @ s.Yu)[:, None] * cu + (c @ s.Yv)[:, None] * cv

    def div(a):
        c = a @ s.A
        return ((c @ s.Yu) * cu + (c @ s.Yv) * cv).sum(1)

    c = (DT * u) @ s.A
    d = [((c @ Y) * s.nrm).sum(1) for Y in (Yuu, Yuv, Yvv)]
    h = 0.5 * (G * d[0] - 2 * F * d[1] + E * d[2])
    f = -KAPPA * (div(grad(h)) + 2 * h * (H * H - K))[:, None] * s.nrm
    f = f + 2 * (H * sig)[:, None] * s.nrm + grad(sig)
    Sf = _evaluate([s], [f.reshape(-1)], None).reshape(s.X.shape)
    return torch.cat([(u - Sf).reshape(-1), -div(Sf).reshape(-1)])


def _near(s, f, g, T):
    """Velocities at T [m][3]: the smooth quadrature of every vesicle at the upsampled order, each
    near vesicle's part replaced by the interpolation along the line from the target's projection."""
    p, q = s.p, s.q
    nv = s.X.shape[0]
    up = _grid(q)
    Y, Yu, Yv = _basis(p, *up), _basis(p, *up, du=1), _basis(p, *up, dv=1)
    Xu = s.S @ Y
    n = _cross(s.S @ Yu, s.S @ Yv, 1)
    area = torch.sqrt((n * n).sum(1))
    w = (area * _smooth_w(q))[:, None]
    fc = f.reshape(s.X.shape) @ s.A
    D, nrm, G = (fc @ Y) * w, None, None
    if g is not None:
        gc = g.reshape(s.X.shape) @ s.A
        nrm, G = n / area[:, None], (gc @ Y) * w
    pts = [None if a is None else _points(a) for a in (Xu, D, nrm, G)]
    out = _sum_pairs(T, None, pts[0], None, pts[1], pts[2], pts[3])
    cen = s.X.mean(2)
    r_near = torch.sqrt(((s.X - cen[:, :, None]) ** 2).sum(1).max()) * 2 / math.sqrt(q)
    it, iv, ik = [], [], []
    for v in range(nv):
        close = ((T - cen[v]) ** 2).sum(1) < (2.0 + r_near) ** 2
        idx = torch.nonzero(close)[:, 0]
        for a in range(0, idx.numel(), 4096):
            i = idx[a:a + 4096]
            d2, k = ((Xu[v][None] - T[i][:, :, None]) ** 2).sum(1).min(1)
            ok = d2 < r_near * r_near
            it.append(i[ok])
            iv.append(torch.full_like(i[ok], v))
            ik.append(k[ok])
    if not it:
        return out
    it, iv, ik = torch.cat(it), torch.cat(iv), torch.cat(ik)
    Vc = s.own(f, g)
    poly = [0.0] + [1 + (l - 1) / (EDGE - 2) for l in range(1, EDGE)]
    for a in range(0, it.numel(), 1024):
        i, v, k = it[a:a + 1024], iv[a:a + 1024], ik[a:a + 1024]
        S, Tn = s.S[v], T[i]
        th, ph = torch.arccos(up[0][k]), up[2][k].clone()

        def at(C, **dd):
            return torch.einsum("bcn,nb->bc", C, _basis(p, torch.cos(th), torch.sin(th), ph, **dd))

        for _ in range(40):  # the scheme stops here, converged or not
            X, a1, a2 = at(S), at(S, du=1), at(S, dv=1)
            r = X - Tn
            b11, b12, b22 = (a1 * a1).sum(1), (a1 * a2).sum(1), (a2 * a2).sum(1)
            reg = 1e-14 * (b11 + b22)
            b11, b22 = b11 + reg, b22 + reg
            g1, g2, det = (a1 * r).sum(1), (a2 * r).sum(1), b11 * b22 - b12 * b12
            th = th - (b22 * g1 - b12 * g2) / det
            ph = ph - (b11 * g2 - b12 * g1) / det
        P, nn = at(S), _cross(at(S, du=1), at(S, dv=1), 1)
        dT = Tn - P
        dist = dT.norm(dim=1)
        y0 = at(Vc[v])
        if g is not None:
            y0 = y0 + torch.where((dT * nn).sum(1) >= 0, 0.5, -0.5)[:, None] * at(gc[v])
        line = torch.stack([P + (r_near * x) * dT / dist[:, None] for x in poly[1:]] + [Tn], 1)
        r = Xu[v][:, None] - line[..., None]
        ri = torch.rsqrt((r * r).sum(2))
        Dv = D[v][:, None]
        vals = (Dv * ri[:, :, None] + r * ((r * Dv).sum(2) * ri ** 3)[:, :, None]).sum(3) / (8 * math.pi)
        if g is not None:
            b = (r * nrm[v][:, None]).sum(2) * (r * G[v][:, None]).sum(2) * ri ** 5
            vals = vals - 3 / (4 * math.pi) * (r * b[:, :, None]).sum(3)
        x = dist / r_near
        new = -vals[:, EDGE - 1]
        for l in range(EDGE):
            c = torch.ones_like(x)
            for m in range(EDGE):
                if m != l:
                    c = c * (x - poly[m]) / (poly[l] - poly[m])
            new = new + c[:, None] * (y0 if l == 0 else vals[:, l - 1])
        out.index_add_(0, i, new)
    return out


def exact(case, seed):
    kind, d = case["kind"], _inputs(case, seed)
    if kind == "interaction":
        X, D = d["src"].reshape(-1, 3), d["den"].reshape(-1, 3)
        return _sum_pairs(X, None, X, None, D).reshape(-1).cpu().numpy()
    if kind == "sht":
        p = case["p"]
        A, Y = _analysis(p), _basis(p, *_grid(p))
        c = d["grid"].reshape(case["nfun"], -1) @ A
        deg = torch.tensor([n for m, _ in _blocks(p) for n in range(m, p + 1)], device=DEV)
        return dict(shc=c.reshape(-1), back=(c @ Y).reshape(-1), low=((c * (deg <= 2 * p // 3)) @ Y).reshape(-1))
    orders = _orders(case)
    if kind in ("eval", "poly"):
        groups, fs, gs, at = [], [], [], 0
        for p in sorted(set(orders)):
            k = 3 * _ng(p) * orders.count(p)
            groups.append(_Surface(d["X"][at:at + k], p, case.get("p_up", 2 * p)))
            fs.append(d["f"][at:at + k])
            if case.get("dl"):
                gs.append(d["g"][at:at + k])
            at += k
        u = _evaluate(groups, fs, gs or None)
        return u.cpu().numpy() if case.get("host") else u
    s = _Surface(d["X"], case["p"], 2 * case["p"])
    if kind == "matvec":
        return _operator(s, d["z"]).cpu().numpy()
    return _near(s, d["f"], d.get("g"), d["T"].reshape(-1, 3)).reshape(-1)
