"""Performance cases: the transforms a program makes through this package, over the sizes they are made at.

A case is one pass through the public entry points: a synthesis followed by an analysis of the
synthesised grid (`sht.synth` / `sht.analys`, scalar, spheroidal-toroidal or three-component vectors),
a differentiable synthesis and analysis with their gradients (`autograd`), a batch of fields of uneven
lmax (`UnevenBatch`), or the values of a field at scattered points (`sht.points`).  Inputs are coefficients
N(0,1) (l+1)^-p, as in the benchmark workloads; plans keep the default polar threshold of 1e-10.

`exact` restates the transforms in 64-bit torch: orthonormal Legendre functions by the three-term
recurrence with an extended exponent on nodes and seeds from long double, dense products per order,
torch.fft along the longitudes."""
import math

import numpy as np
import torch

import shtns_b200
from shtns_b200 import autograd
from shtns_b200.batch import UnevenBatch

THETA = shtns_b200.SHT_THETA_CONTIGUOUS
PHI = shtns_b200.SHT_PHI_CONTIGUOUS


def listed():
    return [
        # one small scalar field: a time step of a small model, bound by launches and latency
        dict(name="scalar_l127_one", what="pair", comps=1, lmax=127, mres=1, nlat=192, nphi=384, layout="theta", fields=1, ltr=0, digits=0),
        # the grid that set_grid() gives by default (phi-contiguous, nphi a power of two): winds of 32 levels
        dict(name="sphtor_l255_default_32", what="pair", comps=2, lmax=255, mres=1, nlat=256, nphi=512, layout="phi", fields=32, ltr=0, digits=0),
        # gridded data at a quarter degree (nphi = 2^5 3^2 5), truncated at degree 359, 13 levels
        dict(name="scalar_l359_1440_13", what="pair", comps=1, lmax=359, mres=1, nlat=720, nphi=1440, layout="phi", fields=13, ltr=0, digits=0),
        # a shell with three-fold symmetry: vectors of 21 radial levels on a ragged grid
        dict(name="qst_l213_mres3_21", what="pair", comps=3, lmax=213, mres=3, nlat=322, nphi=216, layout="theta", fields=21, ltr=0, digits=0),
        # transforms truncated below the plan's lmax on a linear grid, 5 fields
        dict(name="scalar_l511_ltr340_5", what="pair", comps=1, lmax=511, mres=1, nlat=512, nphi=1024, layout="theta", fields=5, ltr=340, digits=0),
        # the benchmark workload: 3-D vectors of 64 radial shells
        dict(name="qst_l511_64", what="pair", comps=3, lmax=511, mres=1, nlat=768, nphi=1536, layout="theta", fields=64, ltr=0, digits=0),
        # a large simulation that transforms one vector field at a time
        dict(name="qst_l1023_one", what="pair", comps=3, lmax=1023, mres=1, nlat=1536, nphi=3072, layout="theta", fields=1, ltr=0, digits=0),
        # learning on the sphere: float32 fields, synthesis, a pointwise square, analysis, gradients
        dict(name="grad_l255_128", what="grad", lmax=255, nlat=384, nphi=768, layout="theta", fields=128),
        # many fields of different lmax, each on its own grid, in one call
        dict(name="uneven_63_1023_64", what="uneven", lmin=63, lmax=1023, steps=5, fields=64),
        # split precision: int8 digits of the Legendre values on the tensor cores
        dict(name="scalar_l2047_digits7_8", what="pair", comps=1, lmax=2047, mres=1, nlat=3072, nphi=6144, layout="theta", fields=8, ltr=0, digits=7),
        # the largest transforms
        dict(name="scalar_l4095_8", what="pair", comps=1, lmax=4095, mres=1, nlat=6144, nphi=12288, layout="theta", fields=8, ltr=0, digits=0),
        # particles or stations: a field's values at scattered points
        dict(name="points_l255_65536", what="points", lmax=255, points=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n, most=6400):
    """the smallest even size >= n with no prime factor above 7"""
    while True:
        n += n & 1
        r = n
        for f in (2, 3, 5, 7):
            while r % f == 0:
                r //= f
        if r == 1 and n <= most:
            return n
        n += 2


def draw(rng):
    kind = rng.choice(["pair"] * 7 + ["grad", "uneven", "points"])
    if kind == "points":
        return dict(what="points", lmax=_log(rng, 31, 511), points=_log(rng, 1000, 60000))
    if kind == "uneven":
        return dict(what="uneven", lmin=_log(rng, 20, 90), lmax=_log(rng, 150, 767), steps=rng.randint(2, 5), fields=_log(rng, 4, 64))
    if kind == "grad":
        lmax = _log(rng, 31, 359)
        nlat = lmax + 1 + rng.randint(0, lmax // 2 + 2)
        return dict(what="grad", lmax=lmax, nlat=nlat + nlat % 2, nphi=_smooth(2 * nlat), layout=rng.choice(["theta", "phi"]),
                    fields=max(1, min(_log(rng, 1, 160), 12000000 // lmax ** 2)))
    comps = rng.choice([1, 1, 2, 3])
    mres = rng.choice([1, 1, 1, 1, 2, 3, 5])
    if rng.random() < 0.4:
        # the sizes that are chosen most: lmax + 1 a power of two, dealiased or linear grid
        lmax = rng.choice([63, 127, 255, 511, 1023])
        nlat = rng.choice([3 * (lmax + 1) // 2, lmax + 1])
        nphi = max(2 * nlat // mres, 2 * (lmax // mres) + 1)
    else:
        lmax = _log(rng, 31, 1400)
        mmax = lmax // mres
        nlat = lmax + 1 + rng.choice([0, rng.randint(0, lmax // 4 + 2), (lmax + 2) // 2])
        nlat += nlat % 2
        nphi = rng.choice([2 * mmax + 1, 3 * mmax + 1, max(2 * nlat // mres, 2 * mmax + 1)])
    mmax = lmax // mres
    most = max(1, min(200, int(2.5e8 / (comps * nlat * nphi)), int(4e10 / (comps * nlat * lmax * mmax))))
    return dict(what="pair", comps=comps, lmax=lmax, mres=mres, nlat=nlat, nphi=_smooth(nphi), layout=rng.choice(["theta", "phi"]),
                fields=_log(rng, 1, most), ltr=rng.choice([0, 0, 0, 2 * lmax // 3]),
                digits=7 if mres == 1 and lmax > 250 and rng.random() < 0.15 else 0)


# ------------------------------------------------------------------ inputs and passes

_plan = {}      # the last plan: a program makes it once and transforms many inputs with it


def _sht(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "fields", "ltr", "points", "what", "comps")))
    if key not in _plan:
        _plan.clear()
        lmax, mres = case["lmax"], case.get("mres", 1)
        sh = shtns_b200.sht(lmax, lmax // mres, mres)
        if case["what"] != "points":
            sh.set_grid(case["nlat"], case["nphi"], flags=shtns_b200.sht_quick_init | (THETA if case["layout"] == "theta" else PHI))
        if case.get("digits"):
            sh.set_split(case["digits"])
        _plan[key] = sh
    return _plan[key]


def _steps(case):
    return [int(round(v)) - 1 for v in np.geomspace(case["lmin"] + 1, case["lmax"] + 1, case["steps"])]


def _lm(lmax, mres):
    """degree and order of every coefficient"""
    l = np.concatenate([np.arange(m, lmax + 1) for m in range(0, lmax + 1, mres)])
    m = np.concatenate([np.full(lmax + 1 - m, m) for m in range(0, lmax + 1, mres)])
    return torch.from_numpy(l).cuda(), torch.from_numpy(m).cuda()


def _coefficients(gen, fields, lmax, mres, power, mean):
    l, m = _lm(lmax, mres)
    q = torch.randn(fields, len(l), dtype=torch.complex128, device="cuda", generator=gen) * (2 ** 0.5 / (l + 1.0) ** power)
    q.imag[:, m == 0] = 0
    if not mean:
        q[:, l == 0] = 0
    return q


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    what = case["what"]
    if what == "uneven":
        lmaxs = _steps(case)
        ub = UnevenBatch([lmaxs[i % len(lmaxs)] for i in range(case["fields"])])
        for q, l in zip(ub.Q, ub.buckets):
            q.copy_(_coefficients(gen, q.shape[0], l, 1, 1.0, True))
        return dict(what=what, batch=ub)
    sh = _sht(case)
    if what == "points":
        q = _coefficients(gen, 1, case["lmax"], 1, 1.0, True)[0]
        cost = torch.rand(case["points"], dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        phi = torch.rand(case["points"], dtype=torch.float64, device="cuda", generator=gen) * (2 * math.pi)
        return dict(what=what, sh=sh, q=q, cost=cost, phi=phi)
    if what == "grad":
        q = _coefficients(gen, case["fields"], case["lmax"], 1, 1.0, True).to(torch.complex64)
        h = torch.randn(q.shape, dtype=torch.complex64, device="cuda", generator=gen)
        return dict(what=what, sh=sh, q=q.requires_grad_(True), h=h)
    comps = case["comps"]
    q = [_coefficients(gen, case["fields"], case["lmax"], case["mres"], 1.0 if comps != 2 and c == 0 else 1.5, comps != 2 and c == 0)
         for c in range(comps)]
    return dict(what=what, sh=sh, q=q, ltr=case["ltr"] or None)


def run(state):
    what = state["what"]
    if what == "uneven":
        state["batch"].pair()
        return [state["batch"].V, state["batch"].R]
    sh = state["sh"]
    if what == "points":
        return sh.points(state["q"], state["cost"], state["phi"])
    if what == "grad":
        q = state["q"]
        v = autograd.synth(sh, q)
        r = autograd.analys(sh, v * v)
        g, = torch.autograd.grad(r, q, state["h"])
        return [v.detach(), r.detach(), g]
    v = sh.synth(*state["q"], ltr=state["ltr"])
    v = v if isinstance(v, tuple) else (v,)
    r = sh.analys(*v, ltr=state["ltr"])
    return [list(v), list(r) if isinstance(r, tuple) else [r]]


# ------------------------------------------------------------------ what a pass cannot do without

def _direction(lmax, mres, nlat, nphi, n, complex_bytes):
    """bytes and flops of one direction of n scalar transforms: coefficients and grid once each; even and odd
    degrees and both hemispheres share one Legendre value (8 flop per row of a hemisphere and pair of degrees),
    and a real FFT along each latitude"""
    mmax = lmax // mres
    nlm = sum(lmax + 1 - m * mres for m in range(mmax + 1))
    pairs = sum((lmax - m * mres) // 2 + 1 for m in range(mmax + 1))
    flops = n * (8.0 * (nlat // 2) * pairs + 2.5 * nlat * nphi * math.log2(nphi))
    return n * complex_bytes * (nlm + 0.5 * nlat * nphi), flops


def work(case):
    what = case["what"]
    if what == "points":
        # each point: a value from every coefficient (complex multiply-add, half of a complex one for the recurrence)
        nlm = (case["lmax"] + 1) * (case["lmax"] + 2) // 2
        return dict(bytes=16.0 * nlm + 24.0 * case["points"], flops=8.0 * nlm * case["points"])
    if what == "uneven":
        lmaxs = _steps(case)
        b = f = 0.0
        for i in range(case["fields"]):
            l = lmaxs[i % len(lmaxs)]
            nlat = (3 * (l + 1) + 1) // 2
            nlat += nlat & 1
            d = _direction(l, 1, nlat, 2 * nlat, 1, 16.0)
            b, f = b + 2 * d[0], f + 2 * d[1]
        return dict(bytes=b, flops=f)
    if what == "grad":
        b, f = _direction(case["lmax"], 1, case["nlat"], case["nphi"], case["fields"], 8.0)
        return dict(bytes=4 * b, flops=4 * f)
    lim = case["ltr"] or case["lmax"]
    b = _direction(case["lmax"], case["mres"], case["nlat"], case["nphi"], case["fields"] * case["comps"], 16.0)[0]
    f = _direction(lim, case["mres"], case["nlat"], case["nphi"], case["fields"] * case["comps"], 16.0)[1]
    return dict(bytes=2 * b, flops=2 * f)


def tolerance(case):
    # measured: 4e-8 against exact() where the arrays are float32, up to 3e-13 between orders of the 64-bit sums
    # and 2e-13 for 7 digits of 8 bits per operand
    if case["what"] == "grad":
        return {"rel": 2e-7, "max": 4e-6}
    return {"rel": 1e-12, "max": 1e-10}


# ------------------------------------------------------------------ the same in plain 64-bit torch

def _gauss(n):
    """north half of the Gauss-Legendre nodes and weights, and the sines of the rounded nodes"""
    i = np.arange(1, n // 2 + 1, dtype=np.longdouble)
    x = np.cos(np.longdouble(math.pi) * (i - 0.25) / (n + np.longdouble(0.5)))
    for _ in range(6):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
        dp = n * (p0 - x * p1) / ((1 - x) * (1 + x))
        x = x - p1 / dp
    x, w = x.astype(np.float64), (2 / ((1 - x) * (1 + x) * dp * dp)).astype(np.float64)
    return x, w


def _orders(lmax, mres, x, limit=4e9):
    """(m0, m1, T) for runs of orders: T[i, j, t] = P_{m+j}^m(x_t), m = mres (m0 + i), orthonormal with the
    Condon-Shortley phase, zero beyond lmax"""
    x = np.asarray(x, dtype=np.float64)
    xl = x.astype(np.longdouble)
    s = np.sqrt((1 - xl) * (1 + xl))
    mant, ex = np.empty((lmax // mres + 1, len(x))), np.empty((lmax // mres + 1, len(x)), dtype=np.int32)
    y, e = np.full(len(x), 1 / np.sqrt(4 * np.longdouble(math.pi))), np.zeros(len(x), dtype=np.int32)
    for m in range(lmax + 1):
        if m:
            y = -y * s * np.sqrt((2 * np.longdouble(m) + 1) / (2 * np.longdouble(m)))
        y, d = np.frexp(y)
        e = e + d
        if m % mres == 0:
            mant[m // mres], ex[m // mres] = y, e
    xt = torch.from_numpy(x).cuda()
    m0 = 0
    while m0 <= lmax // mres:
        J = lmax + 1 - m0 * mres
        m1 = min(lmax // mres + 1, m0 + max(1, int(limit / (8.0 * J * len(x)))))
        E = torch.from_numpy(ex[m0:m1]).cuda()
        p1 = torch.from_numpy(mant[m0:m1]).cuda()
        near = E > -300
        p1 = torch.where(near, torch.ldexp(p1, torch.where(near, E, 0)), p1)
        E = torch.where(near, 0, E)
        sc = torch.exp2(E.double())
        p0 = torch.zeros_like(p1)
        T = torch.zeros(m1 - m0, J, len(x), dtype=torch.float64, device="cuda")
        m = mres * torch.arange(m0, m1, dtype=torch.float64, device="cuda")[:, None]
        T[:, 0] = p1 * sc
        for j in range(1, J):
            l = m + j
            a = torch.sqrt((4 * l * l - 1) / (l * l - m * m))
            b = torch.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1))
            p0, p1 = p1, a * (xt * p1 - b * p0)
            if j % 16 == 0:
                big = (p1.abs() > 2.0 ** 300) & (E < 0)
                k = torch.where(big, torch.clamp(-E, max=300), 0)
                f = torch.exp2(-k.double())
                p0, p1, E = p0 * f, p1 * f, E + k
                sc = torch.exp2(E.double())
            T[:, j] = p1 * sc
            if j > lmax - mres * (m1 - 1):
                T[(m[:, 0] + j) > lmax, j] = 0
        yield m0, m1, T
        del T
        m0 = m1


def _turn(c):
    """i times the complex columns (re, im) of c"""
    c = c.unflatten(2, (c.shape[2] // 2, 2))
    return torch.stack([-c[..., 1], c[..., 0]], -1).flatten(2)


class _Exact:
    """synthesis and analysis of n fields on the grid of a case, the components of a vector together"""

    def __init__(self, lmax, mres, nlat, nphi, ltr, layout):
        self.lmax, self.mres, self.nlat, self.nphi, self.layout = lmax, mres, nlat, nphi, layout
        self.lim = ltr or lmax
        self.x, self.w = _gauss(nlat)
        self.wt = torch.from_numpy(self.w).cuda()
        self.xt = torch.from_numpy(self.x).cuda()
        self.st = torch.sqrt((1 - self.xt) * (1 + self.xt))

    def _runs(self):
        """runs of orders: first and last, Legendre values, their theta derivatives, m / sin(theta) times them,
        degree weights, and the places of the coefficients (nlm where there is none)"""
        starts = np.concatenate([[0], np.cumsum([self.lmax + 1 - m for m in range(0, self.lmax + 1, self.mres)])])
        nlm = int(starts[-1])
        for m0, m1, T in _orders(self.lim, self.mres, self.x):
            J = T.shape[1]
            m = self.mres * np.arange(m0, m1)[:, None]
            l = m + np.arange(J)[None, :]
            at = torch.from_numpy(np.where(l <= self.lim, starts[m0:m1, None] + np.arange(J)[None, :], nlm)).cuda()
            yield m0, m1, T, torch.from_numpy(m).cuda().double(), torch.from_numpy(l).cuda().double(), at

    def _derivative(self, T, m, l):
        """dP/dtheta (of the opposite parity) and m P / sin(theta)"""
        c = torch.sqrt((l * l - m * m).clamp(min=0) * (2 * l + 1) / (2 * l - 1).clamp(min=1))
        D = l[:, :, None] * self.xt * T
        D[:, 1:] -= c[:, 1:, None] * T[:, :-1]
        D /= self.st
        D[l > self.lim] = 0
        return D, T * (m[:, :, None] / self.st)

    def _sum(self, T, C):
        """sums over the even and the odd degree offsets of a run, on the northern rows"""
        Tt = T.transpose(1, 2)
        even, odd = Tt[:, :, 0::2] @ C[:, 0::2], Tt[:, :, 1::2] @ C[:, 1::2]
        return even, odd

    def _rows(self, even, odd):
        return torch.cat([even + odd, (even - odd).flip(1)], 1)         # [orders, nlat, 2 n]

    def synth(self, q):
        n = q[0].shape[0]
        M = self.lim // self.mres + 1
        F = [torch.zeros(M, self.nlat, n, dtype=torch.complex128, device="cuda") for _ in q]
        pad = [torch.cat([a, a.new_zeros(n, 1)], 1) for a in q]
        for m0, m1, T, m, l, at in self._runs():
            C = [torch.view_as_real(a[:, at].permute(1, 2, 0).contiguous()).flatten(2) for a in pad]
            rows = []
            if len(q) != 2:
                rows.append(self._rows(*self._sum(T, C[0])))
            if len(q) > 1:
                D, S = self._derivative(T, m, l)
                s, t = C[-2], C[-1]
                ds, dt = self._sum(D, s), self._sum(D, t)
                is_, it = self._sum(S, _turn(s)), self._sum(S, _turn(t))
                rows.append(self._mix(ds, it, 1.0))
                rows.append(self._mix(dt, is_, -1.0))
            for f, r in zip(F, rows):
                f[m0:m1] = torch.view_as_complex(r.unflatten(2, (n, 2)).contiguous())
        out = []
        for f in F:
            f = f.permute(2, 1, 0)                                      # [n, nlat, M]
            z = f.new_zeros(n, self.nlat, self.nphi // 2 + 1)
            z[..., :M] = f
            v = torch.fft.irfft(z, self.nphi, dim=-1, norm="forward")
            out.append(v if self.layout == "phi" else v.transpose(1, 2).contiguous())
        return out

    def _mix(self, d, s, sign):
        """sign times the derivative's rows, whose parity is the opposite one, plus the others"""
        return self._rows(sign * d[1] + s[0], sign * d[0] + s[1])

    def analys(self, v):
        n = v[0].shape[0]
        M = self.lim // self.mres + 1
        nlm = sum(self.lmax + 1 - m for m in range(0, self.lmax + 1, self.mres))
        F = []
        for a in v:
            a = a if self.layout == "phi" else a.transpose(1, 2)
            f = torch.fft.rfft(a, dim=-1, norm="forward")[..., :M].permute(2, 1, 0)      # [M, nlat, n]
            F.append(torch.view_as_real(f.contiguous()).flatten(2))
        out = [torch.zeros(n, nlm + 1, dtype=torch.complex128, device="cuda") for _ in v]
        h = self.nlat // 2
        for m0, m1, T, m, l, at in self._runs():
            wt = 2 * math.pi * self.wt[:, None]

            def split(f):
                a, b = f[m0:m1, :h], f[m0:m1, h:].flip(1)
                return wt * (a + b), wt * (a - b)

            def sums(T, e, o):                                          # T even for even offsets
                c = T.new_zeros(T.shape[0], T.shape[1], 2 * n)
                c[:, 0::2], c[:, 1::2] = T[:, 0::2] @ e, T[:, 1::2] @ o
                return c

            res = []
            if len(v) != 2:
                res.append(sums(T, *split(F[0])))
            if len(v) > 1:
                D, S = self._derivative(T, m, l)
                (te, to), (pe, po) = split(F[-2]), split(F[-1])
                ll = 1 / (l * (l + 1)).clamp(min=1)[:, :, None]
                res.append((sums(D, to, te) - _turn(sums(S, pe, po))) * ll)
                res.append((-_turn(sums(S, te, to)) - sums(D, po, pe)) * ll)
                if m0 == 0:
                    res[-1][0, 0] = 0
                    res[-2][0, 0] = 0
            found = []
            for o, c in zip(out, res):
                z = torch.view_as_complex(c.unflatten(2, (n, 2)).contiguous()).permute(2, 0, 1)
                if m0 == 0:
                    z = torch.cat([z[:, :1].real + 0j, z[:, 1:]], 1)
                found.append(o.index_copy(1, at.flatten(), z.flatten(1)))
            out = found
        return [o[:, :nlm] for o in out]


def exact(case, seed):
    state = prepare(case, seed)
    what = case["what"]
    if what == "points":
        q, out = state["q"], []
        for at in range(0, case["points"], 8192):
            x, phi = state["cost"][at:at + 8192], state["phi"][at:at + 8192]
            v, o = torch.zeros_like(x), 0
            for m0, m1, T in _orders(case["lmax"], 1, x.cpu().numpy()):
                for i in range(m1 - m0):
                    m = m0 + i
                    n = case["lmax"] + 1 - m
                    f = torch.view_as_real(q[o:o + n]).t() @ T[i, :n]
                    o += n
                    v += (2 if m else 1) * (f[0] * torch.cos(m * phi) - f[1] * torch.sin(m * phi))
            out.append(v)
        return torch.cat(out)
    if what == "uneven":
        V, R = [], []
        ub = state["batch"]
        for q, l, sh in zip(ub.Q, ub.buckets, ub.plans):
            e = _Exact(l, 1, sh.nlat, sh.nphi, 0, "theta")
            V += e.synth([q])
            R += e.analys(V[-1:])
        return [V, R]
    if what == "grad":
        e = _Exact(case["lmax"], 1, case["nlat"], case["nphi"], 0, case["layout"])
        q = state["q"].detach().to(torch.complex128).requires_grad_(True)
        v = e.synth([q])[0]
        r = e.analys([v * v])[0]
        g, = torch.autograd.grad(r, q, state["h"].to(torch.complex128))
        return [v.detach(), r.detach(), g]
    e = _Exact(case["lmax"], case["mres"], case["nlat"], case["nphi"], case["ltr"], case["layout"])
    v = e.synth(state["q"])
    return [v, e.analys(v)]
