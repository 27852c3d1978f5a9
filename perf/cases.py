"""The work that programs have this library do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` more
of the same ranges, ``prepare(case, seed)`` what a program holds before the call (the
channel with its state, the page-locked Fortran arrays), ``run(state)`` one pass through the
public entry points with everything it computes, ``work(case)`` the bytes and operations a
pass cannot do without, and ``exact(case, seed)`` what the pass returns, computed by a plain
FP64 torch restatement of the method (compact operators by their Fourier symbols).

Kinds of pass:
  dns       device-resident run between two outputs: `steps` x step_async, then PRESG and
            the fields in the driver's Fortran arrays
  driver    a driver's time loop: each step waited for and followed by the per-step
            diagnostics (DIVCHECK, CFL, CHKMF, WALLSS), then the fields
  getup     the drop-in for GETUP: host arrays in and out on every step
  les       as dns with an SGS model and the instantaneous wall model, SGSVIS, wall stresses
  ensemble  a batch of uneven channels advanced together, then all their fields
  stats     ENERGY's statistics of the current field: plane moments, spectra with
            correlations, quadrants

The mixed forms compute in FP32 and a program that runs them keeps single-precision
snapshots, so their fields are returned as float32 copies; the FP64 form's as float64.
"""
import math
import random

import numpy as np
import torch

from compact3d_gb300 import lib
from compact3d_gb300.grid import C3D_FP64, C3D_MIXED, C3D_MIXED_IR, Grid

PI = math.pi
PRECISION = {"fp64": C3D_FP64, "mixed": C3D_MIXED, "mixed_ir": C3D_MIXED_IR}
RE_LES = 21222.0      # RE of Re_tau = 2000 by the reference's estimate RET = 0.09 RE^0.88
# Launch schedules as c3d_autotune gave them once for these shapes (a program saves and sets them).
TUNED_192 = "16,16,16,16,16,2,8,1,0,0,1,0,0,0,0,1"
TUNED_384 = "16,8,16,32,8,2,0,3,1,1,1,0,1,0,0,1"


# ------------------------------------------------------------------------------------
# Cases
# ------------------------------------------------------------------------------------
def _dt(n, lx, lz, umax):
    """A time step of CFL number about 0.3."""
    return round(min(0.02, 0.3 / (umax * (1.4 * n[0] / lx + 0.4 * n[2] / lz))), 5)


def _dns(name, n, precision, steps, *, kind="dns", lx=4 * PI, lz=4 * PI / 3, cks=2.0, re=4200.0, schedule=""):
    return {"name": name, "kind": kind, "n1m": n[0], "n2m": n[1], "n3m": n[2], "alx": lx, "alz": lz, "cks": cks,
            "re": re, "dt": _dt(n, lx, lz, 1.0), "precision": precision, "steps": steps, "schedule": schedule,
            "files": 0, "wmodel": 0}


def _les(name, n, precision, steps, files):
    return {"name": name, "kind": "les", "n1m": n[0], "n2m": n[1], "n3m": n[2], "alx": 8 * PI, "alz": 3 * PI,
            "cks": 1.0, "re": RE_LES, "dt": _dt(n, 8 * PI, 3 * PI, 2.3), "precision": precision, "steps": steps,
            "schedule": "", "files": files, "wmodel": 1}


def _ensemble(name, channels, precision, steps, pick):
    return {"name": name, "kind": "ensemble", "channels": channels, "pick": pick, "precision": precision,
            "steps": steps, "dt": 0.008}


def listed():
    return [
        # A driver on the smallest test grid, every step waited for and diagnosed: what one
        # call costs before there is any work in it.
        _dns("driver_small32_fp64", (32, 24, 48), "fp64", 2, kind="driver", lx=2 * PI, lz=PI, re=2000.0),
        # The reference's own CPU configuration (Re_tau 180, 64 x 65 x 64 points) in FP64.
        _dns("dns64_fp64", (64, 64, 64), "fp64", 20),
        # A driver that adapts to the CFL number: the mixed form on a mid-size grid.
        _dns("driver128_mixed", (128, 96, 128), "mixed", 10, kind="driver"),
        # An odd grid: N1M = 108 leaves lanes idle, N2M is odd, N3M = 144 is not a power of two.
        _dns("dns108_ragged_mixed", (108, 81, 144), "mixed", 20),
        # A production FP64 run with the launch schedule that its tuning once gave.
        _dns("dns192_fp64", (192, 128, 144), "fp64", 10, schedule=TUNED_192),
        # The mixed form with the refined pressure solve on the 256 x 193 x 256 grid.
        _dns("dns256_mixed_ir", (256, 192, 256), "mixed_ir", 20),
        # Re_tau 550 channel, the largest configuration: 384 x 257 x 384 points, mixed form, tuned.
        dict(_dns("dns384_mixed", (384, 256, 384), "mixed", 40, lx=2 * PI, lz=PI, cks=2.2, re=15000.0,
                  schedule=TUNED_384), dt=0.003),
        # Wall-modelled LES at Re_tau 2000, Smagorinsky, mixed form.
        _les("les128_mixed", (128, 64, 128), "mixed", 40, 2),
        # The dynamic model in FP64 on a smaller box.
        _les("les96_dynamic_fp64", (96, 48, 64), "fp64", 10, 1),
        # 32 uneven channels in one batch.
        _ensemble("ensemble32_mixed", 32, "mixed", 20, 7),
        # The drop-in call of a driver that keeps its fields on the host.
        _dns("getup256_fp64", (256, 96, 128), "fp64", 2, kind="getup"),
        # Statistics of a field at a driver's output interval.
        _dns("stats192_mixed", (192, 128, 192), "mixed", 1, kind="stats"),
    ]


# Extents the library takes: N1M in lane chunks, N3M multiples of 16, both 2^a 3^b; N2M free.
_N1 = [16, 18, 24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 162, 192, 256, 384]
_N3 = [16, 32, 48, 64, 96, 128, 144, 192, 256, 288, 384]
_MOST = {"fp64": 6e6, "mixed": 3e7, "mixed_ir": 2e7}


def _size(rng, most, n1=_N1):
    """Extents of about a log-uniform number of points."""
    want = math.exp(rng.uniform(math.log(2e4), math.log(most)))
    for _ in range(200):
        n = (rng.choice(n1), int(round(math.exp(rng.uniform(math.log(16), math.log(256))))), rng.choice(_N3))
        p = n[0] * n[1] * n[2]
        if 0.6 * want < p < 1.6 * want and p <= most and max(n) <= 8 * min(n):
            return n
    return 64, 49, 64


def draw(rng):
    kind = rng.choice(["dns", "dns", "dns", "driver", "les", "ensemble", "getup", "stats"])
    precision = rng.choice(["fp64", "mixed", "mixed"])
    if kind == "dns" and rng.random() < 0.15:
        precision = "mixed_ir"
    if kind == "ensemble":
        c = _ensemble("", rng.randint(4, 32), precision, 3 if precision == "fp64" else 8, rng.randrange(1 << 20))
    elif kind == "les":
        c = _les("", _size(rng, 1.5e6), precision, 8, rng.choice([1, 2]))
    else:
        n = _size(rng, min(_MOST[precision], 8e6 if kind in ("getup", "stats") else 1e9))
        p = n[0] * n[1] * n[2]
        budget = 3e7 if precision == "fp64" else 2e8
        steps = 1 if kind == "stats" else 2 if kind == "getup" else max(2, min(20, int(budget / p)))
        c = _dns("", n, precision, steps, kind=kind, re=float(rng.choice([2000, 4200, 7000])))
    del c["name"]
    return c


def _members(case):
    """The channels of an ensemble: Nx, Nz in {48, 64, 96, 128}, Ny in {33, 49, 65, 97} points,
    Re_bulk in [3000, 12000] (Re_bulk = 4/3 RE)."""
    r = random.Random(case["pick"])
    out = []
    for _ in range(case["channels"]):
        c = _dns("", (r.choice([48, 64, 96, 128]), r.choice([32, 48, 64, 96]), r.choice([48, 64, 96, 128])),
                 case["precision"], case["steps"], re=0.75 * r.uniform(3000.0, 12000.0))
        out.append(dict(c, dt=case["dt"]))
    return out


# ------------------------------------------------------------------------------------
# The method in plain FP64 torch (fields indexed [J, k, i], J = 0..N2)
# ------------------------------------------------------------------------------------
class Flow:
    def __init__(self, case):
        self.case = case
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n1, self.n2m, self.n3 = case["n1m"], case["n2m"], case["n3m"]
        self.re, self.dt = case["re"], case["dt"]
        self._mesh(case)
        th1 = 2 * PI * torch.arange(self.n1 // 2 + 1, dtype=torch.float64, device=self.dev) / self.n1
        th3 = 2 * PI * torch.arange(self.n3 // 2 + 1, dtype=torch.float64, device=self.dev) / self.n3
        self.sx = self._symbols(th1, self.dx1)
        self.sz = {k: s[:, None] for k, s in self._symbols(th3, self.dx3).items()}

    def _mesh(self, case):
        n2m, n2 = self.n2m, self.n2m + 1
        y = np.zeros(n2 + 1)
        for j in range(1, n2 + 1):
            y[j] = (2.0 * (j - 1) / n2m if case["wmodel"] else
                    1 - math.tanh(case["cks"] * (1 - 2.0 * (j - 1) / n2m)) / math.tanh(case["cks"]))
        self.aly = float(y[n2])
        self.vol = case["alx"] * self.aly * case["alz"]
        self.dx1, self.dx3 = self.n1 / case["alx"], self.n3 / case["alz"]
        dy = np.zeros(n2 + 1)
        dy[1:n2] = y[2:n2 + 1] - y[1:n2]
        dy[1] = y[2]
        h = np.zeros(n2 + 1)
        h[1:] = 0.5 * (dy[1:] + dy[:-1])
        hp, hc, hm = np.zeros(n2 + 1), np.zeros(n2 + 1), np.zeros(n2 + 1)
        for j in range(1, n2m + 1):
            hp[j], hm[j] = 1 / h[j + 1] / dy[j], 1 / h[j] / dy[j]
            hc[j] = hp[j] + hm[j]
        if case["wmodel"]:
            hm[1] = hp[n2m] = 0.0
            hc[1], hc[n2m] = 1 / h[2] / dy[1], 1 / h[n2m] / dy[n2m]
        else:
            a, b = h[1], h[2]
            hp[1], hc[1], hm[1] = 4 * a / b / (a + b) / dy[1], 4 / b / dy[1], 4 / (a + b) / dy[1]
            a, b = h[n2], h[n2m]
            hm[n2m], hc[n2m], hp[n2m] = 4 * a / b / (a + b) / dy[n2m], 4 / b / dy[n2m], 4 / (a + b) / dy[n2m]
        self.yc = 0.5 * (y[1:n2] + y[2:n2 + 1])
        self.yf = y[1:n2 + 1]
        self.dy, self.h, self.hp, self.hc, self.hm = dy, h, hp, hc, hm
        # wall-normal metrics as columns: of the cells J = 1..N2M and of the inner faces J = 2..N2M
        col = lambda a: torch.tensor(a, dtype=torch.float64, device=self.dev)[:, None, None]  # noqa: E731
        self.DY, self.HP, self.HC, self.HM = (col(a[1:n2]) for a in (dy, hp, hc, hm))
        self.H = col(h[2:n2])
        self.DYP, self.DYM = col(1 / h[2:n2] / dy[2:n2]), col(1 / h[2:n2] / dy[1:n2m])
        self.W0, self.W1 = col(dy[2:n2] / 2 / h[2:n2]), col(dy[1:n2m] / 2 / h[2:n2])

    @staticmethod
    def _symbols(th, d):
        """Fourier symbols of the compact operators (24 D, 12 D^2 and interpolation by 4) at
        the two staggered positions: b from a point and its predecessor, f its successor."""
        c, e = torch.cos(th), torch.polar(torch.ones_like(th), th)
        return {"d2": 12 * d * d * (2 * c - 2) / (10 + 2 * c) + 0j,
                "db": 24 * d * (1 - e.conj()) / (22 + 2 * c), "df": 24 * d * (e - 1) / (22 + 2 * c),
                "ib": 4 * (1 + e.conj()) / (6 + 2 * c), "if": 4 * (1 + e) / (6 + 2 * c), "cos": c}

    def X(self, f, s):
        s = self.sx[s] if isinstance(s, str) else s
        return torch.fft.irfft(torch.fft.rfft(f, dim=2) * s, n=self.n1, dim=2)

    def Z(self, f, s):
        s = self.sz[s] if isinstance(s, str) else s
        return torch.fft.irfft(torch.fft.rfft(f, dim=1) * s, n=self.n3, dim=1)

    def face(self, f):
        """Cell values J = 1..N2M to the inner faces J = 2..N2M."""
        return self.W0 * f[:-1] + self.W1 * f[1:]

    @staticmethod
    def walls(f):
        """Inner-face values with zeros on both walls: J = 1..N2."""
        return torch.nn.functional.pad(f, (0, 0, 0, 0, 1, 1))

    @staticmethod
    def thomas(a, b, c, r):
        """Tridiagonal solve along dim 0 of r (in place); a, b, c: a value per row."""
        n, g = r.shape[0], [None] * r.shape[0]
        bet = 1.0 / b[0]
        g[0] = c[0] * bet
        r[0] *= bet
        for j in range(1, n):
            bet = 1.0 / (b[j] - a[j] * g[j - 1])
            g[j] = c[j] * bet
            r[j] = (r[j] - a[j] * r[j - 1]) * bet
        for j in range(n - 2, -1, -1):
            r[j] -= g[j] * r[j + 1]
        return r

    def poisson(self, rhs):
        """GETDP: FFTs in x and z, a tridiagonal system in y per mode; DP = 0 at J = 1 of the mean."""
        n = self.n2m
        f = torch.fft.rfft2(rhs, dim=(1, 2))
        c1, c3 = self.sx["cos"], torch.cos(2 * PI * torch.arange(self.n3, dtype=torch.float64, device=self.dev) / self.n3)
        k2 = (288 * self.dx1 ** 2 * (1 - c1) / (11 + c1) ** 2)[None, :] + (288 * self.dx3 ** 2 * (1 - c3) / (11 + c3) ** 2)[:, None]
        lo = [0.0] + [1 / self.dy[j] / self.h[j] for j in range(2, n + 1)]
        up = [1 / self.dy[j] / self.h[j + 1] for j in range(1, n)] + [0.0]
        one = torch.ones_like(k2)
        a, b, c = list(lo), [-(lo[j] + up[j]) - k2 for j in range(n)], [up[j] * one for j in range(n)]
        b[0][0, 0], c[0][0, 0] = 1.0, 0.0
        f[0][0, 0] = 0.0
        return torch.fft.irfft2(self.thomas(a, b, c, f), s=(self.n3, self.n1), dim=(1, 2))

    def divergence(self, u, v, w):
        return (v[2:] - v[1:-1]) / self.DY + self.X(u[1:-1], "df") + self.Z(w[1:-1], "df")

    def correct(self, u, v, w, dp, dt):
        u[1:-1] -= dt * self.X(dp, "db")
        v[2:-1] -= dt * (dp[1:] - dp[:-1]) / self.H
        w[1:-1] -= dt * self.Z(dp, "db")

    # ---- start ----
    def start(self, seed):
        """A developed field's scales on a mean profile (laminar; Reichardt's law of the wall with a wall
        model): the curl of a random potential that vanishes at the walls, with energy up to a third of the
        resolved wavenumbers and fluctuations of about a tenth of the centreline velocity, made discretely
        divergence-free."""
        g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
        n1, n3 = self.n1, self.n3
        k1, k3 = n1 // 6, n3 // 6
        m1 = torch.arange(n1 // 2 + 1, dtype=torch.float64, device=self.dev)[None, :]
        m3 = torch.fft.fftfreq(n3, 1.0 / n3, dtype=torch.float64, device=self.dev)[:, None]
        F = []
        for _ in range(3):
            s = torch.zeros(n3, n1 // 2 + 1, dtype=torch.complex128)
            q = torch.complex(*(torch.randn(2 * k3 + 1, k1, generator=g, dtype=torch.float64) for _ in range(2)))
            for r in range(-k3, k3 + 1):
                s[r % n3, 1:k1 + 1] = q[r + k3]
            F.append(s.to(self.dev) / (1 + (m1 / 3) ** 2 + (m3 / 3) ** 2) ** 0.5)

        def at(s, px, pz, dx=0, dz=0):
            s = s * torch.exp(2j * PI * (m1 * px / n1 + m3 * pz / n3))
            s = s * (2j * PI / self.case["alx"] * m1) if dx else s
            s = s * (2j * PI / self.case["alz"] * m3) if dz else s
            return torch.fft.irfft2(s, s=(n3, n1))[None]

        col = lambda a: torch.tensor(a, dtype=torch.float64, device=self.dev)[:, None, None]  # noqa: E731
        ec, dc, ef = ((col(self.yc * (2 - self.yc)) ** 2), col(4 * self.yc * (2 - self.yc) * (1 - self.yc)),
                      col((self.yf * (2 - self.yf)) ** 2))
        pu = dc * at(F[2], 0, .5) - ec * at(F[1], 0, .5, dz=1)
        pv = ef * (at(F[0], .5, .5, dz=1) - at(F[2], .5, .5, dx=1))
        pw = ec * at(F[1], .5, 0, dx=1) - dc * at(F[0], .5, 0)
        if self.case["wmodel"]:
            yp = np.minimum(self.yc, 2 - self.yc) * 2000.0
            mean = 2000.0 / self.re * (np.log1p(0.41 * yp) / 0.41 + 7.8 * (1 - np.exp(-yp / 11) - yp / 11 * np.exp(-yp / 3)))
            amp = 0.4 * float(mean.max())
        else:
            mean, amp = self.yc * (2 - self.yc), 0.5
        amp /= float(max(pu.abs().max(), pv.abs().max(), pw.abs().max()))
        u, v, w = (torch.zeros(self.n2m + 2, n3, n1, dtype=torch.float64, device=self.dev) for _ in range(3))
        u[1:-1] = col(mean) + amp * pu
        v[2:-1] = (amp * pv)[1:-1]
        w[1:-1] = amp * pw
        self.correct(u, v, w, self.poisson(self.divergence(u, v, w)), 1.0)
        self.u, self.v, self.w = u, v, w
        self.p = torch.zeros(self.n2m, n3, n1, dtype=torch.float64, device=self.dev)
        self.hh = [torch.zeros(self.n2m, n3, n1, dtype=torch.float64, device=self.dev) for _ in range(3)]
        self.presg, self.wsm, self.nu, self.tau = [0.0, 0.0], 0.0, None, None
        return self

    # ---- SGS model and wall model ----
    def strain(self):
        u, v, w = self.u, self.v, self.w
        ip, im = (lambda f: f.roll(-1, 2)), (lambda f: f.roll(1, 2))
        kp, km = (lambda f: f.roll(-1, 1)), (lambda f: f.roll(1, 1))
        uc, wc = 0.5 * (u + ip(u))[1:-1], 0.5 * (w + kp(w))[1:-1]
        vc = 0.5 * (v[1:-1] + v[2:])
        f2 = torch.ones(self.n2m, 1, 1, dtype=torch.float64, device=self.dev)
        f2[0] = f2[-1] = 2.0
        edge = lambda c: torch.cat((c[:1], self.face(c), c[-1:]))  # noqa: E731
        du, dw = ((e[1:] - e[:-1]) * f2 / self.DY for e in (edge(uc), edge(wc)))
        a, c = self.dx1, self.dx3
        return [a * (ip(u) - u)[1:-1], 0.5 * (a * 0.5 * (ip(vc) - im(vc)) + du),
                0.5 * (a * 0.5 * (ip(wc) - im(wc)) + c * 0.5 * (kp(uc) - km(uc))), (v[2:] - v[1:-1]) / self.DY,
                0.5 * (dw + c * 0.5 * (kp(vc) - km(vc))), c * (kp(w) - w)[1:-1]], (uc, vc, wc)

    @staticmethod
    def _contract(a, b):
        return a[0] * b[0] + a[3] * b[3] + a[5] * b[5] + 2 * (a[1] * b[1] + a[2] * b[2] + a[4] * b[4])

    def sgs(self):
        s, c = self.strain()
        d23 = (self.DY / self.dx1 / self.dx3) ** (2.0 / 3.0)
        mag = torch.sqrt(2 * self._contract(s, s))
        if self.case["files"] == 2:
            yp = torch.tensor(self.yc, dtype=torch.float64, device=self.dev)[:, None, None] * math.sqrt(abs(self.wsm)) * self.re
            coef = (0.1 * (1 - torch.exp(-yp / 26.0))) ** 2
        else:
            def fil(f):
                for d in (2, 1):
                    f = (f.roll(1, d) + 4 * f + f.roll(-1, d)) / 6
                return f
            fs = [fil(q) for q in s]
            fm = 4 * d23 * torch.sqrt(2 * self._contract(fs, fs))
            m = [fm * q - fil(d23 * mag * r) for q, r in zip(fs, s)]
            fc = [fil(q) for q in c]
            pairs = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
            lo = [fil(c[p] * c[q]) - fc[p] * fc[q] for p, q in pairs]
            coef = -0.5 * self._contract(lo, m).sum((1, 2), keepdim=True) / self._contract(m, m).sum((1, 2), keepdim=True)
        self.nu = torch.clamp(coef * d23 * mag, min=-1.0 / self.re)

    def wall(self):
        """WALLMODEL_INSTANT: the damped Newton iteration for u_tau at the bottom wall's points."""
        u, w = self.u[3], self.w[3]
        d = self.dy[1] + self.dy[2] + self.dy[3] / 2
        ua = torch.sqrt(u * u + w * w)
        t1, t2, lam = torch.ones_like(ua), torch.full_like(ua, 1e-6), torch.ones_like(ua)
        f = lambda t: ua / t - torch.log(t * d * self.re) / 0.41 - 5.2  # noqa: E731
        for _ in range(10000):
            on = (t2 - t1).abs() > 1e-6
            if not bool(on.any()):
                break
            t1 = torch.where(on, t2, t1)
            f1 = f(t1)
            t2 = torch.where(on, t1 - lam * f1 / (-ua / (t1 * t1) - 1 / 0.41 / t1), t2)
            lam = torch.where(on & (f(t2).abs() > f1.abs()), 0.5 * lam, lam)
        tau = t1 * t1
        self.wsm = float(tau.mean())
        self.tau = (tau * u / ua, tau * w / ua)

    def sgs_terms(self, hh):
        u, v, w, nu = self.u[1:-1], self.v, self.w[1:-1], self.nu
        nx, nz = self.X(nu, "ib"), self.Z(nu, "ib")
        t13 = self.Z(nx, "ib") * (self.Z(u, "db") + self.X(w, "db"))
        t12 = self.walls(self.face(nx) * ((u[1:] - u[:-1]) / self.H + self.X(v[2:-1], "db")))
        t23 = self.walls(self.face(nz) * ((w[1:] - w[:-1]) / self.H + self.Z(v[2:-1], "db")))
        nvy = nu * (v[2:] - v[1:-1]) / self.DY
        hh[0] -= 2 * self.X(nu * self.X(u, "df"), "db") + self.Z(t13, "df") + (t12[1:] - t12[:-1]) / self.DY
        hh[1][1:] -= 2 * (nvy[1:] - nvy[:-1]) / self.H + self.X(t12[1:-1], "df") + self.Z(t23[1:-1], "df")
        hh[2] -= self.X(t13, "df") + (t23[1:] - t23[:-1]) / self.DY + 2 * self.Z(nu * self.Z(w, "df"), "db")

    # ---- one step (GETUP) ----
    def step(self):
        dt, re = self.dt, self.re
        if self.case["files"]:
            self.sgs()
            self.wall()
        for f in (self.u, self.v, self.w):
            f[0] = 0.0
            f[-1] = 0.0
        self.v[1] = 0.0
        U, V, W = self.u, self.v, self.w
        u, w, v = U[1:-1], W[1:-1], V[2:-1]
        exy = self.walls(self.X(v, "ib") * self.face(u))
        exz = self.Z(u, "ib") * self.X(w, "ib")
        eyz = self.walls(self.Z(v, "ib") * self.face(w))
        vc2 = (0.5 * (V[1:-1] + V[2:])) ** 2
        hh = [(exy[1:] - exy[:-1]) / self.DY + self.X(self.X(u, "if") ** 2, "db") + self.Z(exz, "df"),
              torch.zeros_like(u),
              self.Z(self.Z(w, "if") ** 2, "db") + self.X(exz, "df") + (eyz[1:] - eyz[:-1]) / self.DY]
        hh[1][1:] = (vc2[1:] - vc2[:-1]) / self.H + self.X(exy[1:-1], "df") + self.Z(eyz[1:-1], "df")
        if self.case["files"]:
            self.sgs_terms(hh)
        r = []
        for F, px, L in ((U, self.X(self.p, "db") + self.presg[0], "c"), (V, None, "f"), (W, self.Z(self.p, "db") + self.presg[1], "c")):
            if L == "c":
                f = F[1:-1]
                visc = self.HP * F[2:] - self.HC * f + self.HM * F[:-2]
            else:
                f = F[2:-1]
                visc = self.DYP * F[3:] - (self.DYP + self.DYM) * f + self.DYM * F[1:-2]
                px = (self.p[1:] - self.p[:-1]) / self.H
            r.append((visc + self.X(f, "d2") + self.Z(f, "d2")) / re - px)
        for c in (0, 2):
            r[c] -= 1.5 * hh[c] - 0.5 * self.hh[c]
        r[1] -= (1.5 * hh[1] - 0.5 * self.hh[1])[1:]
        if self.tau is not None:
            r[0][0] -= self.tau[0] / self.dy[1]
            r[2][0] -= self.tau[1] / self.dy[1]
        n = self.n2m
        q = 0.5 * dt / re
        ch = dict(a=[0.0] + [-q * self.hm[j] for j in range(2, n + 1)], b=[1 + q * self.hc[j] for j in range(1, n + 1)],
                  c=[-q * self.hp[j] for j in range(1, n)] + [0.0])
        # the v system couples to the wall faces, where the increment vanishes
        dyp = [1 / self.h[j] / self.dy[j] for j in range(2, n + 1)]
        dym = [1 / self.h[j] / self.dy[j - 1] for j in range(2, n + 1)]
        cv = dict(a=[0.0] + [-q * s for s in dym[1:]], b=[1 + q * (s + t) for s, t in zip(dyp, dym)],
                  c=[-q * s for s in dyp[:-1]] + [0.0])
        cx = (10 + 2 * self.sx["cos"]) / (10 + 24 * q * self.dx1 ** 2 + 2 * (1 - 12 * q * self.dx1 ** 2) * self.sx["cos"])
        cz = (10 + 2 * self.sz["cos"]) / (10 + 24 * q * self.dx3 ** 2 + 2 * (1 - 12 * q * self.dx3 ** 2) * self.sz["cos"])
        d = [self.Z(self.X(self.thomas(r=dt * f, **(cv if c == 1 else ch)), cx), cz) for c, f in enumerate(r)]
        vol = self.DY / self.dx1 / self.dx3
        dm = [float((d[c] * vol).sum()) / self.vol / dt for c in (0, 2)]
        u += d[0]
        v += d[1]
        w += d[2]
        dp = self.poisson(self.divergence(U, V, W) / dt)
        self.correct(U, V, W, dp, dt)
        u -= dt * dm[0]
        w -= dt * dm[1]
        self.p += dp
        self.hh = hh
        self.presg = [self.presg[0] + dm[0], self.presg[1] + dm[1]]

    # ---- the driver's arrays (C order: the Fortran ones with the first index last) ----
    def wrap(self, f):
        """[J, k, i] planes to [K, J, I] with the periodic ghost columns."""
        f = f.permute(1, 0, 2)
        f = torch.cat((f[-1:], f, f[:1]))
        return torch.cat((f[:, :, -1:], f, f[:, :, :1]), dim=2)

    def fortran(self):
        pad = torch.nn.functional.pad
        U = torch.stack([self.wrap(f) for f in (self.u, self.v, self.w)])
        HH = torch.stack([self.wrap(pad(f, (0, 0, 0, 0, 1, 1))) for f in self.hh])
        P = self.wrap(pad(self.p, (0, 0, 0, 0, 0, 1)))[1:, :, 1:]
        return {"U": U, "P": P, "HH": HH}

    def diagnostics(self):
        """CFL, the flow rates and WALLSS as the driver prints them."""
        u, v, w, a, c = self.u, self.v, self.w, self.dx1, self.dx3
        cfl = ((u + u.roll(-1, 2))[1:-1].abs() * 0.5 * a + (v[1:-1] + v[2:]).abs() * 0.5 / self.DY
               + (w + w.roll(-1, 1))[1:-1].abs() * 0.5 * c).max()
        area = self.case["alx"] * self.case["alz"]
        f1 = (u[1:-1, :, 0] * self.DY[:, :, 0]).sum() / c / a * self.n1 / area
        f3 = (w[1:-1, 0, :] * self.DY[:, 0, :]).sum() / c / a * self.n3 / area
        top = ((u[-2] - u[-1]) / (self.dy[self.n2m] / 2)).mean() * (self.aly - 1)
        bot = [(u[1] - u[0]).mean() / (self.dy[1] / 2), (v[2] - v[1]).mean() / self.dy[1], (w[1] - w[0]).mean() / (self.dy[1] / 2)]
        return [float(x) for x in (cfl, f1, f3, *((b + top) / self.re / self.aly for b in bot))]

    # ---- ENERGY's statistics ----
    def statistics(self):
        u, v, w, p, a, c = self.u, self.v, self.w, self.p, self.dx1, self.dx3
        uc, wc = 0.5 * (u + u.roll(-1, 2)), 0.5 * (w + w.roll(-1, 1))
        vc = 0.5 * (v[1:-1] + v[2:])
        edge = lambda f: torch.cat((f[:1], self.face(f[1:-1]), f[-1:]))  # noqa: E731
        dudy, dwdy = ((e[1:] - e[:-1]) / self.DY for e in (edge(uc), edge(wc)))
        dvdy = (v[2:] - v[1:-1]) / self.DY
        uc, wc = uc[1:-1], wc[1:-1]
        ddx = lambda f: (f.roll(-1, 2) - f.roll(1, 2)) * 0.5 * a  # noqa: E731
        ddz = lambda f: (f.roll(-1, 1) - f.roll(1, 1)) * 0.5 * c  # noqa: E731
        om = [dwdy - ddz(vc), ddz(uc) - ddx(wc), ddx(vc) - dudy]
        m = lambda f: f.mean((1, 2))  # noqa: E731
        mean = [m(f)[:, None, None] for f in (uc, vc, wc)]
        f = [q - r for q, r in zip((uc, vc, wc), mean)]
        cols = [m(uc), m(vc), m(wc), m(p), *(m(q) for q in om), m(uc * uc), m(vc * vc), m(wc * wc), m(uc * vc), m(uc * wc),
                m(vc * wc), m(p * p), m(p * vc), *(m(q * q) for q in om), m(uc * uc * vc), m(vc * wc * wc),
                *(m(q ** 3) for q in f), *(m(q ** 4) for q in f), m(dudy), m(dvdy), m(dwdy)]
        out = {"stats": torch.stack(cols, 1)}
        xs, zs, rxx, rzz, rxy = [], [], [], [], []
        vj = torch.cat((vc[:-1], v[self.n2m][None]))      # V at (J, JPA(J)), JPA(N2M) = N2M
        for L, (full, q) in enumerate(zip((uc, vc, wc), f)):
            xs.append(torch.fft.fft(q, dim=2).abs().square().sum(1) / self.n1 / (PI * a) / self.n3)
            zs.append(torch.fft.fft(q, dim=1).abs().square().sum(2) / self.n3 / (PI * c) / self.n1)
            var = m(full * full) - m(full) ** 2
            g = (vj if L == 1 else full) - mean[L]
            rxx.append((g[:, :, self.n1 // 2, None] * g).sum(1) / self.n3 / var[:, None])
            rzz.append((g[:, self.n3 // 2, None, :] * g).sum(2) / self.n1 / var[:, None])
            rxy.append((g[0, :, self.n1 // 2, None] * g).sum(1) / self.n3 / torch.sqrt(var * var[0])[:, None])
        for k, t in (("xspec", xs), ("zspec", zs), ("rxx", rxx), ("rzz", rzz), ("rxy", rxy)):
            out[k] = torch.stack(t).permute(2, 1, 0)
        uv = uc * vc
        sign = [(uc > 0) & (vc > 0), (uc < 0) & (vc > 0), (uc < 0) & (vc < 0), (uc > 0) & (vc < 0)]
        out["quadrants"] = torch.stack([-m(torch.where(s, uv, 0.0)) for s in sign] + [m(s.double()) for s in sign], 1)
        return out


# ------------------------------------------------------------------------------------
# What a program holds, and its pass
# ------------------------------------------------------------------------------------
def _grid(case):
    return Grid(n1m=case["n1m"], n2m=case["n2m"], n3m=case["n3m"], alx=case["alx"], aly=2.0, alz=case["alz"],
                re=case["re"], cks=case["cks"], wmodel=case["wmodel"], files=case["files"],
                precision=PRECISION[case["precision"]])


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available())


class Fields:
    """The Fortran arrays U, P, HH of one or more channels in page-locked host memory, and the
    float32 copies that programs of the mixed forms keep."""

    def __init__(self, grids, single):
        self.host, self.single, self.views = {}, {}, [dict() for _ in grids]
        for name, shape in (("U", Grid.shape_u), ("P", Grid.shape_p), ("HH", Grid.shape_u)):
            sizes = [int(np.prod(shape(g))) for g in grids]
            self.host[name] = _pinned(sum(sizes))
            for i, g in enumerate(grids):
                part = self.host[name][sum(sizes[:i]):sum(sizes[:i + 1])]
                self.views[i][name] = part.view(*reversed(shape(g)))
            if single:
                self.single[name] = torch.empty(sum(sizes), dtype=torch.float32)

    def set(self, i, fields):
        for k, t in fields.items():
            self.views[i][k].copy_(t)

    def array(self, i, k):
        return self.views[i][k].numpy().T

    def out(self):
        if not self.single:
            return dict(self.host)
        return {k: self.single[k].copy_(self.host[k]) for k in self.host}


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    members = _members(case) if case["kind"] == "ensemble" else [case]
    grids = [_grid(c) for c in members]
    s.fields = Fields(grids, case["precision"] != "fp64" and case["kind"] != "stats")
    s.dt = case["dt"]
    s.ntime = 1
    if case["kind"] == "ensemble":
        s.batch = lib.Batch(grids)
        channels = s.batch.channels
        s.presg = [[0.0] * len(grids), [0.0] * len(grids)]
    else:
        s.ch = lib.Channel(grids[0])
        channels = [s.ch]
        s.presg = [0.0, 0.0]
    for i, c in enumerate(members):
        flow = Flow(c).start(seed + 1000 * i)
        if case["kind"] == "stats":
            flow.p = flow.w[1:-1] * flow.u[1:-1]
        s.fields.set(i, flow.fortran())
        channels[i].upload(*(s.fields.array(i, k) for k in ("U", "P", "HH")))
    if case.get("schedule"):
        s.ch.set_schedule(dict(zip(lib.Channel.SCHEDULE_KEYS, map(int, case["schedule"].split(",")))))
    if case["kind"] in ("dns", "les"):
        s.ch.set_presg(0.0, 0.0)
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    single = case["precision"] != "fp64"
    num = np.float32 if single else np.float64
    if kind == "stats":
        out = {"stats": s.ch.plane_stats(), "quadrants": s.ch.plane_quadrants()}
        out.update(s.ch.plane_spectra())
        return out
    U, P, HH = (s.fields.array(0, k) for k in ("U", "P", "HH"))
    diag = []
    for _ in range(case["steps"]):
        if kind in ("dns", "les"):
            s.ch.step_async(s.ntime, s.dt)
        elif kind == "driver":
            s.presg = s.ch.step(s.ntime, s.dt, *s.presg)
            d = s.ch.diagnose()
            diag.append([d["cflm"], d["flow1"], d["flow3"], *d["wsm"]])
        elif kind == "getup":
            s.presg = s.ch.getup(U, P, HH, s.ntime, s.dt, *s.presg)
        else:
            n = len(s.batch.channels)
            s.presg = s.batch.step(s.ntime, [s.dt] * n, *s.presg)
        s.ntime += 1
    if kind in ("dns", "les"):
        s.presg = s.ch.get_presg()
    if kind == "ensemble":
        for i, ch in enumerate(s.batch.channels):
            ch.download(*(s.fields.array(i, k) for k in ("U", "P", "HH")))
    elif kind != "getup":
        s.ch.download(U, P, HH)
    out = s.fields.out()
    out["presg"] = np.array(s.presg, dtype=num)
    if diag:
        out["diagnostics"] = np.array(diag, dtype=num)
    if kind == "les":
        out["sgsvis"] = s.ch.download_sgsvis().astype(num)
        out["tauw"], out["taub"] = (t.astype(num) for t in s.ch.download_wall())
    return out


def work(case):
    """Each step reads and writes the state once: u, v, w, P in 8 bytes, the three AB2 terms in the
    working precision; the fields leave once as the driver's FP64 arrays.  Operations: 30 compact solves
    at 6 each, the stencils, products and updates, and the FFTs both ways."""
    members = _members(case) if case["kind"] == "ensemble" else [case]
    nbytes = flops = 0.0
    for c in members:
        n = c["n1m"] * c["n2m"] * c["n3m"]
        r = 8 if case["precision"] == "fp64" else 4
        if case["kind"] == "stats":
            nbytes += n * 32.0 + c["n2m"] * 8.0 * (29 + 8 + 9 * c["n1m"] + 6 * c["n3m"])
            flops += n * (3 * 2.5 * math.log2(c["n1m"] * c["n3m"]) + 120)
            continue
        per = 4 * 8 * 2 + 3 * r * 2
        nbytes += case["steps"] * n * per + 56.0 * n
        if case["kind"] == "getup":
            nbytes += (2 * case["steps"] - 1) * 56.0 * n
        flops += case["steps"] * n * (30 * 6 + 80 + 2 * 2.5 * math.log2(c["n1m"] * c["n3m"]) * 2
                                      + (200 if c["files"] else 0))
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    members = _members(case) if case["kind"] == "ensemble" else [case]
    outs, presg, diag = [], [], []
    for i, c in enumerate(members):
        flow = Flow(c).start(seed + 1000 * i)
        if case["kind"] == "stats":
            flow.p = flow.w[1:-1] * flow.u[1:-1]
            return flow.statistics()
        for _ in range(case["steps"]):
            flow.step()
            if case["kind"] == "driver":
                diag.append(flow.diagnostics())
        outs.append(flow.fortran())
        presg.append(flow.presg)
    out = {k: torch.cat([o[k].reshape(-1) for o in outs]) for k in ("U", "P", "HH")}
    out["presg"] = np.array(presg).T if case["kind"] == "ensemble" else np.array(presg[0])
    if diag:
        out["diagnostics"] = np.array(diag)
    if case["kind"] == "les":
        pad = torch.nn.functional.pad
        out["sgsvis"] = flow.wrap(pad(flow.nu, (0, 0, 0, 0, 1, 1))).permute(2, 1, 0)
        for k, t in zip(("tauw", "taub"), flow.tau):
            full = torch.stack([t, torch.zeros_like(t)])
            out[k] = pad(full, (1, 1, 1, 1)).permute(2, 1, 0)
    return out
