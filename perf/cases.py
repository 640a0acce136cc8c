"""Performance cases of the spectral dynamical core: what its users run, through the public API.

Two kinds of program use this library.  Analysis and coupling code calls the transforms on arrays of
its own (the reference's `!` methods); simulations keep a model on the device, advance it by hours or
days and read its state out.  Both are here, from one level of T21 (launch latency) to ensembles that
exceed the L2 cache, with both directions of the transforms, the forward and the reverse mode of the
Held-Suarez step, and every precision mode.

`exact` restates the transforms and the three models in plain torch FP64 (Sphere, barotropic_steps,
shallow_water_steps, held_suarez_steps); initial states are formed with the same FP64 functions.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "idealizedspectralgcm.jl_gb300"))

# truncation -> (nlat, nlon, time step of the three-dimensional model); T31 and T63 have latitude
# counts that are not powers of two
GRID = {21: (32, 64, 1200), 31: (48, 128, 1200), 42: (64, 128, 1200), 63: (96, 256, 900), 85: (128, 256, 600)}
RADIUS, OMEGA = 6.371e6, 7.292e-5
COMMON = dict(robert_coef=0.04, damping_order=4, omega=OMEGA, grav=9.80, rdgas=287.04, kappa=2.0 / 7.0,
              do_mass_correction=0, do_energy_correction=0, h0=0.0, kappa_m=0.0, kappa_t=0.0, sigma_b=0.7, k_f=1.0,
              k_a=1.0 / 40.0, k_s=1.0 / 4.0, dT_y=60.0, dtheta_z=10.0, ps_ref=1.0e5, t_ref=300.0,
              sea_level_ps_ref=1.0e5, init_t=264.0)
STATE = ("spe_vor_c", "spe_vor_p", "spe_div_c", "spe_div_p", "spe_lnps_c", "spe_lnps_p", "spe_t_c", "spe_t_p",
         "grid_u_c", "grid_u_p", "grid_v_c", "grid_v_p", "grid_ps_c", "grid_ps_p", "grid_t_c", "grid_t_p", "grid_vor",
         "grid_div")
SINGLE_LEVEL = ("spe_lnps_c", "spe_lnps_p", "grid_ps_c", "grid_ps_p")
BARO_OUT = ("spe_vor_c", "spe_vor_p", "grid_u_c", "grid_v_c", "grid_vor")
SW_OUT = ("spe_vor_c", "spe_div_c", "spe_lnps_c", "grid_u_c", "grid_v_c", "grid_ps_c", "grid_vor", "grid_div")


# ------------------------------------------------------------------------------------------------
# the cases
def listed():
    return [
        # one surface field synthesised in host code between other work: the smallest call there is
        {"name": "s2g_t21l1_fp32", "kind": "s2g", "trunc": 21, "levels": 1, "precision": "fp32"},
        # analysis of a whole three-dimensional field in full precision (pre- and post-processing)
        {"name": "g2s_t42l20_fp64", "kind": "g2s", "trunc": 42, "levels": 20, "precision": "fp64"},
        # winds from vorticity and divergence on a grid that is no power of two, an odd level count
        {"name": "uv_t63l13_fp32", "kind": "uv", "trunc": 63, "levels": 13, "precision": "fp32"},
        # vorticity and divergence from winds, the largest truncation, on the tensor-core contraction
        {"name": "vordiv_t85l20_tf32x3", "kind": "vordiv", "trunc": 85, "levels": 20, "precision": "tf32x3"},
        # device buffers of a host with a memory pool of its own (coupled codes): asynchronous, no copies
        {"name": "device_s2g_t42l20_fp32", "kind": "device_s2g", "trunc": 42, "levels": 20, "precision": "fp32"},
        # the barotropic experiment, FP64, one day between outputs
        {"name": "barotropic_t42_fp64", "kind": "barotropic", "trunc": 42, "steps": 48, "precision": "fp64"},
        # the shallow-water experiment at its truncation, six hours between outputs
        {"name": "shallow_water_t85_fp32", "kind": "shallow_water", "trunc": 85, "steps": 36, "precision": "fp32"},
        # the headline: one day of Held-Suarez T42L20, state from and to pinned host memory
        {"name": "hs_t42l20_fp32", "kind": "held_suarez", "trunc": 42, "levels": 20, "members": 1, "tracers": 0,
         "steps": 72, "precision": "fp32"},
        # the same model in full precision, eight hours
        {"name": "hs_t42l20_fp64", "kind": "held_suarez", "trunc": 42, "levels": 20, "members": 1, "tracers": 0,
         "steps": 24, "precision": "fp64"},
        # the small members of the ensemble configuration, all advanced together for a day
        {"name": "hs_t21l20x128_fp32", "kind": "held_suarez", "trunc": 21, "levels": 20, "members": 128, "tracers": 0,
         "steps": 72, "precision": "fp32"},
        # the large members of the ensemble configuration, half a day: the working set exceeds the L2 cache
        {"name": "hs_t42l20x32_fp32", "kind": "held_suarez", "trunc": 42, "levels": 20, "members": 32, "tracers": 0,
         "steps": 36, "precision": "fp32"},
        # a gradient through the model (data assimilation, calibration) at the precision at which it is checked
        # against differences: forward, recompute, reverse
        {"name": "gradient_t42l20_fp64", "kind": "gradient", "trunc": 42, "levels": 20, "steps": 24, "checkpoint": 8,
         "precision": "fp64"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _columns(c):
    return GRID[c["trunc"]][0] * GRID[c["trunc"]][1] * c["levels"]


def draw(rng):
    kind = rng.choice(["s2g", "g2s", "uv", "vordiv", "device_s2g", "barotropic", "shallow_water", "held_suarez",
                       "held_suarez", "held_suarez", "held_suarez", "gradient"])
    c = {"kind": kind}
    if kind in ("s2g", "g2s", "uv", "vordiv", "device_s2g"):
        c["trunc"] = rng.choice([21, 31, 42, 63, 85])
        c["levels"] = rng.randint(1, 30)
        c["precision"] = rng.choice(["fp32", "fp32", "fp64", "tf32x3", "bf16x3"])
        if GRID[c["trunc"]][0] % 32 and c["precision"].endswith("x3"):
            c["precision"] = "fp32"  # the tensor-core modes need nlat to be a multiple of 32
        if kind == "device_s2g":  # its static scratch holds 8 MiB of Fourier coefficients
            size = 16 if c["precision"] == "fp64" else 8
            c["levels"] = min(c["levels"], (8 << 20) // ((c["trunc"] + 1) * GRID[c["trunc"]][0] * size))
    elif kind in ("barotropic", "shallow_water"):
        c["trunc"] = rng.choice([42, 63, 85])
        c["steps"] = rng.randint(12, 36)
        c["precision"] = rng.choice(["fp32", "fp64"])
    elif kind == "gradient":
        c["trunc"] = rng.choice([21, 31, 42])
        c["levels"] = rng.randint(8, 20)
        c["steps"] = rng.randint(6, 24)
        c["checkpoint"] = rng.choice([4, 6, 8])
        c["precision"] = "fp64"
    else:
        c["trunc"] = rng.choice([21, 31, 42, 63])
        c["levels"] = rng.randint(7, 26)
        c["precision"] = rng.choice(["fp32", "fp32", "fp32", "fp64"])
        most = 32 * 64 * 128 * 20 // 4 // _columns(c)  # at most a quarter of the largest case's columns
        c["members"] = _log_int(rng, 1, max(1, most // (4 if c["precision"] == "fp64" else 1)))
        c["tracers"] = rng.choice([0, 0, 1, 3]) if c["members"] <= 4 else 0
        c["steps"] = rng.randint(18, 72 if c["precision"] == "fp32" else 24)
    return c


# ------------------------------------------------------------------------------------------------
# plain FP64 restatement (torch): the sphere and its transforms
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class Sphere:
    """Gaussian grid, normalised Legendre functions (half the integral of P^2 over mu is 1) and the
    transforms of fields [..., lat, lon] and triangular spectra [..., m, n], n = 0 .. N+1."""

    def __init__(self, N, nlat, nlon, a=RADIUS):
        self.N, self.nlat, self.nlon, self.a = N, nlat, nlon, a
        mu, w = np.polynomial.legendre.leggauss(nlat)
        m, n = np.meshgrid(np.arange(N + 1), np.arange(N + 4), indexing="ij")
        eps = np.where(n >= m, np.sqrt(np.maximum(n * n - m * m, 0) / (4.0 * n * n - 1.0)), 0.0)
        eps[0, 0] = 0.0
        c = np.sqrt(1.0 - mu * mu)
        P = np.zeros((N + 1, N + 3, nlat))
        pmm = np.ones(nlat)
        for k in range(N + 1):
            if k:
                pmm = np.sqrt((2 * k + 1) / (2 * k)) * c * pmm
            P[k, k] = pmm
            for q in range(k, N + 2):
                P[k, q + 1] = (mu * P[k, q] - (eps[k, q] * P[k, q - 1] if q > k else 0.0)) / eps[k, q + 1]
        dP = np.zeros((N + 1, N + 2, nlat))  # dP/dmu
        for k in range(N + 1):
            for q in range(k, N + 2):
                dP[k, q] = (-q * eps[k, q + 1] * P[k, q + 1] + ((q + 1) * eps[k, q] * P[k, q - 1] if q > k else 0.0)) / c ** 2
        e, m, n = eps[:, :N + 2], m[:, :N + 2], n[:, :N + 2]
        e1 = np.where(n <= N, eps[:, 1:N + 3], 0.0)
        tri = n >= m
        n1 = np.maximum(n, 1)

        def t(x):
            return torch.tensor(np.ascontiguousarray(x), dtype=torch.float64, device=_device())

        self.mu, self.w, self.cos = t(mu), t(w), t(c)[:, None]
        self.P = t(P[:, :N + 2])
        self.PW = t(P[:, :N + 2] * w * 0.5)
        self.CA = t(P[:, :N + 2] * w / c ** 2 * np.arange(N + 1)[:, None, None] / (2 * a))
        self.CB = t(-dP * w / (2 * a))
        self.tri = t(tri)
        self.eig = t(np.where(tri, -n * (n + 1.0) / a ** 2, 0.0))
        self.dlam, self.dthm, self.dthp = t(tri * m / a), t(tri * -(n - 1) * e / a), t(tri * (n + 2) * e1 / a)
        self.uvm, self.uvc, self.uvp = t(tri * a * e / n1), t(tri * -a * m / (n1 * (n1 + 1.0))), t(tri * -a * e1 / (n + 1))
        self.coriolis = 2 * OMEGA * self.mu[:, None]

    def _sum(self, x, table, spec):
        return torch.complex(torch.einsum(spec, x.real, table), torch.einsum(spec, x.imag, table))

    def _fourier(self, g):
        return (torch.fft.rfft(g, dim=-1)[..., :self.N + 1] / self.nlon).transpose(-1, -2)  # [..., m, j]

    def to_grid(self, s):
        f = self._sum(s * self.tri, self.P, "...mn,mnj->...mj")
        return torch.fft.irfft(f.transpose(-1, -2), n=self.nlon, dim=-1) * self.nlon

    def _last_row_zero(self, s):
        keep = torch.ones(self.N + 2, dtype=torch.float64, device=s.device)
        keep[-1] = 0
        return s * keep

    def to_spec(self, g):
        return self._last_row_zero(self._sum(self._fourier(g), self.PW, "...mj,mnj->...mn"))

    def vor_div(self, ucos, vcos):
        """from u cos(lat), v cos(lat)"""
        fu, fv = self._fourier(ucos), self._fourier(vcos)
        s = "...mj,mnj->...mn"
        return (self._last_row_zero(1j * self._sum(fv, self.CA, s) - self._sum(fu, self.CB, s)),
                self._last_row_zero(1j * self._sum(fu, self.CA, s) + self._sum(fv, self.CB, s)))

    @staticmethod
    def _dn(s):  # the value at n - 1
        return torch.nn.functional.pad(s[..., :-1], (1, 0))

    @staticmethod
    def _up(s):  # the value at n + 1
        return torch.nn.functional.pad(s[..., 1:], (0, 1))

    def wind(self, vor, div):
        uc = 1j * self.uvc * div - self.uvm * self._dn(vor) - self.uvp * self._up(vor)
        vc = 1j * self.uvc * vor + self.uvm * self._dn(div) + self.uvp * self._up(div)
        return self.to_grid(uc) / self.cos, self.to_grid(vc) / self.cos

    def gradient(self, s):
        return (self.to_grid(1j * self.dlam * s) / self.cos,
                self.to_grid(self.dthp * self._up(s) + self.dthm * self._dn(s)) / self.cos)

    def damping(self, coef, order):
        return coef * (self.eig / self.eig[0, self.N]) ** order


@functools.lru_cache(maxsize=8)
def _sphere(trunc):
    return Sphere(trunc, GRID[trunc][0], GRID[trunc][1])


def _leapfrog(dq, qp, qc, d, dt, r):
    """damping and the Robert-Asselin filtered leapfrog: the new level and the filtered current one"""
    dq = (dq - qp * d) / (1.0 + 2 * dt * d)
    qn = qp + 2 * dt * dq
    return qn, qc + r * (qp - 2 * qc + qn)


def barotropic_steps(sp, p, s, nsteps):
    d = sp.damping(p["damping_coef"], p["damping_order"])
    s = dict(s)
    for _ in range(nsteps):
        av = s["grid_vor"] + sp.coriolis
        dvor, _ = sp.vor_div(av * s["grid_v_c"] * sp.cos, -av * s["grid_u_c"] * sp.cos)
        n, c = _leapfrog(dvor, s["spe_vor_p"], s["spe_vor_c"], d, p["dt"], p["robert_coef"])
        s["spe_vor_p"], s["spe_vor_c"] = c, n
        s["grid_vor"] = sp.to_grid(n)
        s["grid_u_c"], s["grid_v_c"] = sp.wind(n, torch.zeros_like(n))
    return s


def shallow_water_steps(sp, p, s, nsteps):
    d, dt, r, h0 = sp.damping(p["damping_coef"], p["damping_order"]), p["dt"], p["robert_coef"], p["h0"]
    mu = p["implicit_coef"] * 2 * dt
    s = dict(s)
    for _ in range(nsteps):
        u, v, h = s["grid_u_c"], s["grid_v_c"], s["grid_ps_c"]
        gl, gt = sp.gradient(s["spe_lnps_c"])
        av = s["grid_vor"] + sp.coriolis
        dvor, ddiv = sp.vor_div((av * v - p["kappa_m"] * u) * sp.cos, (-av * u - p["kappa_m"] * v) * sp.cos)
        dh = sp.to_spec(-p["kappa_t"] * (h - s["grid_h_eq"]) - (u * gl + v * gt) - h * s["grid_div"])
        hc, hp, dc, dp = s["spe_lnps_c"], s["spe_lnps_p"], s["spe_div_c"], s["spe_div_p"]
        ddiv = ddiv - sp.eig * (sp.to_spec(0.5 * (u * u + v * v)) + hc) + sp.eig * (hc - hp)
        dh = dh + h0 * (dc - dp)
        ddiv = (ddiv - mu * sp.eig * dh) / (1.0 - mu * mu * sp.eig * h0)
        dh = dh - mu * h0 * ddiv
        vn, vc = _leapfrog(dvor, s["spe_vor_p"], s["spe_vor_c"], d, dt, r)
        dn, dc = _leapfrog(ddiv, dp, dc, d, dt, r)
        hn, hc = _leapfrog(dh, hp, hc, d, dt, r)
        s.update(spe_vor_p=vc, spe_vor_c=vn, spe_div_p=dc, spe_div_c=dn, spe_lnps_p=hc, spe_lnps_c=hn)
        s["grid_vor"], s["grid_div"], s["grid_ps_c"] = sp.to_grid(vn), sp.to_grid(dn), sp.to_grid(hn)
        s["grid_u_c"], s["grid_v_c"] = sp.wind(vn, dn)
    return s


class Vertical:
    """Evenly spaced sigma levels and the semi-implicit solver's reference column."""

    def __init__(self, nd, p):
        b = np.arange(nd + 1) / nd
        db = np.diff(b)
        lb = np.log(np.maximum(b, 1e-300))
        cf = np.array([lb[1] - 1.0] + [lb[k + 1] + b[k] * (lb[k + 1] - lb[k]) / db[k] - 1.0 for k in range(1, nd)])
        self.nd = nd
        dev = _device()

        def t(x):
            return torch.tensor(x, dtype=torch.float64, device=dev)

        def col(x):
            return t(x)[:, None, None]

        self.b_lo, self.b_hi, self.db, self.cf, self.sigma = col(b[:-1]), col(b[1:]), col(db), col(cf), col(np.exp(cf))
        dlp = np.concatenate([[0.0], np.diff(lb)[1:]])
        dlpp = lb[1:] - cf
        dlpm = np.concatenate([[0.0], cf[1:] - lb[1:-1]])
        self.dlp, self.dlpp, self.dlpm = col(dlp), col(dlpp), col(dlpm)
        # reference column
        kappa, R, T0, ps = p["kappa"], p["rdgas"], p["t_ref"], p["ps_ref"]
        ph = b * ps
        dpr = np.diff(ph)
        lh = np.concatenate([[0.0], np.log(ph[1:])])
        lf = np.array([lh[1] - 1.0] + [lh[k + 1] + ph[k] * (lh[k + 1] - lh[k]) / dpr[k] - 1.0 for k in range(1, nd)])
        dh, dhf = np.diff(lh), lh[1:] - lf
        # temperature tendency of a divergence column (uniform reference temperature: no vertical advection)
        low = np.tril(np.ones((nd, nd)), -1) * dpr[None, :]
        tau = -kappa * T0 * (low * dh[:, None] + np.diag(dpr * dhf)) / dpr[:, None]
        # geopotential of a temperature column
        up = np.triu(np.ones((nd, nd)), 1) * (R * dh)[None, :]
        gamma = up + np.diag(R * dhf)
        dlh = np.concatenate([[0.0], b[1:] / ph[1:]])
        dlf = (b[1:] * (lh[1:] - lf) + b[:-1] * (lf - lh[:-1])) / dpr
        h1 = R * T0 * dlf
        g2 = np.zeros(nd + 1)
        for k in range(nd - 1, 0, -1):
            g2[k] = g2[k + 1] + R * T0 * (dlh[k + 1] - dlh[k])
        h = h1 + g2[1:] + R * T0 * (dlh[1:] - dlf)
        self.tau, self.gamma, self.nu, self.h = t(tau), t(gamma), t(dpr), t(h)
        self.div_mat = t(np.outer(h, dpr) - gamma @ tau)


def _levels(mat, x):  # a vertical operator on spectra [..., k, m, n]
    return torch.einsum("rk,...kmn->...rmn", mat.to(torch.complex128), x)


def _advect(x, M, dp):
    """centred vertical advection with the flux M at the lower faces (zero at the surface)"""
    w = dp[..., :-1, :, :] / (dp[..., :-1, :, :] + dp[..., 1:, :, :])
    f = M[..., :-1, :, :] * (x[..., :-1, :, :] + (x[..., 1:, :, :] - x[..., :-1, :, :]) * w)
    pad = torch.nn.functional.pad
    lo, hi, m_lo = pad(f, (0, 0, 0, 0, 1, 0)), pad(f, (0, 0, 0, 0, 0, 1)), pad(M[..., :-1, :, :], (0, 0, 0, 0, 1, 0))
    return (lo - hi + x * (M - m_lo)) / dp


def held_suarez_steps(sp, vc, p, s, nsteps):
    """Leapfrog steps of the Held-Suarez model; fields [member, level, ...]."""
    dt, nd, R, kappa = p["dt"], vc.nd, p["rdgas"], p["kappa"]
    cp, Dt, xi = R / kappa, 2.0 * p["dt"], 2.0 * p["dt"] * p["implicit_coef"]
    damp, rob = sp.damping(p["damping_coef"], p["damping_order"]), p["robert_coef"]
    eye = torch.eye(nd, dtype=torch.float64, device=sp.w.device)
    W = torch.linalg.inv(eye - xi * xi * sp.eig[0, :sp.N + 1, None, None] * vc.div_mat).to(torch.complex128)
    day, sb, sin2 = 86400.0, p["sigma_b"], sp.mu[:, None] ** 2
    cos2 = 1.0 - sin2
    smax = torch.clamp(vc.sigma - sb, min=0.0)
    kv = p["k_f"] / day / (1.0 - sb) * smax
    kt = p["k_a"] / day + (p["k_s"] - p["k_a"]) / day / (1.0 - sb) * smax * cos2 ** 2

    def area(x):
        return (x * sp.w[:, None]).sum((-1, -2), keepdim=True)

    s = dict(s)
    for _ in range(nsteps):
        u, v, t, ps = s["grid_u_c"], s["grid_v_c"], s["grid_t_c"], s["grid_ps_c"]
        up, vp, tp, psp = s["grid_u_p"], s["grid_v_p"], s["grid_t_p"], s["grid_ps_p"]
        # forcing of the previous level
        lpn = vc.cf + torch.log(ps) - math.log(1.0e5)
        teq = torch.clamp((315.0 - p["dT_y"] * sin2 - p["dtheta_z"] * cos2 * lpn) * torch.exp(kappa * lpn), min=200.0)
        du, dv = -kv * up, -kv * vp
        dT = -((up + 0.5 * du * Dt) * du + (vp + 0.5 * dv * Dt) * dv) / cp - kt * (tp - teq)
        ep = 0.5 * ((up + Dt * du) ** 2 + (vp + Dt * dv) ** 2) + cp * (tp + Dt * dT)
        s3, s4 = area(psp), area((ep * vc.db * psp).sum(-3, keepdim=True))
        # dynamics
        gl, gt = sp.gradient(s["spe_lnps_c"])
        gl, gt = gl * ps, gt * ps
        dp = vc.db * ps
        x1 = (vc.b_lo * vc.dlpm + vc.b_hi * vc.dlpp) / dp
        D = s["grid_div"] * dp + vc.db * (u * gl + v * gt)
        incl = torch.cumsum(D, -3)
        tot = incl[..., -1:, :, :]
        du, dv = du - R * t * x1 * gl, dv - R * t * x1 * gt
        dT = dT + kappa * t * (-((incl - D) * vc.dlp + D * vc.dlpp) / dp + u * x1 * gl + v * x1 * gt)
        M = -incl + tot * vc.b_hi
        M = torch.cat([M[..., :-1, :, :], torch.zeros_like(tot)], -3)
        du, dv, dT = du + _advect(u, M, dp), dv + _advect(v, M, dp), dT + _advect(t, M, dp)
        tl, tt = sp.gradient(s["spe_t_c"])
        av = s["grid_vor"] + sp.coriolis
        dT = dT - (u * tl + v * tt)
        du, dv = du + av * v, dv - av * u
        term = R * t * vc.dlp
        phi = torch.flip(torch.cumsum(torch.flip(term, (-3,)), -3), (-3,)) - term + R * t * vc.dlpp
        # spectral tendencies
        dvor, ddiv = sp.vor_div(du * sp.cos, dv * sp.cos)
        ddiv = ddiv - sp.eig * sp.to_spec(phi + 0.5 * (u * u + v * v))
        sT, sl = sp.to_spec(dT), sp.to_spec(-tot / ps)
        vp_, vc_, dp_, dc_ = s["spe_vor_p"], s["spe_vor_c"], s["spe_div_p"], s["spe_div_c"]
        tp_, tc_, lp_, lc_ = s["spe_t_p"], s["spe_t_c"], s["spe_lnps_p"], s["spe_lnps_c"]
        # semi-implicit correction
        nu = vc.nu[:, None, None]
        sT = sT + _levels(vc.tau, dp_ - dc_)
        sl = sl - ((dp_ - dc_) * nu).sum(-3, keepdim=True) / p["ps_ref"]
        t2, l2 = tp_ - tc_ + xi * sT, lp_ - lc_ + xi * sl
        ddiv = ddiv - sp.eig * (_levels(vc.gamma, t2) + vc.h[:, None, None] * p["ps_ref"] * l2)
        solved = torch.einsum("nrk,...kmn->...rmn", W, ddiv[..., :-1])
        ddiv = torch.cat([solved, ddiv[..., -1:]], -1)
        sT = sT + xi * _levels(vc.tau, ddiv)
        sl = sl - xi / p["ps_ref"] * (ddiv * nu).sum(-3, keepdim=True)
        vn, vcf = _leapfrog(dvor, vp_, vc_, damp, dt, rob)
        dn, dcf = _leapfrog(ddiv, dp_, dc_, damp, dt, rob)
        tn, tcf = _leapfrog(sT, tp_, tc_, damp, dt, rob)
        ln, lcf = _leapfrog(sl, lp_, lc_, 0.0, dt, rob)
        if "spe_q_c" in s:  # passive tracers [member, tracer, level, ...]
            q = s["grid_q_c"]
            ql, qt = sp.gradient(s["spe_q_c"])
            w = lambda x: x[:, None]  # noqa: E731
            dq = _advect(q, w(M).expand_as(q), w(dp).expand_as(q)) - (w(u) * ql + w(v) * qt)
            qn, qcf = _leapfrog(sp.to_spec(dq), s["spe_q_p"], s["spe_q_c"], damp, dt, rob)
            s.update(spe_q_c=qn, spe_q_p=qcf, grid_q_p=q, grid_q_c=sp.to_grid(qn))
        un, vn_g = sp.wind(vn, dn)
        Tn, psn = sp.to_grid(tn), torch.exp(sp.to_grid(ln))
        # mass and energy fixers
        en = 0.5 * (un * un + vn_g * vn_g) + cp * Tn
        factor = s3 / area(psn)
        corr = (s4 - factor * area((en * vc.db * psn).sum(-3, keepdim=True))) / (cp * s3)
        first = torch.zeros_like(sp.eig)
        first[0, 0] = 1.0
        s.update(spe_vor_c=vn, spe_vor_p=vcf, spe_div_c=dn, spe_div_p=dcf, spe_t_c=tn + corr * first, spe_t_p=tcf,
                 spe_lnps_c=ln + torch.log(factor) * first, spe_lnps_p=lcf, grid_u_p=u, grid_v_p=v, grid_t_p=t,
                 grid_ps_p=ps, grid_u_c=un, grid_v_c=vn_g, grid_t_c=Tn + corr, grid_ps_c=psn * factor,
                 grid_vor=sp.to_grid(vn), grid_div=sp.to_grid(dn))
    return s


# ------------------------------------------------------------------------------------------------
# inputs, from the seed alone
def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _noise(sp, g, lead, slope=1.5, scale=1.0):
    """a random real field's spectrum, amplitudes falling as (n + 4)^-slope, row N+1 empty"""
    n = torch.arange(sp.N + 2, device=g.device, dtype=torch.float64)
    x = torch.view_as_complex(torch.randn(lead + (sp.N + 1, sp.N + 2, 2), generator=g, device=g.device,
                                          dtype=torch.float64))
    x = x * sp.tri * (n + 4.0) ** -slope * scale
    x = sp._last_row_zero(x)
    x[..., 0, :] = x[..., 0, :].real + 0j
    return x


def _params(case):
    kind, trunc = case["kind"], case["trunc"]
    if kind == "barotropic":
        return dict(COMMON, kind=kind, damping_coef=1.0e-4, implicit_coef=0.0, dt={42: 1800, 63: 1200, 85: 900}[trunc])
    if kind == "shallow_water":
        return dict(COMMON, kind=kind, damping_coef=1.0e-4, implicit_coef=0.5, dt=600, h0=9.80 * 1.0e4)
    return dict(COMMON, kind="held_suarez", damping_coef=1.15741e-4, implicit_coef=0.5, dt=GRID[trunc][2],
                do_mass_correction=1, do_energy_correction=1)


def _barotropic_state(sp, seed):
    """a Rossby-Haurwitz wave 4 with seeded noise on every mode"""
    g = _generator(seed)
    K, R = 7.848e-6, 4
    lat = torch.arcsin(sp.mu)[:, None]
    lon = 2 * math.pi * torch.arange(sp.nlon, device=sp.w.device, dtype=torch.float64) / sp.nlon
    vor = 2 * K * torch.sin(lat) - K * torch.sin(lat) * torch.cos(lat) ** R * (R * R + 3 * R + 2) * torch.cos(R * lon)
    s = sp.to_spec(vor[None]) + _noise(sp, g, (1,), 0.0, 1.0e-7)
    s[..., 0, 0] = 0
    u, v = sp.wind(s, torch.zeros_like(s))
    return dict(spe_vor_c=s, spe_vor_p=s, grid_u_c=u, grid_v_c=v, grid_vor=sp.to_grid(s))


def _shallow_water_state(sp, p, seed):
    """a balanced mid-latitude jet with a height bump and weak seeded turbulence"""
    g = _generator(seed)
    lon_c = float(torch.rand(1, generator=g, device=g.device, dtype=torch.float64)) * 2 * math.pi
    fine = np.linspace(-math.pi / 2, math.pi / 2, 20001)
    jet = 80.0 * np.exp(-((fine - math.pi / 4) / 0.16) ** 2) * np.cos(fine)
    dphi = -sp.a * jet * (2 * OMEGA * np.sin(fine) + jet * np.tan(np.clip(fine, -1.57, 1.57)) / sp.a)
    phi = np.concatenate([[0.0], np.cumsum(0.5 * (dphi[1:] + dphi[:-1]) * np.diff(fine))])
    lat = np.arcsin(sp.mu.cpu().numpy())
    dev = sp.w.device
    u = torch.tensor(np.interp(lat, fine, jet), device=dev)[:, None].expand(sp.nlat, sp.nlon)[None]
    h = torch.tensor(np.interp(lat, fine, phi), device=dev)[:, None]
    lon = 2 * math.pi * torch.arange(sp.nlon, device=dev, dtype=torch.float64) / sp.nlon
    dl = torch.remainder(lon - lon_c + math.pi, 2 * math.pi) - math.pi
    la = torch.tensor(lat, device=dev)[:, None]
    h = h - (h * sp.w[:, None]).sum() / 2 + p["h0"] + 9.80 * 120.0 * torch.cos(la) * torch.exp(
        -(3.0 * dl) ** 2 - (15.0 * (math.pi / 4 - la)) ** 2)
    vor, div = sp.vor_div(u * sp.cos, torch.zeros_like(u))
    vor, div = vor + _noise(sp, g, (1,), 1.0, 2.0e-6), div + _noise(sp, g, (1,), 1.0, 1.5e-6)
    vor[..., 0, 0] = 0
    div[..., 0, 0] = 0
    sh = sp.to_spec(h[None])
    gu, gv = sp.wind(vor, div)
    return dict(spe_vor_c=vor, spe_vor_p=vor, spe_div_c=div, spe_div_p=div, spe_lnps_c=sh, spe_lnps_p=sh, grid_u_c=gu,
                grid_v_c=gv, grid_ps_c=sp.to_grid(sh), grid_vor=sp.to_grid(vor), grid_div=sp.to_grid(div),
                grid_h_eq=torch.zeros_like(gu))


def _held_suarez_state(sp, case, seed):
    """a developed flow: westerlies with a meridional temperature gradient and seeded eddies"""
    g = _generator(seed)
    nd, E = case["levels"], case.get("members", 1)
    z = torch.linspace(1.0, 0.0, nd, device=g.device, dtype=torch.float64)
    vor = _noise(sp, g, (E, nd), 1.5, 2.0e-5)
    vor[..., 0, 1] += 2.0 * (5.0 + 15.0 * z) / (sp.a * math.sqrt(3.0))
    div = _noise(sp, g, (E, nd), 1.5, 1.0e-5)
    vor[..., 0, 0] = 0
    div[..., 0, 0] = 0
    t = _noise(sp, g, (E, nd), 1.5, 5.0)
    t[..., 0, 0] = 285.0 - 70.0 * z
    t[..., 0, 2] += -12.0
    lnps = _noise(sp, g, (E, 1), 2.0, 2.0e-2)
    lnps[..., 0, 0] = math.log(1.0e5)
    u, v = sp.wind(vor, div)
    T, ps = sp.to_grid(t), torch.exp(sp.to_grid(lnps))
    s = {}
    for lev in ("c", "p"):
        s.update({"spe_vor_" + lev: vor, "spe_div_" + lev: div, "spe_lnps_" + lev: lnps, "spe_t_" + lev: t,
                  "grid_u_" + lev: u, "grid_v_" + lev: v, "grid_ps_" + lev: ps, "grid_t_" + lev: T})
    s.update(grid_vor=sp.to_grid(vor), grid_div=sp.to_grid(div))
    nq = case.get("tracers", 0)
    if nq:
        q = _noise(sp, g, (E, nq, nd), 1.5, 1.0)
        q[..., 0, 0] = 2.0
        for lev in ("c", "p"):
            s.update({"spe_q_" + lev: q, "grid_q_" + lev: sp.to_grid(q)})
    return s


def _target(sp, s, seed):
    """observations of an atmosphere nearer to radiative equilibrium, with large-scale seeded departures"""
    t, p = s["grid_t_c"][0], COMMON
    lpn, sin2 = Vertical(t.shape[0], p).cf, sp.mu[:, None] ** 2
    teq = torch.clamp((315.0 - p["dT_y"] * sin2 - p["dtheta_z"] * (1.0 - sin2) * lpn) * torch.exp(p["kappa"] * lpn),
                      min=200.0)
    return t + 0.1 * (teq - t) + sp.to_grid(_noise(sp, _generator(seed + 1), t.shape[:1], 2.0, 5.0))


def _pack(s):
    """the model's state order, each field level-major with m (or longitude) fastest: [member, values]"""
    parts = []
    for k in STATE:
        x = s[k]
        x = torch.view_as_real(x.transpose(-1, -2).resolve_conj().contiguous()) if x.is_complex() else x
        parts.append(x.reshape(x.shape[0], -1))
    return torch.cat(parts, 1)


def _split(case, packed):
    """[member, values] -> {field: [member, values of the field]}"""
    nlat, nlon, _ = GRID[case["trunc"]]
    N, out, off = case["trunc"], {}, 0
    for k in STATE:
        lev = 1 if k in SINGLE_LEVEL else case["levels"]
        n = lev * (2 * (N + 1) * (N + 2) if k.startswith("spe_") else nlat * nlon)
        out[k] = packed[:, off:off + n]
        off += n
    return out


def _host(x):
    """a field [level, lat, lon] or spectrum [level, m, n] as the reference's host array"""
    x = x.permute(1, 2, 0) if x.is_complex() else x.permute(2, 1, 0)
    return np.asfortranarray(x.cpu().numpy())


def _transform_inputs(sp, case, seed):
    g, L = _generator(seed), case["levels"]
    kind = case["kind"]
    if kind in ("s2g", "device_s2g"):
        s = _noise(sp, g, (L,), 1.5, 10.0)
        s[..., 0, 0] = 250.0
        return (s,)
    if kind == "g2s":
        s = _noise(sp, g, (L,), 1.5, 10.0)
        return (250.0 + sp.to_grid(s) + 0.1 * torch.randn((L, sp.nlat, sp.nlon), generator=g, device=g.device,
                                                           dtype=torch.float64),)
    vor, div = _noise(sp, g, (L,), 1.5, 1.0e-4), _noise(sp, g, (L,), 1.5, 5.0e-5)
    vor[..., 0, 0] = 0
    div[..., 0, 0] = 0
    return (vor, div) if kind == "uv" else sp.wind(vor, div)


# ------------------------------------------------------------------------------------------------
def _real(case):
    """the type of the results: FP64 meshes compute in FP64, every other mode holds FP32 values"""
    return np.float64 if case["precision"] == "fp64" else np.float32


def prepare(case, seed):
    import jgcm

    kind, sp = case["kind"], _sphere(case["trunc"])
    nd = case.get("levels", 1)
    mesh = jgcm.Spectral_Spherical_Mesh(sp.N, sp.N + 1, sp.nlat, sp.nlon, nd, sp.a, precision=case["precision"])
    st = {"case": case, "jgcm": jgcm, "mesh": mesh}
    if kind in ("s2g", "g2s", "uv", "vordiv", "device_s2g"):
        ins = _transform_inputs(sp, case, seed)
        if kind == "device_s2g":  # the library's device layout: [m][n][level], mesh precision
            dt = torch.complex128 if case["precision"] == "fp64" else torch.complex64
            st["spec"] = ins[0].permute(1, 2, 0).contiguous().to(dt)
            st["grid"] = torch.zeros((nd, sp.nlat, sp.nlon), device="cuda",
                                     dtype=torch.float64 if case["precision"] == "fp64" else torch.float32)
            st["stream"] = torch.cuda.Stream()  # the host program's own stream
            st["lib"] = jgcm.lib()
            torch.cuda.synchronize()
            return st
        st["in"] = [_host(x) for x in ins]
        make = mesh.spectral if kind in ("g2s", "vordiv") else mesh.grid
        st["out"] = [make(nd) for _ in range(1 if kind in ("s2g", "g2s") else 2)]
        return st
    p = _params(case)
    if kind == "barotropic" or kind == "shallow_water":
        s = _barotropic_state(sp, seed) if kind == "barotropic" else _shallow_water_state(sp, p, seed)
        md = jgcm.Model(mesh, p)
        for name, x in s.items():
            md.set(name, _host(x))
        if kind == "shallow_water":
            md.set("spe_lnps_n", _host(s["spe_lnps_c"]))
        md.update_init_step()
        st["model"] = md
        return st
    s = _held_suarez_state(sp, case, seed)
    E = case.get("members", 1)
    packed = _pack(s).cpu().pin_memory()
    st["one"] = one = jgcm.Model(mesh, p, num_tracers=case.get("tracers", 0))
    one.update_init_step()
    st["init"] = packed.numpy()
    if kind == "gradient":
        st["target"] = _host(_target(sp, s, seed))
        return st
    st["buf"] = torch.empty_like(packed, pin_memory=True)
    st["rows"] = [st["buf"][e].numpy() for e in range(E)]
    nq = case.get("tracers", 0)
    st["ens"] = ens = one
    if E > 1:
        st["ens"] = ens = jgcm.Model(mesh, p, members=E, num_tracers=nq)
        ens.update_init_step()
    for e in range(E):
        one.set_state(st["init"][e])
        for lev in ("c", "p") if nq else ():
            for f in ("spe", "grid"):
                one.set(f"{f}_tracers_{lev}", _tracer_host(s[f"{f}_q_{lev}"][e]))
        if E > 1:
            ens.copy_member(e, one)
    if E > 1:  # a one-member model past its first step, as the ensemble's: members are read out through it
        st["out"] = one
    return st


def _tracer_host(x):
    """[tracer, level, ...] -> the reference's [.., .., level, tracer]"""
    x = x.permute(2, 3, 1, 0) if x.is_complex() else x.permute(3, 2, 1, 0)
    return np.asfortranarray(x.cpu().numpy())


def run(st):
    case, jg, mesh = st["case"], st["jgcm"], st["mesh"]
    kind = case["kind"]
    if kind == "device_s2g":
        status = st["lib"].jgcm_trans_spherical_to_grid_noalloc(
            mesh._h, ctypes.c_void_p(st["spec"].data_ptr()), case["levels"], ctypes.c_void_p(st["grid"].data_ptr()),
            ctypes.c_void_p(st["stream"].cuda_stream))
        if status:
            raise RuntimeError("jgcm_trans_spherical_to_grid_noalloc: %d" % status)
        return st["grid"]
    if kind in ("s2g", "g2s", "uv", "vordiv"):
        call = {"s2g": jg.Trans_Spherical_To_Grid, "g2s": jg.Trans_Grid_To_Spherical, "uv": jg.UV_Grid_From_Vor_Div,
                "vordiv": jg.Vor_Div_From_Grid_UV}[kind]
        call(mesh, *st["in"], *st["out"])
        return [_kept(case, x) for x in st["out"]]
    if kind in ("barotropic", "shallow_water"):
        st["model"].step(case["steps"])
        return {k: _kept(case, st["model"].get(k)) for k in (BARO_OUT if kind == "barotropic" else SW_OUT)}
    if kind == "gradient":
        st["one"].set_state(st["init"][0])
        loss, g, gp = jg.HS_Gradient(st["one"], case["steps"], st["target"], case["checkpoint"])
        return {"loss": np.array([loss]).astype(_real(case)), "t0": _kept(case, g), "params": gp.astype(_real(case))}
    if case["members"] == 1 and not case["tracers"]:  # a restart: the state comes from the host every time
        st["one"].set_state(st["init"][0])
    st["ens"].step(case["steps"])
    for e in range(case["members"]):
        if case["members"] > 1:
            st["out"].copy_member(0, st["ens"], e)
        st["one"].get_state(out=st["rows"][e])
    out = _split(case, st["buf"] if case["precision"] == "fp64" else st["buf"].float())
    if case["tracers"]:
        for e in range(case["members"]):
            if case["members"] > 1:
                st["out"].copy_member(0, st["ens"], e)
            out["tracers_%d" % e] = _kept(case, st["one"].get("grid_tracers_c"))
    return out


def _kept(case, x):
    """what the program keeps of a host array: FP64 results as they are, the other modes' as FP32"""
    if case["precision"] == "fp64":
        return x
    return x.astype(np.complex64 if x.dtype.kind == "c" else np.float32)


# ------------------------------------------------------------------------------------------------
def exact(case, seed):
    kind, sp = case["kind"], _sphere(case["trunc"])
    if kind in ("s2g", "device_s2g", "g2s", "uv", "vordiv"):
        ins = _transform_inputs(sp, case, seed)
        if kind == "device_s2g":
            return sp.to_grid(ins[0])
        if kind == "s2g":
            out = (sp.to_grid(ins[0]),)
        elif kind == "g2s":
            out = (sp.to_spec(ins[0]),)
        elif kind == "uv":
            out = sp.wind(*ins)
        else:
            out = sp.vor_div(ins[0] * sp.cos, ins[1] * sp.cos)
        return [_host(x * sp.tri if x.is_complex() else x) for x in out]
    p = _params(case)
    if kind == "barotropic":
        s = barotropic_steps(sp, p, _barotropic_state(sp, seed), case["steps"])
        return {k: _host(s[k]) for k in BARO_OUT}
    if kind == "shallow_water":
        s = shallow_water_steps(sp, p, _shallow_water_state(sp, p, seed), case["steps"])
        return {k: _host(s[k]) for k in SW_OUT}
    vc = Vertical(case["levels"], p)
    s = _held_suarez_state(sp, case, seed)
    if kind == "gradient":
        return _exact_gradient(sp, vc, p, s, case, seed)
    s = held_suarez_steps(sp, vc, p, s, case["steps"])
    out = _split(case, _pack(s))
    if case["tracers"]:
        for e in range(case["members"]):
            out["tracers_%d" % e] = _tracer_host(s["grid_q_c"][e])
    return out


def _exact_gradient(sp, vc, p, s, case, seed):
    """reverse mode through the FP64 steps, recomputing each of them"""
    g, target = _generator(seed), _target(sp, s, seed)
    names = ("k_f", "k_a", "k_s", "dT_y", "dtheta_z")
    par = [torch.tensor(float(p[k]), dtype=torch.float64, device=g.device, requires_grad=True) for k in names]
    t0 = s["spe_t_c"].clone().requires_grad_(True)
    T = sp.to_grid(t0)
    s = dict(s, spe_t_c=t0, spe_t_p=t0, grid_t_c=T, grid_t_p=T)
    keys = list(s)

    def step(*args):
        r = held_suarez_steps(sp, vc, dict(p, **dict(zip(names, args[len(keys):]))), dict(zip(keys, args)), 1)
        return tuple(r[k] for k in keys)

    vals = tuple(s[k] for k in keys)
    for _ in range(case["steps"]):
        vals = torch.utils.checkpoint.checkpoint(step, *vals, *par, use_reentrant=False)
    d = dict(zip(keys, vals))["grid_t_c"][0] - target
    loss = (d * d * sp.w[:, None]).sum() / (2 * sp.nlon * case["levels"])
    loss.backward()
    return {"loss": loss.detach().reshape(1).cpu().numpy(), "t0": _host(sp._last_row_zero(t0.grad[0] * sp.tri)),
            "params": np.array([float(x.grad) for x in par])}


# ------------------------------------------------------------------------------------------------
def work(case):
    """One pass: every input read once and every output written once, at the precision that the path
    holds them in; the model cases count each step's state read and written once (the level-coupled
    fields of one step are the inputs of the next) and the state's read-out."""
    N, (nlat, nlon, _) = case["trunc"], GRID[case["trunc"]]
    nd, kind = case.get("levels", 1), case["kind"]
    es = 8 if case["precision"] == "fp64" else 4
    modes = (N + 1) * (N + 4) // 2
    G, S = nlat * nlon, 2 * modes
    legendre = 2.0 * 2 * modes * nlat / 2          # one field and level: even and odd halves
    fft = 2.5 * nlat * nlon * math.log2(nlon)
    one = legendre + fft
    if kind in ("s2g", "g2s", "uv", "vordiv", "device_s2g"):
        nf = 2 if kind in ("uv", "vordiv") else 1
        host = es if kind == "device_s2g" else 8
        return {"bytes": nf * nd * (G + S) * host, "flops": nf * nd * (one + (legendre if kind == "vordiv" else 0))}
    if kind == "barotropic":
        step = {"bytes": (6 * G + 4 * S) * es, "flops": 5 * one}
        return {"bytes": step["bytes"] * case["steps"] + 3 * G * 8 + 2 * S * 8, "flops": step["flops"] * case["steps"]}
    if kind == "shallow_water":
        step = {"bytes": (11 * G + 15 * S) * es, "flops": 13 * one}
        return {"bytes": step["bytes"] * case["steps"] + 5 * G * 8 + 3 * S * 8, "flops": step["flops"] * case["steps"]}
    # Held-Suarez: reads u, v, T, ps of two levels, vor, div and the spectra's two levels; writes the
    # new level of the grid state, vor, div and the spectra's new and filtered levels
    E, nq = case.get("members", 1), case.get("tracers", 0)
    state = (10 * nd + 2) * G + (6 * nd + 2) * S
    step_bytes = E * es * ((6 * nd + 2) * G + (5 * nd + 1) * G + 2 * nd * G + (6 * nd + 2) * S + (6 * nd + 2) * S
                           + nq * nd * (2 * G + 4 * S))
    step_flops = E * ((11 * nd + 4 + 4 * nq * nd) * one + 250.0 * nd * G + 8.0 * modes * nd * nd)
    if kind == "gradient":  # forward, recomputation and a reverse step of about twice the forward's work
        return {"bytes": 4.0 * step_bytes * case["steps"] + 8.0 * state, "flops": 4.0 * step_flops * case["steps"]}
    return {"bytes": step_bytes * case["steps"] + 8.0 * E * state, "flops": step_flops * case["steps"]}
