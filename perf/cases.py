"""Timed workloads of the library, through its public entry points.

A case is a dict of plain values.  ``kind`` names the entry point, ``bodies``,
``npts`` and ``nouter`` the geometry's sizes:

* ``operator``  one application of the boundary operator from host arrays
                (``stokes.matvec``, the reference's near rules, FP64);
* ``noalloc``   the trapezoid operator on device pointers and the caller's
                stream (``erosion_matvec_noalloc``), as a program with its own
                Krylov loop on the GPU calls it;
* ``solve``     the drop-in solve of the reference: unrestarted FP64 GMRES to
                1e-8 (``stokes.solve``);
* ``step``      one RK2 erosion step from host arrays (``erosion_rk2_step``):
                two solves, two shear stresses, the theta-L update.  ``mixed``
                is the production method (FP32 far field in FP64 refinement,
                block preconditioner), otherwise the reference's plain FP64
                loop with its fixed pressure drop;
* ``stress``    wall shear stress of a density (``stokes.shear_stress``);
* ``targets``   velocity, pressure and vorticity on a grid of ``targets``
                points (``stokes.qoi_targets``);
* ``ensemble``  ``geometries`` independent channels in one call
                (``stokes.solve_batch``), body counts between half of
                ``bodies`` and ``bodies``.

Densities handed to operator, stress and targets are what a solve returns in
kind: smooth on the wall, on every body a rigid motion plus Fourier content
that decays, and stokeslet/rotlet strengths.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from erosion_b200 import _lib, geometry as G, stokes

# ---------------------------------------------------------------------------
# The cases.


def listed():
    return [
        # the smallest call: three bodies in the reference's wall, all near rules active
        dict(name="operator_3x64", kind="operator", bodies=3, npts=64, nouter=256),
        # a caller's own GPU-resident Krylov loop on the 10-circle channel
        dict(name="noalloc_10x128", kind="noalloc", bodies=10, npts=128, nouter=1024),
        # an operator application of the 100-body and of the 400-body channel
        dict(name="operator_100x256", kind="operator", bodies=100, npts=256, nouter=2048),
        dict(name="operator_400x256", kind="operator", bodies=400, npts=256, nouter=4096),
        # the drop-in solve that the reference's Julia code calls, 10 circles
        dict(name="solve_10x128", kind="solve", bodies=10, npts=128, nouter=1024),
        # the reference's own loop at a small size: one plain FP64 step, fixed pressure drop
        dict(name="step_3x64", kind="step", mixed=False, bodies=3, npts=64, nouter=256, tol=1e-8, dt=1e-4),
        # production erosion steps: 100 perturbed bodies, and 200 bodies with 4096 wall nodes
        dict(name="step_100x256", kind="step", mixed=True, bodies=100, npts=256, nouter=2048, tol=1e-9, dt=5e-7),
        dict(name="step_200x256", kind="step", mixed=True, bodies=200, npts=256, nouter=4096, tol=1e-9, dt=1e-7),
        # shear stress of a run's saved states: sizes that fill no tile, and the 400-body channel
        dict(name="stress_37x200", kind="stress", bodies=37, npts=200, nouter=1000),
        dict(name="stress_400x256", kind="stress", bodies=400, npts=256, nouter=4096),
        # a picture of the flow: velocity, pressure and vorticity on an 80 x 40 grid
        dict(name="targets_50x128", kind="targets", bodies=50, npts=128, nouter=1024, targets=3200),
        # an ensemble of small porous channels solved together, to a tight tolerance
        dict(name="ensemble_12x40x128", kind="ensemble", geometries=12, bodies=40, npts=128, nouter=1024, tol=1e-11),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(rng, lo, hi):
    return 2 * _log(rng, lo // 2, hi // 2)


def draw(rng):
    kind = rng.choice(["operator", "operator", "noalloc", "solve", "step", "step", "stress", "stress", "targets",
                       "ensemble"])
    c = {"kind": kind}
    if kind in ("operator", "stress"):
        c.update(bodies=_log(rng, 3, 400), npts=_even(rng, 64, 256), nouter=_even(rng, 512, 4096))
    elif kind == "noalloc":
        c.update(bodies=_log(rng, 3, 96), npts=_even(rng, 64, 256), nouter=_even(rng, 512, 4096))
    elif kind == "solve":
        c.update(bodies=_log(rng, 3, 12), npts=_even(rng, 64, 160), nouter=_even(rng, 512, 1536))
    elif kind == "step" and rng.random() < 0.4:
        c.update(mixed=False, bodies=_log(rng, 2, 5), npts=_even(rng, 64, 128), nouter=_even(rng, 256, 768), tol=1e-8,
                 dt=1e-4)
    elif kind == "step":
        c.update(mixed=True, bodies=_log(rng, 16, 120), npts=_even(rng, 96, 256), nouter=_even(rng, 1024, 3072),
                 tol=1e-9, dt=1e-7)
    elif kind == "targets":
        c.update(bodies=_log(rng, 5, 100), npts=_even(rng, 64, 192), nouter=_even(rng, 512, 2048),
                 targets=_log(rng, 400, 6000))
    else:
        c.update(geometries=_log(rng, 4, 12), bodies=_log(rng, 16, 40), npts=_even(rng, 64, 128),
                 nouter=_even(rng, 512, 1024), tol=1e-11)
    return c


# ---------------------------------------------------------------------------
# Inputs.


def _reference_wall(case):
    """The small plain-step and operator geometries sit in the reference's 3 x 1 wall."""
    return case["kind"] in ("step", "operator") and not case.get("mixed") and case["bodies"] <= 5


def _geometry(case, seed):
    M, n, nout = case["bodies"], case["npts"], case["nouter"]
    rng = np.random.default_rng([seed, 1])
    if _reference_wall(case):
        wall, ibc = G.REFERENCE_WALL, 1
        radii, cs = G.pack(M, 0.15, 0.3, (2.0,) + wall[1:], lambda r: 0.1 * r, rng)   # clear of the inlet and outlet
    else:
        named = {(100, 256, 2048): "c2", (400, 256, 4096): "c3", (200, 256, 4096): "c5", (10, 128, 1024): "c1"}
        if (M, n, nout) in named:   # the repository's own workloads of these sizes
            return G.workload(named[(M, n, nout)], seed)
        wall, ibc = G.CHANNEL_WALL, 0
        radii, cs, _ = G.lattice_pack(M, n, float(rng.uniform(0.6, 0.8)), wall, rng)
    xx, yy = G.make_bodies(n, radii, cs)
    return G.Geometry(n, nout, xx, yy, wall, ibc, radii, cs)


def _density(g, seed):
    """A density as a solve leaves it: see the module's docstring."""
    rng = np.random.default_rng([seed, 2])
    no, n, M = g.nout, g.n, g.M

    def curves(count, npts, modes):
        th = 2 * np.pi * np.arange(npts) / npts
        k = np.arange(1, modes + 1)
        a, b = rng.standard_normal((2, count, modes)) / k ** 2
        return a @ np.cos(np.outer(k, th)) + b @ np.sin(np.outer(k, th))

    den = np.empty(g.ntot)
    den[:2 * no] = 20 * curves(2, no, 24).reshape(-1)
    x, y = g.xx.reshape(M, n), g.yy.reshape(M, n)
    t = 5 * rng.standard_normal((3, M, 1)) / g.radii[:, None]
    rot = t[2] / g.radii[:, None]
    sx = t[0] - rot * (y - y.mean(1, keepdims=True)) + curves(M, n, 20)
    sy = t[1] + rot * (x - x.mean(1, keepdims=True)) + curves(M, n, 20)
    den[2 * no:2 * no + 2 * n * M] = np.stack([sx, sy], 1).reshape(-1)
    den[2 * no + 2 * n * M:] = rng.standard_normal(3 * M)
    return den


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "ensemble":
        count = case["geometries"]
        s["geoms"] = [_geometry(dict(case, bodies=-(-case["bodies"] * (count + k) // (2 * count))), seed + 1000 * k)
                      for k in range(count)]
        return s
    g = s["g"] = _geometry(case, seed)
    if kind == "step":
        s["state"] = G.to_thetalen(g)
    elif kind == "noalloc":
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        s["xx"], s["yy"], s["den"] = dev(g.xx), dev(g.yy), dev(_density(g, seed))
        s["p"] = stokes.params_for(g, ibary=0)
    elif kind != "solve":
        s["den"] = _density(g, seed)
    if kind == "targets":
        a, b, _ = g.wall
        ny = max(1, int(math.sqrt(case["targets"] / 2)))
        nx = -(-case["targets"] // ny)
        x, y = np.meshgrid(0.9 * a * np.linspace(-1, 1, nx), 0.9 * b * np.linspace(-1, 1, ny))   # inside the wall
        s["xt"], s["yt"] = x.reshape(-1)[:case["targets"]].copy(), y.reshape(-1)[:case["targets"]].copy()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "ensemble":
        dens, _, _ = stokes.solve_batch(s["geoms"], precision=1, precond=1, tol=case["tol"])
        return dens
    g = s["g"]
    if kind == "operator":
        return stokes.matvec(g, s["den"])
    if kind == "solve":
        return stokes.solve(g)[0]
    if kind == "stress":
        tau, E = stokes.shear_stress(g, s["den"])
        return {"tau": tau, "E": E}
    if kind == "targets":
        return dict(zip("uvpw", stokes.qoi_targets(g, s["den"], s["xt"], s["yt"])))
    L = _lib.load()
    if kind == "noalloc":
        vel = torch.empty_like(s["den"])
        _lib.check(L.erosion_matvec_noalloc(ctypes.byref(s["p"]), g.n, g.M, g.nout, s["xx"].data_ptr(),
                                            s["yy"].data_ptr(), s["den"].data_ptr(), vel.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
        return vel
    th, ln, xs, ys = (a.copy() for a in s["state"])   # the step updates its arrays in place
    mixed = case["mixed"]
    p = stokes.params_for(g, tol=case["tol"], precision=int(mixed), precond=int(mixed))
    sp = _lib.StepParams()
    L.erosion_default_step_params(ctypes.byref(sp), g.n)
    sp.dt, sp.fixpdrop = case["dt"], int(not mixed)
    nb, t, gone = np.array([g.M], np.int64), np.zeros(1), np.zeros(g.M, np.int64)
    i64 = lambda a: a.ctypes.data_as(_lib.PI64)
    _lib.check(L.erosion_rk2_step(ctypes.byref(p), ctypes.byref(sp), g.n, i64(nb), g.nout, _lib.ptr(th), _lib.ptr(ln),
                                  _lib.ptr(xs), _lib.ptr(ys), _lib.ptr(t), i64(gone)))
    k = int(nb[0])
    return {"theta": th[:k * g.n], "len": ln[:k], "xsm": xs[:k], "ysm": ys[:k], "t": float(t[0]), "bodies": k}


def work(case):
    """Bytes: every input read and every output written once.  Flops: 20 per
    pair of nodes of one curve, which every summation method has to take
    directly, and 20 per node and body for the stokeslets and rotlets nearby;
    a solve counts the operator once per iteration it takes at this size and
    the two Gram-Schmidt passes over its basis."""
    M, n, no = case["bodies"], case["npts"], case["nouter"]
    kind = case["kind"]
    count = case.get("geometries", 1)
    if kind == "ensemble":
        M = 0.75 * M
    N, ntot = no + n * M, 2 * no + 2 * n * M + 3 * M
    op_flops = 20.0 * (M * n * n + no * no)
    op_bytes = 8.0 * (2 * n * M + 2 * ntot)
    its = {"solve": 180, "ensemble": 500, "step": 600 if case.get("mixed") else 130}.get(kind, 1)
    if kind in ("solve", "ensemble", "step"):
        cyc = its / 2 if kind == "step" else its   # two solves a step
        krylov = (its / cyc) * 8.0 * ntot * cyc * cyc   # flops: four passes of k columns, k = 1..cyc
        return {"bytes": count * (its * op_bytes + krylov), "flops": count * (its * op_flops + krylov)}
    if kind == "stress":
        return {"bytes": 8.0 * (2 * n * M + ntot + 4 * n * M), "flops": 2 * op_flops}
    if kind == "targets":
        t = case["targets"]
        return {"bytes": 8.0 * (2 * n * M + ntot + 6 * t), "flops": 20.0 * t * (n + M)}
    return {"bytes": op_bytes, "flops": op_flops}


# ---------------------------------------------------------------------------
# The same outputs in plain torch, 64 bits.


class _Curves:
    """Nodes, normals (the wall's negated), speeds, weights and curvature of
    every curve, by FFT differentiation with the Nyquist mode zeroed."""

    def __init__(self, g):
        self.g = g
        t = 2 * np.pi * np.arange(g.nout) / g.nout
        a, b, p = g.wall
        r = (np.abs(np.cos(t)) ** p + np.abs(np.sin(t)) ** p) ** (-1 / p)
        zs = [(a * r * np.cos(t) + 1j * b * r * np.sin(t))[None], (g.xx + 1j * g.yy).reshape(g.M, g.n)]
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.parts = []
        for q, z in enumerate(zs):
            z = torch.from_numpy(z).to(self.dev)
            d1, d2 = self.diff(z), self.diff(self.diff(z))
            s = d1.abs()
            nrm = 1j * d1 / s
            cur = (d1.imag * d2.real - d1.real * d2.imag) / s ** 3
            if q == 0:
                nrm, cur = -nrm, -cur
            self.parts.append(dict(z=z, d1=d1, sp=s, nrm=nrm, cur=cur, dz=d1 * 2 * math.pi / z.shape[1],
                                   w=2 * s / z.shape[1]))
        flat = lambda k: torch.cat([q[k].reshape(-1) for q in self.parts])
        self.z, self.nrm, self.sp, self.w = flat("z"), flat("nrm"), flat("sp"), flat("w")
        self.cen = self.parts[1]["z"].mean(1)
        self.rad = self.parts[1]["sp"].mean(1)

    @staticmethod
    def diff(f):
        n = f.shape[-1]
        k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=f.device)
        k[n // 2] = 0
        return torch.fft.ifft(1j * k * torch.fft.fft(f, dim=-1), dim=-1)

    def split(self, den):
        """sigma of every node as a complex number, and (l1, l2, xi) of every body."""
        g = self.g
        d = torch.from_numpy(np.asarray(den)).to(self.dev)
        w = torch.complex(d[:g.nout], d[g.nout:2 * g.nout])
        b = d[2 * g.nout:2 * g.nout + 2 * g.n * g.M].reshape(g.M, 2, g.n)
        return torch.cat([w, torch.complex(b[:, 0], b[:, 1]).reshape(-1)]), d[2 * g.nout + 2 * g.n * g.M:].reshape(-1, 3)

    def curve(self, c):
        part, row = (self.parts[0], 0) if c == 0 else (self.parts[1], c - 1)
        return {k: v[row] for k, v in part.items()}

    def nodes(self, c):
        g = self.g
        return slice(0, g.nout) if c == 0 else slice(g.nout + (c - 1) * g.n, g.nout + c * g.n)

    def layers(self, sig, c, zt, gradient):
        """Barycentric Stokes double layer of curve c at the points zt:
        (u + i v, and with gradient u_x, u_y, v_x, v_y)."""
        q = self.curve(c)
        s, z, dz = sig[self.nodes(c)], q["z"], q["dz"]
        nx, ny = q["nrm"].real, q["nrm"].imag
        f = torch.stack([z.real * s.real + z.imag * s.imag + 0j, s.real + 0j, s.imag + 0j, s * nx / q["nrm"],
                         s * ny / q["nrm"]])
        n = len(z)
        d = z[None, :] - z[:, None]
        d.fill_diagonal_(1.0)
        cc = dz[None, :] / d
        cc.fill_diagonal_(0.0)
        S = -(f @ cc.T - f * cc.sum(1)) - 2 * math.pi / n * self.diff(f)
        b = -1j * S / (2 * math.pi) - f if c == 0 else 1j * S / (2 * math.pi)
        d = z[None, :] - zt[:, None]
        c1 = dz / d
        den = c1.sum(1)
        u = (c1 @ b.T) / (den - (0 if c == 0 else 2j * math.pi))[:, None]
        if c == 0:
            fac = 1 / den
        else:
            a = self.cen[c - 1]
            fac = 1 / ((zt - a) * (c1 / (z - a)).sum(1))
        bu = [b[k][None, :] - u[:, k, None] for k in range(5)]
        c2 = c1 / d
        du = [(v * c2).sum(1) * fac for v in bu]
        x, y = zt.real, zt.imag
        vel = torch.complex(du[0].real - x * du[1].real - y * du[2].real + u[:, 3].real,
                            -du[0].imag + x * du[1].imag + y * du[2].imag + u[:, 4].real)
        if not gradient:
            return vel
        c3 = c2 / d
        h = [2 * ((v - du[k][:, None] * d) * c3).sum(1) * fac for k, v in enumerate(bu)]
        return (vel, h[0].real - du[1].real - x * h[1].real - y * h[2].real + du[3].real,
                -h[0].imag + x * h[1].imag - du[2].real + y * h[2].imag - du[3].imag,
                -h[0].imag + du[1].imag + x * h[1].imag + y * h[2].imag + du[4].real,
                -h[0].real + x * h[1].real + du[2].imag + y * h[2].real - du[4].imag)

    def near_pairs(self):
        """Target nodes of every source curve that the reference's rules give
        to the barycentric formulas."""
        g = self.g
        bh = g.wall[1]
        z, cen, rad = self.z.cpu().numpy(), self.cen.cpu().numpy(), self.rad.cpu().numpy()
        lw = 0
        for v in self.parts[0]["sp"][0].cpu().numpy():
            lw = int(lw + v)
        lw //= g.nout
        near = [set() for _ in range(g.M + 1)]
        idx = np.arange(g.n)
        for b in range(g.M):
            lim = bh - (rad[b] + 4.0 * lw * 2 * np.pi / g.nout)
            if abs(cen[b].imag) >= lim:
                k = g.nout + b * g.n + idx
                near[0].update(k[np.abs(z[k].imag) >= lim])
                near[1 + b].update(np.flatnonzero(np.abs(z[:g.nout] - cen[b]) <= bh - abs(cen[b].imag) + 2 * rad[b]))
            rs = (rad[b] + rad) * (1 + 4.0 * 2 * np.pi / g.n)
            for t in np.flatnonzero(np.abs(cen - cen[b]) <= rs):
                if t != b:
                    k = g.nout + t * g.n + idx
                    near[1 + b].update(k[np.abs(z[k] - cen[b]) <= rs[t]])
        return [np.array(sorted(v), dtype=np.int64) for v in near]

    def operator(self, sig, lam, near):
        g = self.g
        N = len(self.z)
        out = torch.zeros_like(self.z)
        v = self.w * sig
        cut = torch.zeros((N, g.M + 1), dtype=torch.bool, device=self.dev)
        if near is not None:
            for c, k in enumerate(near):
                if len(k):
                    k = torch.from_numpy(k).to(self.dev)
                    cut[k, c] = True
                    out[k] += self.layers(sig, c, self.z[k], False)
        own = torch.cat([torch.zeros(g.nout, dtype=torch.long), 1 + torch.arange(g.M).repeat_interleave(g.n)]).to(self.dev)
        step = max(1, int(5e7) // N)
        for i in range(0, N, step):
            zi = self.z[i:i + step]
            r = zi[:, None] - self.z[None, :]
            rho2 = r.real ** 2 + r.imag ** 2
            q = (r.real * self.nrm.real + r.imag * self.nrm.imag) * (r.real * v.real + r.imag * v.imag) / rho2 ** 2
            q = torch.where(cut[i:i + step][:, own], 0.0, q)
            k = torch.arange(len(zi), device=self.dev)
            q[k, i + k] = 0.0
            out[i:i + step] += torch.complex((q * r.real).sum(1), (q * r.imag).sum(1))
        cnt = torch.cat([torch.full((g.nout,), g.nout), torch.full((N - g.nout,), g.n)]).to(self.dev)
        cur = torch.cat([q["cur"].reshape(-1) for q in self.parts])
        tdd = self.nrm.imag * sig.real - self.nrm.real * sig.imag
        out += cur * tdd * self.sp / cnt * torch.complex(-self.nrm.imag, self.nrm.real) - 0.5 * sig
        for b in range(g.M):
            r = self.z - self.cen[b]
            l = torch.complex(lam[b, 0], lam[b, 1])
            rho2 = r.abs() ** 2
            out += (-0.5 * torch.log(rho2) * l + (r.real * lam[b, 0] + r.imag * lam[b, 1]) / rho2 * r) / (4 * math.pi)
            out += -1j * lam[b, 2] * r / rho2
        wall = slice(0, g.nout)
        flux = ((self.nrm.conj() * sig).real * self.sp)[wall].sum() * 2 * math.pi / g.nout
        out[wall] += flux * self.nrm[wall]
        sb, zb, spb = (a[g.nout:].reshape(g.M, g.n) for a in (sig, self.z, self.sp))
        rows = torch.stack([lam[:, 0] - (sb.real * spb).mean(1), lam[:, 1] - (sb.imag * spb).mean(1),
                            lam[:, 2] - ((sb * zb.conj()).conj().imag * spb).mean(1)], 1)
        ub = out[g.nout:].reshape(g.M, g.n)
        return torch.cat([out[wall].real, out[wall].imag, torch.stack([ub.real, ub.imag], 1).reshape(-1),
                          rows.reshape(-1)])

    def stress(self, sig, lam):
        g = self.g
        zb = self.z[g.nout:]
        e = torch.zeros((3, g.M * g.n), dtype=torch.float64, device=self.dev)
        for c in range(g.M + 1):
            keep = torch.ones(g.M * g.n, dtype=torch.bool, device=self.dev)
            if c:
                keep[(c - 1) * g.n:c * g.n] = False
            at = torch.nonzero(keep).reshape(-1)
            for k in at.split(max(1, int(3e7) // len(self.curve(c)["z"]))):
                _, ux, uy, vx, vy = self.layers(sig, c, zb[k], True)
                e[:, k] += torch.stack([ux, 0.5 * (uy + vx), vy])
        sb = sig[g.nout:].reshape(g.M, g.n)
        odd = torch.arange(g.n, device=self.dev)
        odd = (odd[:, None] - odd[None, :]) % 2 == 1
        for b in range(g.M):
            q = self.curve(1 + b)
            z, s = q["z"], sb[b]
            r = z[:, None] - z[None, :]
            ds = s[None, :] - s[:, None]
            r2 = torch.where(odd, r.abs() ** 2, 1.0)
            wg = torch.where(odd, q["w"][None, :] + 0 * r2, 0.0)
            rx, ry, px, py, sx, sy = r.real, r.imag, q["nrm"].real[None], q["nrm"].imag[None], ds.real, ds.imag
            rn, ro, rs, rt = rx * px + ry * py, rx * py + ry * px, rx * sx + ry * sy, rx * sy + ry * sx
            i4, i6 = 1 / r2 ** 2, 1 / r2 ** 3
            e11 = ((2 * rn * rs + 2 * rs * rx * px + 2 * rn * rx * sx) * i4 - 8 * rn * rs * i6 * rx * rx) * wg
            e12 = ((rs * ro + rn * rt) * i4 - 8 * rn * rs * rx * ry * i6) * wg
            e22 = ((2 * rn * rs + 2 * rs * ry * py + 2 * rn * ry * sy) * i4 - 8 * rn * rs * i6 * ry * ry) * wg
            t = -1j * q["nrm"] * -1     # the tangent (-n_y, n_x)
            dd = (self.diff(s) / q["sp"] * t.conj()).real
            tx, ty = t.real, t.imag
            k = slice(b * g.n, (b + 1) * g.n)
            e[0, k] += e11.sum(1) + 0.5 * dd * (tx * tx - ty * ty)
            e[1, k] += e12.sum(1) + dd * tx * ty
            e[2, k] += e22.sum(1) - 0.5 * dd * (tx * tx - ty * ty)
        for b in range(g.M):
            r = zb - self.cen[b]
            rx, ry = r.real, r.imag
            i2 = 1 / r.abs() ** 2
            rd = rx * lam[b, 0] + ry * lam[b, 1]
            k, xi = 1 / (4 * math.pi), lam[b, 2]
            e[0] += k * (rd * i2 - 2 * rx * rx * rd * i2 ** 2) - 2 * xi * rx * ry * i2 ** 2
            e[1] += -2 * k * rd * rx * ry * i2 ** 2 + xi * (rx * rx - ry * ry) * i2 ** 2
            e[2] += k * (rd * i2 - 2 * ry * ry * rd * i2 ** 2) + 2 * xi * rx * ry * i2 ** 2
        nx, ny = self.nrm.real[g.nout:], self.nrm.imag[g.nout:]
        tx, ty = -2 * (e[0] * nx + e[1] * ny), -2 * (e[1] * nx + e[2] * ny)
        return {"tau": tx * ny - ty * nx, "E": e}

    def targets(self, sig, lam, zt):
        g = self.g
        vel, p, w = torch.zeros_like(zt), torch.zeros_like(zt.real), torch.zeros_like(zt.real)
        for c in range(g.M + 1):
            v, _, uy, vx, _ = self.layers(sig, c, zt, True)
            vel, w = vel + v, w + vx - uy
            k = self.nodes(c)
            r = zt[:, None] - self.z[k][None, :]
            r2 = r.abs() ** 2
            rn, rs = (r.conj() * self.nrm[k]).real, (r.conj() * sig[k]).real
            p = p + ((2 * rn * rs / r2 ** 2 - (self.nrm[k].conj() * sig[k]).real / r2) * self.w[k]).sum(1)
        for b in range(g.M):
            r = zt - self.cen[b]
            r2 = r.abs() ** 2
            l = torch.complex(lam[b, 0], lam[b, 1])
            rd = (r.conj() * l).real
            vel = vel + (-0.5 * torch.log(r2) * l + rd / r2 * r) / (4 * math.pi) - 1j * lam[b, 2] * r / r2
            p = p + rd / r2 / (2 * math.pi)
            w = w + (l * r.conj()).conj().imag / r2 / (2 * math.pi)
        zb, nb = self.z[g.nout:], self.nrm[g.nout:]
        k = torch.cat([(t[:, None] - zb[None, :]).abs().argmin(1) for t in zt.split(512)])
        out = ((zt - zb[k]).conj() * nb[k]).real
        return {n: torch.where(out < 0, v, 0.0) for n, v in zip("uvpw", (vel.real, vel.imag, p, w))}


def _gmres(op, b, tol):
    """Unrestarted GMRES by modified Gram-Schmidt, twice."""
    beta = b.norm()
    V, H = [b / beta], torch.zeros((1, 0), dtype=b.dtype, device=b.device)
    while True:
        w = op(V[-1])
        basis = torch.stack(V)
        h = torch.zeros(len(V), dtype=b.dtype, device=b.device)
        for _ in range(2):
            q = basis @ w
            w, h = w - q @ basis, h + q
        H = torch.cat([torch.cat([H, h[:, None]], 1),
                       torch.cat([torch.zeros((1, H.shape[1]), dtype=b.dtype, device=b.device), w.norm().reshape(1, 1)], 1)])
        V.append(w / w.norm())
        e = torch.zeros(len(V), dtype=b.dtype, device=b.device)
        e[0] = beta
        y = torch.linalg.lstsq(H, e[:, None]).solution[:, 0]
        if (H @ y - e).norm() <= tol * beta or len(V) > 600:
            return y @ basis


def exact(case, seed):
    """Steps and ensembles have no value here: their solves in plain torch
    take minutes."""
    kind = case["kind"]
    if kind in ("step", "ensemble"):
        return None
    s = prepare(case, seed)
    g = s["g"]
    C = _Curves(g)
    if kind == "solve":
        near = C.near_pairs()
        z = C.z[:g.nout]
        b = torch.zeros(g.ntot, dtype=torch.float64, device=C.dev)
        b[:g.nout] = 1 - (z.imag / g.wall[1]) ** 2 if g.ibc == 0 else 1.0
        return _gmres(lambda v: C.operator(*C.split(v.cpu().numpy()), near), b, 1e-12)
    den = s["den"].cpu().numpy() if kind == "noalloc" else s["den"]
    sig, lam = C.split(den)
    if kind == "noalloc":
        return C.operator(sig, lam, None)
    if kind == "operator":
        return C.operator(sig, lam, C.near_pairs())
    if kind == "stress":
        return C.stress(sig, lam)
    return C.targets(sig, lam, torch.from_numpy(s["xt"] + 1j * s["yt"]).to(C.dev))
