"""The cut of the expansions by which separated clusters act, one source node at a time: the
field of a single node with a unit density, at bodies 2.7 to 220 radii away (every class of
order, close to its edge: distances 6 to 10% apart) and at the wall, against the pair term in 80
bits.  The bound is the one the kernels state, 5e-16 of the node's field (3^-32), and the
rounding of one expansion: 32 terms, so 32 eps for the velocity; 64 eps for the strain, the
derivative of the same series.  (A field or a strain is measured by |w sigma|/r or |w sigma|/r^2, summed
over the sources.)"""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu

N, A, L = 64, 0.004, np.longdouble
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def spiral():
    c = [np.zeros(2)]
    rng = np.random.default_rng(4)
    d = 2.65 * A
    while d < 0.93:
        phi = rng.uniform(0, 2 * np.pi, 400)   # the most open direction
        p = d * np.stack([np.cos(phi), np.sin(phi)], 1)
        gap = np.min(np.linalg.norm(p[:, None] - np.array(c)[None], axis=2), axis=1)
        assert gap.max() > 2.4 * A
        c.append(p[np.argmax(gap)])
        d *= 1.1 if d < 6 * A else 1.06
    c = np.array(c)
    r = np.full(len(c), A)
    xx, yy = G.make_bodies(N, r, c)
    g = G.Geometry(N, 512, xx, yy, (3.0, 1.0, 8.0), 0, r, c)
    assert g.M * N + 512 >= 3200   # the size from which clusters act through expansions
    return g


def nodes(g):
    q = stokes.geometry(g)
    x = np.concatenate([q["xo"], g.xx]).astype(L), np.concatenate([q["yo"], g.yy]).astype(L)
    w = q["speed"][:N].astype(L) * 2 / N
    return np.stack(x, 1), np.stack([q["px"][:N], q["py"][:N]], 1).astype(L), w, q["speed"][:N].astype(L)


def unit_density(g, j, comp):
    den = np.zeros(g.ntot)
    den[2 * g.nout + comp * N + j] = 1.0   # node j of the first body
    return den


def test_velocity(lib, spiral):
    g = spiral
    x, n, w, _ = nodes(g)
    xs = x[g.nout:g.nout + N]
    tgt = np.r_[0:g.nout, g.nout + N:g.nout + g.M * N]
    for j in range(0, N, 5):
        for comp in (0, 1):
            u = stokes.matvec(g, unit_density(g, j, comp), ibary=0)
            body = u[2 * g.nout:2 * g.nout + 2 * N * g.M].reshape(g.M, 2, N)
            got = np.stack([np.concatenate([u[k * g.nout:(k + 1) * g.nout], body[:, k].ravel()]) for k in (0, 1)], 1)
            r = x[tgt] - xs[j]
            r2 = (r ** 2).sum(1)
            # the wall's rank-one term is zero (its density is), so is every jump but the source's own
            ref = ((r @ n[j]) * r[:, comp] * w[j] / r2 ** 2)[:, None] * r
            err = np.sqrt(((got[tgt] - ref) ** 2).sum(1)) / (w[j] / np.sqrt(r2))
            assert err.max() < 3.0 ** -32 + 32 * EPS, (j, comp, float(err.max()))


def test_stokeslet_and_rotlet(lib, spiral):
    """A body's stokeslet and rotlet ride on the same expansions, at the disc's centre: to
    the rounding of 32 terms of (|log r| + 1) / (4 pi) and of 1 / r."""
    g = spiral
    x = nodes(g)[0]
    c = np.array([stokes.geometry(g)[k][0] for k in ("cx", "cy")], L)
    tgt = np.r_[0:g.nout, g.nout + N:g.nout + g.M * N]
    r = x[tgt] - c
    r2 = (r ** 2).sum(1)
    for k in range(3):
        den = np.zeros(g.ntot)
        den[2 * g.nout + 2 * N * g.M + k] = 1.0   # of the first body
        u = stokes.matvec(g, den, ibary=0)
        body = u[2 * g.nout:2 * g.nout + 2 * N * g.M].reshape(g.M, 2, N)
        got = np.stack([np.concatenate([u[q * g.nout:(q + 1) * g.nout], body[:, q].ravel()]) for q in (0, 1)], 1)
        if k < 2:
            ref = r[:, k, None] * r / r2[:, None]
            ref[:, k] -= np.log(r2) / 2
            ref, mag = ref / (4 * L(np.pi)), (np.abs(np.log(r2)) / 2 + 1) / (4 * L(np.pi))
        else:
            ref, mag = np.stack([r[:, 1], -r[:, 0]], 1) / r2[:, None], 1 / np.sqrt(r2)
        err = np.sqrt(((got[tgt] - ref) ** 2).sum(1)) / mag
        assert err.max() < 3.0 ** -32 + 32 * EPS, (k, float(err.max()))


def test_strain(lib, spiral):
    g = spiral
    x, n, w, sp = nodes(g)
    xs = x[g.nout:g.nout + N]
    # bodies that no barycentric rule connects with the source: 12 of its spacings from its disc
    far = np.linalg.norm(g.centers, axis=1) > 2 * A + 12 * 2 * np.pi * A / N + 1e-6
    assert far.sum() > 60
    tgt = (N * np.nonzero(far)[0][:, None] + np.arange(N)).ravel()
    r = x[g.nout + tgt][:, None] - xs[None]
    r2 = (r ** 2).sum(2)
    rn = (r * n).sum(2)
    xb = (sp[:, None] * xs).sum(0) / sp.sum()
    rot = np.stack([-(xs[:, 1] - xb[1]), xs[:, 0] - xb[0]], 1)
    for j in range(0, N, 5):
        for comp in (0, 1):
            _, E = stokes.shear_stress(g, unit_density(g, j, comp))
            s = np.zeros((N, 2), L)
            s[j, comp] = 1
            # the sums take a body's density without its rigid part, which has no field outside
            t = (sp[:, None] * s).sum(0) / sp.sum()
            s = s - t - ((sp[:, None] * rot * s).sum() / (sp[:, None] * rot ** 2).sum()) * rot
            v = w[:, None] * s
            rv = (r * v).sum(2)
            h = (rn[:, :, None] * v + rv[:, :, None] * n) / 2   # S r, S the symmetric part of n v
            q = rn * rv
            e11 = ((h[..., 0] * r[..., 0] - h[..., 1] * r[..., 1]) / r2 ** 2
                   - 2 * q * (r[..., 0] ** 2 - r[..., 1] ** 2) / r2 ** 3).sum(1)
            e12 = ((h[..., 0] * r[..., 1] + h[..., 1] * r[..., 0]) / r2 ** 2
                   - 4 * q * r[..., 0] * r[..., 1] / r2 ** 3).sum(1)
            mag = (np.sqrt((v ** 2).sum(1)) / r2).sum(1)
            err = np.sqrt((E[0][tgt] - e11) ** 2 + (E[1][tgt] - e12) ** 2) / mag
            assert err.max() < 3.0 ** -32 + 64 * EPS, (j, comp, float(err.max()))
