"""Barycentric sums over every curve where a warp takes a short curve by itself: curves of 8 to
32 nodes and one just past them, body counts that fill no stage of eight, one body, targets
that fill no warp, a target on the branch of coincident nodes.  Against the CPU FP64 oracle
at the bounds the other sizes have (1e-10 of the largest value for targets, 1e-9 for the
stress); the coincident target, whose distance of 5e-11 has five digits in 64 bits but the
same ones on both sides, to 1e-6."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("M,n,nout", [(1, 8, 16), (7, 8, 34), (33, 8, 64), (9, 14, 300), (40, 16, 130), (65, 20, 64),
                                      (11, 24, 258), (8, 32, 64), (17, 32, 514), (17, 34, 514)])
def test_short_curves(lib, oracle, M, n, nout):
    rng = np.random.default_rng(M + n)
    radii, cs, _ = G.lattice_pack(M, 64, 0.8, G.CHANNEL_WALL, rng)
    xx, yy = G.make_bodies(n, radii, cs)
    g = G.Geometry(n, nout, xx, yy, G.CHANNEL_WALL, 0, radii, cs)
    den = rng.standard_normal(g.ntot)
    xt, yt = rng.uniform(-0.8, 0.8, 1000), rng.uniform(-0.4, 0.4, 1000)
    # no closer to a node than a node spacing, where the values are not those of a field
    far = np.min(np.hypot(xt[:, None] - xx, yt[:, None] - yy), 1) > 2 * np.pi * radii.max() / n
    xt, yt = xt[far], yt[far]
    for k in (len(xt), 33, 1):
        for a, b in zip(stokes.qoi_targets(g, den, xt[:k], yt[:k]), oracle.qoi_targets(g, den, xt[:k], yt[:k])):
            assert rel(a, b) < 1e-10
    tau = stokes.shear_stress(g, den, stress_all_bary=1)[0]
    assert rel(tau, oracle.shear_stress(g, den)[0]) < 1e-9


@pytest.mark.parametrize("M,n", [(9, 16), (3, 34)])
def test_coincident_node(lib, oracle, M, n):
    rng = np.random.default_rng(M)
    radii, cs, _ = G.lattice_pack(M, 64, 0.8, G.CHANNEL_WALL, rng)
    xx, yy = G.make_bodies(n, radii, cs)
    g = G.Geometry(n, 128, xx, yy, G.CHANNEL_WALL, 0, radii, cs)
    den = rng.standard_normal(g.ntot)
    k = n * (M - 1) + 3
    u = np.array([xx[k], yy[k]]) - cs[-1]
    p = np.array([[xx[k], yy[k]] + 5e-11 * u / np.linalg.norm(u), [0.0, 0.31]])
    a, b = (f(g, den, *p.T) for f in (stokes.qoi_targets, oracle.qoi_targets))
    for q in (0, 1, 3):
        assert rel(a[q], b[q]) < 1e-6
