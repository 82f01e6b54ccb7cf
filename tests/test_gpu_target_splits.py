"""Velocity, pressure and vorticity at targets where their launches split the work
differently: one target (a part per curve), one CTA of targets and one lane more,
counts with more and with fewer than a wave of CTAs, a wall longer than every
part and shorter than one body, a single body, fewer body nodes than parts.
Targets evaluated in pieces have other parts than all at once: the sums, of some
1e4 FP64 terms, agree to 1e4 eps ~ 1e-12 of their magnitudes (1e-11 asked, as of
the operator); which targets are inside a body is the same exactly."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ibary", [1, 0])
@pytest.mark.parametrize("M,n,nout", [(1, 16, 64), (1, 256, 128), (24, 64, 2048), (50, 128, 514)])
def test_targets_in_pieces(lib, M, n, nout, ibary):
    rng = np.random.default_rng(M + n)
    radii, cs, _ = G.lattice_pack(M, max(n, 64), 0.7, G.CHANNEL_WALL, rng)
    xx, yy = G.make_bodies(n, radii, cs)
    g = G.Geometry(n, nout, xx, yy, G.CHANNEL_WALL, 0, radii, cs)
    den = rng.standard_normal(g.ntot)
    xt, yt = rng.uniform(-0.8, 0.8, 2400), rng.uniform(-0.4, 0.4, 2400)
    xt[5], yt[5] = cs[0]   # inside a body
    whole = stokes.qoi_targets(g, den, xt, yt, ibary=ibary)
    assert all(f[5] == 0.0 for f in whole)
    for lo, hi in ((0, 1), (4, 6), (1, 33), (1, 34), (100, 1400)):
        part = stokes.qoi_targets(g, den, xt[lo:hi], yt[lo:hi], ibary=ibary)
        for a, b in zip(part, whole):
            assert np.array_equal(a == 0.0, b[lo:hi] == 0.0)
            assert np.abs(a - b[lo:hi]).max() <= 1e-11 * np.abs(b).max()
