"""The wall's part of the shear stress (clusters of CTAs that share its nodes, over
a packed list of the body nodes near to it) where it can go wrong: no node near,
a few lanes of one group, more groups than clusters at a time, shares of a few
nodes, shares of several staged tiles, totals that 8 does not divide.  Against
the all-barycentric stress, with the 1e-10 asked of the hybrid evaluation
elsewhere, on densities that the nodes resolve (modes up to n/10, decaying)."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def smooth(n, rng):
    th = 2 * np.pi * np.arange(n) / n
    k = np.arange(1, max(2, n // 10))
    c = rng.standard_normal((2, len(k))) * 0.5 ** k
    return c[0] @ np.cos(np.outer(k, th)) + c[1] @ np.sin(np.outer(k, th))


@pytest.mark.parametrize("radius,gap,count,n,nout", [
    (0.05, 0.3, 1, 64, 512),      # far from the wall: an empty list
    (0.1, 0.02, 1, 64, 130),      # a few nodes; shares of 16 and 17 wall nodes
    (0.1, 0.02, 3, 66, 514),
    (0.1, 0.01, 8, 130, 4098),    # shares of more than two staged tiles
    (0.03, 0.01, 24, 128, 512),   # more than 37 groups of 32
])
def test_wall_part_of_the_stress(lib, radius, gap, count, n, nout):
    wall = G.CHANNEL_WALL
    x = (np.arange(count) - (count - 1) / 2) * 1.6 * radius
    y = np.where(np.arange(count) % 2 == 0, 1, -1) * (wall[1] - radius - gap)
    cs = np.stack([x, y], 1)
    radii = np.full(count, radius)
    xx, yy = G.make_bodies(n, radii, cs)
    g = G.Geometry(n, nout, xx, yy, wall, 0, radii, cs)
    rng = np.random.default_rng(n)
    den = np.concatenate([smooth(nout, rng), smooth(nout, rng)]
                         + [smooth(n, rng) for _ in range(2 * count)] + [rng.standard_normal(3 * count)])
    tau, E = stokes.shear_stress(g, den)
    tau_b, E_b = stokes.shear_stress(g, den, stress_all_bary=1)
    assert rel(tau, tau_b) < 1e-10
    assert rel(E, E_b) < 1e-10
    again, _ = stokes.shear_stress(g, den)
    assert np.array_equal(tau, again)   # whatever the order of the list
