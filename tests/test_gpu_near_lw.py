"""The integer wall length scale of the near-wall rules (an implicitly typed INTEGER in the
reference: every partial sum truncated, then an integer division) for walls so large that
the running sum's own rounding decides at a node, against the same sum on the host over the
speeds the library reports."""
import numpy as np
import pytest

from erosion_b200 import geometry as G, stokes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e3, 1e6, 1e9, 1e11])
def test_integer_length_scale(lib, scale):
    for k in range(48):
        n = 512 + 64 * k
        wall = (3.0 * scale, (1.0 + 0.01 * k) * scale, 8.0)
        xx, yy = G.make_bodies(16, np.array([0.1 * scale]), np.zeros((1, 2)))
        g = G.Geometry(16, n, xx, yy, wall, 0, np.array([0.1 * scale]), np.zeros((1, 2)))
        speed = stokes.geometry(g)["speed0"]
        lw = 0
        for v in speed:
            lw = int(float(lw) + v)
        assert stokes.near_info(1)[0] == lw // n, (k, n)
