"""The near-field set-up on the device against the rules stated in plain
Python (stokesSolver.f:694-926): wall length scale, near-wall bodies and the
number of barycentric pairs, at sizes with odd tails of 32-node items and masks
of several words, with bodies exactly on the edge of a rule, and the refusal of
nodes that are not finite or not inside the wall."""
import numpy as np
import pytest

from erosion_b200 import _lib, geometry as G, stokes

pytestmark = pytest.mark.gpu


def rules(g):
    """Pairs counted with the reference's loops (separately rounded doubles)."""
    geo = stokes.geometry(g)
    n, M, bw = g.n, g.M, g.wall[1]
    cx, cy = geo["cx"], geo["cy"]
    rb = geo["speed"].reshape(M, n)
    rb = np.array([np.sum(r) / n for r in rb])
    lw = 0
    for v in geo["speed0"]:
        lw = int(lw + v)
    lw //= g.nout
    x, y = g.xx.reshape(M, n), g.yy.reshape(M, n)
    wall, pairs = [], 0
    for b in range(M):
        lim = bw - (rb[b] + 4.0 * lw * (2 * np.pi) / g.nout)
        if abs(cy[b]) >= lim:
            wall.append(b)
            pairs += int((np.abs(y[b]) >= lim).sum())
            r = bw - abs(cy[b]) + 2.0 * rb[b]
            dx, dy = cx[b] - geo["xo"], cy[b] - geo["yo"]
            pairs += int((dx * dx + dy * dy <= r * r).sum())
        for t in range(M):
            rs = rb[b] + rb[t] + 4.0 * (rb[b] + rb[t]) * (2 * np.pi) / n
            dx, dy = cx[b] - cx[t], cy[b] - cy[t]
            if t != b and dx * dx + dy * dy <= rs * rs:
                ex, ey = cx[b] - x[t], cy[b] - y[t]
                pairs += int((ex * ex + ey * ey <= rs * rs).sum())
    return lw, wall, pairs


@pytest.mark.parametrize("M,n,nout,wall", [(1, 34, 66, G.REFERENCE_WALL), (3, 64, 256, G.REFERENCE_WALL),
                                           (31, 50, 258, G.CHANNEL_WALL), (33, 96, 514, G.CHANNEL_WALL),
                                           (70, 130, 1000, G.CHANNEL_WALL)])
def test_near_bookkeeping(lib, M, n, nout, wall):
    rng = np.random.default_rng(M)
    radii, cs, _ = G.lattice_pack(M, n, 0.6 if M > 3 else 0.8, wall, rng)
    xx, yy = G.make_bodies(n, radii, cs)
    g = G.Geometry(n, nout, xx, yy, wall, 0, radii, cs)
    want = rules(g)
    stokes.matvec(g, np.zeros(g.ntot))
    assert stokes.near_info(M) == want
    stokes.matvec(g, np.zeros(g.ntot), ifmm=0)
    assert stokes.near_info(M)[2] == M * n + M * (g.N - n)
    stokes.matvec(g, np.zeros(g.ntot), ibary=0)
    assert stokes.near_info(M)[2] == 0


@pytest.mark.parametrize("bad", [np.nan, np.inf, 0.5, 0.7])
def test_bad_nodes_refused(lib, bad):
    g = G.workload("c1")
    stokes.matvec(g, np.zeros(g.ntot))
    h = G.Geometry(g.n, g.nout, g.xx.copy(), g.yy.copy(), g.wall, g.ibc, g.radii, g.centers)
    h.xx[-1], h.yy[-1] = 0.0, bad     # (0, 0.5) is on the wall
    for call in (lambda: stokes.matvec(h, np.zeros(h.ntot)), lambda: stokes.shear_stress(h, np.zeros(h.ntot))):
        with pytest.raises(_lib.ErosionError) as e:
            call()
        assert e.value.code == _lib.EROSION_BAD_INPUT
    stokes.matvec(g, np.zeros(g.ntot))   # still usable
