"""GMRES by captured steps where the captures change: more columns than one
capture is made for (256), more than two (512), and more than all of them
(1024, which go on without); unknowns just past the size (75000) from which a
thread owns a row of the Gram-Schmidt update; solves that alternate between sizes,
so that captures made for one are brought up to date for the other.  The FP64
residual of the density that comes back, formed from the operator and the right-hand side
by themselves, is the tolerance at most, up to 1e-11 for the operator's rounding
(its parity bound) and 1% for the estimate that stops the iteration; the plain
method's basis stays orthogonal to that (Gram-Schmidt is done twice)."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def packing(M, n, nout, seed):
    radii, cs, _ = G.lattice_pack(M, n, 0.7, G.CHANNEL_WALL, np.random.default_rng(seed))
    xx, yy = G.make_bodies(n, radii, cs)
    return G.Geometry(n, nout, xx, yy, G.CHANNEL_WALL, 0, radii, cs)


def residual(g, x):
    b = stokes.rhs(g)
    return np.linalg.norm(b - stokes.matvec(g, x)) / np.linalg.norm(b)


@pytest.mark.parametrize("M,more,upto", [(14, 256, 512), (30, 512, 1024)])
def test_columns_past_the_captures(lib, M, more, upto):
    g = packing(M, 64, 512, M)
    tol = 1e-10
    x, its, st = stokes.solve(g, tol=tol, maxl=3000)
    assert more < its <= upto
    assert residual(g, x) < 1.01 * tol + 1e-11


@pytest.mark.parametrize("maxl", [1024, 1025, 1040])
def test_columns_past_the_last_capture(lib, maxl):
    """Stopped unconverged around column 1024, from which the steps are launched
    one by one: the estimate of the residual is still that of the density, to the 1%."""
    g = packing(90, 64, 512, 90)
    x, its, st = stokes.solve(g, tol=1e-10, maxl=maxl, allow=(0, 1))
    assert its == maxl
    assert abs(residual(g, x) - st["est_residual"]) < 0.01 * st["est_residual"]


def test_row_per_thread_update(lib):
    g = packing(148, 256, 514, 3)   # 2 x 38402 + 444 = 77248 unknowns
    x, its, st = stokes.solve(g, tol=1e-8, precond=1, maxl=1000)
    assert residual(g, x) < 1.01e-8 + 1e-11


def test_alternating_sizes_reuse_captures(lib):
    a, b = packing(6, 64, 256, 1), packing(9, 66, 258, 2)
    xa, na, _ = stokes.solve(a, tol=1e-10)
    xb, nb, _ = stokes.solve(b, tol=1e-10)
    for g, x0, n0 in ((a, xa, na), (b, xb, nb), (a, xa, na)):
        x, its, _ = stokes.solve(g, tol=1e-10)
        assert its == n0 and np.array_equal(x, x0)
        assert residual(g, x) < 1.01e-10 + 1e-11
