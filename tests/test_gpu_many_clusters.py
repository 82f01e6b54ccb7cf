"""More than 4096 clusters (4100 bodies and a wall of eight arcs): the operator, the solve and
the shear stress then sum every pair directly over tile ranges.  The operator against the
CPU FP64 oracle at its parity bound of 1e-11, in the precisions of a solve at theirs (with the
near rules on a density without rigid part: on 16 nodes the trapezoid rule's field of a rigid
motion, which the operator leaves out, is 2e-10); the solve by the FP64 residual of its
density; the stress against the all-barycentric one at the 1e-10 asked of the hybrid
evaluation elsewhere."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu
N, NOUT, COLS, ROWS = 16, 256, 100, 41


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.fixture(scope="module")
def lattice():
    x, y = np.meshgrid(np.linspace(-2.8, 2.8, COLS), np.linspace(-0.88, 0.88, ROWS))
    c = np.stack([x.ravel(), y.ravel()], 1)
    r = np.random.default_rng(1).uniform(0.009, 0.012, len(c))
    xx, yy = G.make_bodies(N, r, c)
    return G.Geometry(N, NOUT, xx, yy, (3.0, 1.0, 8.0), 0, r, c)


@pytest.fixture(scope="module")
def density(lattice):
    """Modes that 16 nodes resolve, stokeslets and rotlets."""
    g = lattice
    rng = np.random.default_rng(2)
    th, tw = (2 * np.pi * np.arange(k) / k for k in (N, NOUT))
    body = lambda: (rng.standard_normal(g.M)[:, None] + rng.standard_normal(g.M)[:, None]
                    * np.cos(th + rng.uniform(0, 6.3, (g.M, 1))))
    wall = [np.cos(tw + p) + 0.3 * np.cos(5 * tw + p) for p in (0.1, 0.7)]
    return np.concatenate([*wall, np.stack([body(), body()], 1).ravel(), 0.1 * rng.standard_normal(3 * g.M)])


def without_rigid(g, den):
    den = den.copy()
    b = den[2 * g.nout:2 * g.nout + 2 * g.M * N].reshape(g.M, 2, N)   # circles: equal weights
    b -= b.mean(2, keepdims=True)
    t = np.stack([-(g.yy.reshape(g.M, N) - g.centers[:, 1:]), g.xx.reshape(g.M, N) - g.centers[:, :1]], 1)
    b -= ((b * t).sum((1, 2)) / (t * t).sum((1, 2)))[:, None, None] * t
    return den


@pytest.mark.parametrize("ibary", [0, 1])
def test_operator(lib, oracle, lattice, density, ibary):
    den = without_rigid(lattice, density) if ibary else density
    ref = oracle.matvec(lattice, den, mode=ibary)
    assert rel(stokes.matvec(lattice, den, ibary=ibary), ref) < 1e-11
    assert rel(stokes.matvec(lattice, den, ibary=ibary, precision=2), ref) < 1e-10
    assert rel(stokes.matvec(lattice, den, ibary=ibary, precision=1), ref) < 1e-5


def test_solve(lib, lattice):
    g = lattice
    x, its, st = stokes.solve(g, precision=1, precond=1, tol=1e-4, maxl=2000)
    b = stokes.rhs(g)
    assert np.linalg.norm(b - stokes.matvec(g, x)) / np.linalg.norm(b) < 1.01e-4


def test_stress(lib, lattice, density):
    tau, E = stokes.shear_stress(lattice, density)
    tau_b, E_b = stokes.shear_stress(lattice, density, stress_all_bary=1)
    assert rel(tau, tau_b) < 1e-10
    assert rel(E, E_b) < 1e-10


def test_near_wall_bodies(lib, lattice):
    """The list of near-wall bodies comes back in pieces of 256: all of it, by the rule."""
    g = lattice
    stokes.matvec(g, np.zeros(g.ntot))
    lw, bodies, _ = stokes.near_info(g.M)
    speed = stokes.geometry(g)["speed"].reshape(g.M, N)
    lim = g.wall[1] - (speed.mean(1) + 4 * lw * 2 * np.pi / NOUT)
    y = g.yy.reshape(g.M, N).mean(1)
    want = np.nonzero(np.abs(y) >= lim)[0]
    assert 256 < len(want) < g.M and not (np.abs(np.abs(y) - lim) < 1e-9).any()
    assert bodies == want.tolist()
