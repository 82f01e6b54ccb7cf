"""What one erosion_solve_batch call leaves for the next: nothing of an earlier ensemble's
geometry reaches a later one."""
import numpy as np
import pytest

from erosion_b200 import geometry as G, stokes

pytestmark = pytest.mark.gpu


def ensemble(seed):
    return [G.ensemble(1, seed=seed + k, bodies=(m, m), npts=(n,), porosity=(0.7, 0.7), nout=256)[0]
            for k, (m, n) in enumerate([(5, 64), (3, 128)])]


def test_inverses_are_not_kept_between_calls(lib):
    """precond_refresh lets the set-ups of one erosion run share block inverses; the
    geometries of two ensembles of equal sizes have nothing to do with each other.  The second
    ensemble's solve is bit for bit the one of a library without history."""
    kw = dict(tol=1e-10, precond=1, precond_refresh=4)
    stokes.solve_batch(ensemble(70), **kw)
    after, n_after, _ = stokes.solve_batch(ensemble(90), **kw)
    lib.erosion_release()
    fresh, n_fresh, _ = stokes.solve_batch(ensemble(90), **kw)
    assert n_after.tolist() == n_fresh.tolist()
    for a, f in zip(after, fresh):
        assert np.array_equal(a, f)
