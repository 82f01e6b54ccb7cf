"""What one erosion_solve_batch call leaves for the next and for its caller: nothing of an
earlier ensemble's geometry reaches a later one, its buffers stay within a share of the
device's memory and give way where a later one needs their room; a call that fails
leaves the caller's densities as they were."""
import ctypes

import numpy as np
import pytest

from erosion_b200 import _lib, geometry as G, stokes

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


def test_failed_call_leaves_the_densities(lib):
    """A geometry that fails in its solve (a guess that is not finite) fails the call; the
    others' densities stay the caller's guesses, as its own does."""
    ens = ensemble(50)
    den = np.concatenate([np.full(ens[0].ntot, 1e-3), np.full(ens[1].ntot, np.nan)])
    kept = den.copy()
    nits = np.full(2, -1, np.int64)
    size = [np.array(v, np.int64) for v in ([g.n for g in ens], [g.M for g in ens], [g.nout for g in ens])]
    xx, yy = (np.concatenate([getattr(g, k) for g in ens]) for k in ("xx", "yy"))
    p = stokes.params_for(ens[0], tol=1e-8)
    rc = lib.erosion_solve_batch(ctypes.byref(p), 2, *[v.ctypes.data_as(_lib.PI64) for v in size], _lib.ptr(xx),
                                 _lib.ptr(yy), _lib.ptr(den), nits.ctypes.data_as(_lib.PI64))
    assert rc == _lib.EROSION_BREAKDOWN
    assert np.array_equal(den, kept, equal_nan=True)
    assert nits.tolist() == [-1, -1]


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()


def test_what_is_kept_is_bounded(lib):
    """Sixteen geometries whose bases take a gigabyte each: the call may keep a sixteenth of
    the device's memory, and a gigabyte for streams, graphs and the driver."""
    lib.erosion_release()
    before, total = free_bytes()
    ens = [G.ensemble(1, seed=3 + k, bodies=(100, 100), npts=(512,), porosity=(0.7, 0.7), nout=2048)[0]
           for k in range(16)]
    stokes.solve_batch(ens, tol=1e-14, maxl=1100, allow=(_lib.EROSION_OK, _lib.EROSION_MAXITER))
    assert before - free_bytes()[0] < total / 16 + 2 ** 30
    lib.erosion_release()


def test_room_for_another_ensemble(lib):
    """Two ensembles with their large geometry in different places, on a device with room for
    one such geometry and not for two: what the first left does not fail the second."""
    import torch
    large = G.ensemble(1, seed=1, bodies=(60, 60), npts=(256,), porosity=(0.7, 0.7), nout=2048)[0]
    small = ensemble(20)[0]
    kw = dict(tol=1e-14, maxl=1500, allow=(_lib.EROSION_OK, _lib.EROSION_MAXITER))
    lib.erosion_release()
    torch.cuda.empty_cache()
    want = [stokes.solve_batch(e, **kw)[0] for e in ([large, small], [small, large])]
    lib.erosion_release()
    # its basis takes 420 MB, and 267 MB more while it grows for the last time
    hold = torch.empty(free_bytes()[0] - 1000 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        got = [stokes.solve_batch(e, **kw)[0] for e in ([large, small], [small, large])]
    finally:
        del hold
        torch.cuda.empty_cache()
        lib.erosion_release()
    for w, g in zip(want, got):
        for a, b in zip(w, g):
            assert np.array_equal(a, b)
