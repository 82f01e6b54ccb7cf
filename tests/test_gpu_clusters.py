"""The far field by clusters against the direct sum over tile ranges (a forced
launch shape) and against the CPU FP64 oracle, at the sizes where clusters go
wrong: just below and above the size from which separated clusters act through
expansions, bodies of several clusters (the last of 2 nodes), odd tails of the
wall's clusters, many clusters per staged batch, all near rules.  Both sums
take ~1e4 terms per node in FP64, so they agree to 1e4 eps ~ 1e-12 of the sum
of their magnitudes; the operator's parity bound of 1e-11 is asked of both."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def packing(M, n, nout, seed=2):
    rng = np.random.default_rng(seed)
    radii, cs, _ = G.lattice_pack(M, n, 0.7, G.CHANNEL_WALL, rng)
    xx, yy = G.make_bodies(n, radii, cs)
    return G.Geometry(n, nout, xx, yy, G.CHANNEL_WALL, 0, radii, cs)


@pytest.mark.parametrize("M,n,nout", [(1, 64, 64), (17, 128, 1020), (17, 128, 1026), (12, 258, 514), (12, 320, 1024),
                                      (90, 34, 770), (30, 256, 2050), (3, 512, 2500)])
@pytest.mark.parametrize("kw,mode", [({}, 1), ({"ibary": 0}, 0), ({"ifmm": 0}, 2)])
def test_clusters_match_direct_sum(lib, oracle, M, n, nout, kw, mode):
    g = packing(M, n, nout)
    den = np.random.default_rng(M).standard_normal(g.ntot)
    a = {p: stokes.matvec(g, den, precision=p, **kw) for p in (0, 1, 2)}
    assert lib.erosion_set_far_shape(0, 0) == 0
    try:
        b = stokes.matvec(g, den, **kw)
        b32 = stokes.matvec(g, den, precision=1, **kw)
    finally:
        assert lib.erosion_set_far_shape(0, -1) == 0
    assert rel(a[0], b) < 1e-11
    assert rel(a[2], b) < 1e-11
    # FP32 pair terms: no further from the FP64 operator than the direct FP32 sum, or 1e-6
    assert rel(a[1], b) < max(1e-6, 1.5 * rel(b32, b))
    if mode != 2:   # (the all-barycentric oracle takes minutes at these sizes)
        # no further from the oracle than the direct sum: the curvature of a 2500-node wall and a
        # rigid part before a wall of 64 nodes put it 3e-11 and 3e-10 off, whatever the far field
        ref = oracle.matvec(g, den, mode=mode)
        assert rel(a[0], ref) < max(1e-11, 1.5 * rel(b, ref))


@pytest.mark.parametrize("M,n,nout", [(1, 64, 130), (17, 128, 1020), (17, 128, 1026), (12, 258, 514), (40, 66, 770),
                                      (30, 256, 2050)])
def test_stress_by_clusters_matches_all_barycentric(lib, M, n, nout):
    """On a density that the nodes resolve (modes up to n/10, decaying) the
    stress by clusters and the all-barycentric one agree to the 1e-10 asked of
    the hybrid evaluation elsewhere."""
    g = packing(M, n, nout)
    rng = np.random.default_rng(n)
    th, tw = (2 * np.pi * np.arange(k) / k for k in (n, nout))
    k = np.arange(1, n // 10 + 1)
    f = lambda t: (rng.standard_normal(len(k)) / k ** 2) @ np.cos(np.outer(k, t) + rng.uniform(0, 6.3, (len(k), 1)))
    den = np.concatenate([f(tw), f(tw)] + [f(th) for _ in range(2 * M)] + [rng.standard_normal(3 * M)])
    tau, E = stokes.shear_stress(g, den)
    tau_b, E_b = stokes.shear_stress(g, den, stress_all_bary=1)
    assert rel(tau, tau_b) < 1e-10
    assert rel(E, E_b) < 1e-10


@pytest.mark.parametrize("M,n,nout", [(2, 16, 16), (17, 128, 1020), (17, 128, 1026), (12, 258, 514), (128, 34, 770)])
def test_noalloc_by_clusters(lib, M, n, nout):
    """erosion_matvec_noalloc keeps its clusters, lists and expansions in its
    fixed memory; both operators sum the same terms in another order."""
    import ctypes
    import torch
    g = packing(M, n, nout)
    den = np.random.default_rng(M).standard_normal(g.ntot)
    x, y, d = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (g.xx, g.yy, den))
    v = torch.empty_like(d)
    p = stokes.params_for(g, ibary=0)
    st = torch.cuda.current_stream()
    assert lib.erosion_matvec_noalloc(ctypes.byref(p), g.n, g.M, g.nout, x.data_ptr(), y.data_ptr(), d.data_ptr(),
                                      v.data_ptr(), st.cuda_stream) == 0
    assert rel(v.cpu().numpy(), stokes.matvec(g, den, ibary=0)) < 1e-11
