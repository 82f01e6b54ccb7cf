"""The shift of the expansions as it is compiled for two and for three CTAs per SM: cluster
counts to both sides of two an SM (296 here), the wall's last cluster of two nodes, and
the operator without allocation, whose sizes end at 350 clusters.  Against the direct sum of
a forced launch shape, to the operator's parity bound of 1e-11, as at the other sizes."""
import ctypes

import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def packing(M, n, nout):
    radii, cs, _ = G.lattice_pack(M, 64, 0.7, G.CHANNEL_WALL, np.random.default_rng(M))
    xx, yy = G.make_bodies(n, radii, cs)
    return G.Geometry(n, nout, xx, yy, G.CHANNEL_WALL, 0, radii, cs)


@pytest.mark.parametrize("M,n,nout", [(200, 34, 96 * 32), (200, 34, 96 * 32 + 2), (110, 66, 4098), (430, 16, 514),
                                      (600, 16, 130)])
def test_operator(lib, M, n, nout):
    g = packing(M, n, nout)
    den = np.random.default_rng(M).standard_normal(g.ntot)
    a = stokes.matvec(g, den)
    assert lib.erosion_set_far_shape(0, 0) == 0
    try:
        b = stokes.matvec(g, den)
    finally:
        assert lib.erosion_set_far_shape(0, -1) == 0
    assert rel(a, b) < 1e-11


def test_noalloc(lib):
    import torch
    g = packing(111, 258, 4094)   # 128 + 2 x 111 clusters
    den = np.random.default_rng(3).standard_normal(g.ntot)
    x, y, d = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (g.xx, g.yy, den))
    v = torch.empty_like(d)
    p = stokes.params_for(g, ibary=0)
    assert lib.erosion_matvec_noalloc(ctypes.byref(p), g.n, g.M, g.nout, x.data_ptr(), y.data_ptr(), d.data_ptr(),
                                      v.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert rel(v.cpu().numpy(), stokes.matvec(g, den, ibary=0)) < 1e-11
