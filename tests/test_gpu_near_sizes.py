"""The barycentric kernels at the sizes where their splits can go wrong: curves
shorter and longer than a shared-memory tile of 256 sources and not divisible
by the 8 warps that share it, target counts that fill no CTA of 32, against
the CPU FP64 oracle.  Tolerances as for the other sizes: 1e-11 for the
operator, 1e-9 for the shear stress, 1e-10 for the target quantities."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("n,nout", [(8, 64), (34, 130), (66, 250), (256, 258), (258, 520), (300, 770)])
def test_near_sizes_match_oracle(lib, oracle, n, nout):
    g = G.custom(n, nout, [0.3, 0.25, 0.2], [[-1.0, 0.1], [-0.35, 0.0], [0.6, 0.72]])
    den = np.random.default_rng(n).standard_normal(g.ntot)
    if n > 8:   # the near rules leave pairs to the trapezoid rule, which drops the bodies' rigid
                # parts: on 8 nodes that rule itself is 2e-5 off zero for them
        assert rel(stokes.matvec(g, den), oracle.matvec(g, den, mode=1)) < 1e-11
    assert rel(stokes.matvec(g, den, ifmm=0), oracle.matvec(g, den, mode=2)) < 1e-11
    for kw in ({}, {"stress_all_bary": 1}):
        if not kw and n < 66:
            continue    # a white-noise density on few nodes: the trapezoid part differs by its aliasing
        tau, _ = stokes.shear_stress(g, den, **kw)
        assert rel(tau, oracle.shear_stress(g, den)[0]) < 1e-9
    xt, yt = np.linspace(-2.0, 2.0, 37), np.linspace(-0.7, 0.55, 37)
    for a, b in zip(stokes.qoi_targets(g, den, xt, yt), oracle.qoi_targets(g, den, xt, yt)):
        assert rel(a, b) < 1e-10
