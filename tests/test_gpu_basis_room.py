"""The basis of GMRES grows when a step needs it, not for a step that is launched ahead of the
host: a solve that ends on the last column there is room for runs on a device that could
not hold the next growth."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


def test_a_solve_that_ends_on_the_last_column(lib):
    import torch
    radii, cs, _ = G.lattice_pack(200, 64, 0.7, G.CHANNEL_WALL, np.random.default_rng(1))
    xx, yy = G.make_bodies(512, radii, cs)
    g = G.Geometry(512, 2048, xx, yy, G.CHANNEL_WALL, 0, radii, cs)
    column = 8 * g.ntot   # 1.7 MB; the first basis has 64
    run = lambda **kw: stokes.solve(g, allow=(0, 1), **kw)
    r = [run(tol=1e-14, maxl=k)[2]["est_residual"] for k in (62, 63)]
    tol = np.sqrt(r[0] * r[1])   # met by step 63, which fills the 64 columns
    lib.erosion_release()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    run(tol=1e-14, maxl=40)
    used = before - torch.cuda.mem_get_info()[0]
    lib.erosion_release()
    # room for the solve and 60 columns: the next growth takes 128
    hold = torch.empty(torch.cuda.mem_get_info()[0] - used - 60 * column, dtype=torch.uint8, device="cuda")
    try:
        x, its, st = run(tol=tol)
    finally:
        del hold
        torch.cuda.empty_cache()
        lib.erosion_release()
    assert its == 63 and st["est_residual"] <= tol
