"""The preconditioner's block inversion at the sizes where its kernels change:
blocks of 2 n + 3 rows of one panel and of a partial last one, of one and of two
rows per thread (1024 threads' worth starts at 513), panels of 16 past the
shared memory of 32, and the form past those.  The preconditioned solve reaches
the unpreconditioned one's density (both to 1e-12: 1e-9 of it) in fewer
iterations, which a wrong inverse would not."""
import numpy as np
import pytest

from erosion_b200 import geometry as G
from erosion_b200 import stokes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 46, 62, 64, 190, 254, 256, 398, 400, 512, 740, 780])
def test_block_inverse_sizes(lib, n):
    g = G.custom(n, 256, [0.3, 0.22], [[-0.6, 0.05], [0.5, -0.1]])
    a, na, _ = stokes.solve(g, tol=1e-12)
    b, nb, st = stokes.solve(g, tol=1e-12, precond=1)
    assert st["precond_active"] == 1 and st["precond_singular_blocks"] == 0
    assert np.linalg.norm(a - b) / np.linalg.norm(a) < 1e-9
    assert nb < na
