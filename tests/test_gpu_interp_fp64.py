"""The FP64 interpolation at the edges of its work split, against the oracle:
orders 4, 6, 8, meshes without TMA boxes (odd K), boxes that wrap or are wider
than the mesh, tiles that do not divide K, more particles in a tile than one
round of a block takes (a cluster), several right-hand sides.

Tolerance 1e-12 relative L2, the repository's FP64 bound."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,p,tile,R,n", [
    (32, 6, None, 1, 600),
    (32, 4, (16, 8, 4), 3, 600),
    (36, 8, (16, 8, 4), 2, 600),     # 23-wide rows, last tiles short
    (30, 6, (7, 5, 4), 1, 600),      # odd tile starts: plain loads
    (27, 6, None, 2, 600),           # odd K: no TMA
    (45, 8, (12, 12, 8), 1, 600),
    (9, 8, None, 1, 200),            # box wider than the mesh
    (8, 4, (4, 4, 4), 1, 3),
    (48, 6, None, 5, 2500),
])
def test_interpolation(gpu_lib, K, p, tile, R, n):
    L, xi = 40.0, 0.4
    rng = np.random.default_rng(K * p + R)
    pos = rng.uniform(0, L, (n, 3))
    pos[: n // 4] = 0.06 * pos[: n // 4] + 7.0  # a cluster within a tile or two
    f = rng.standard_normal((R, 3 * n))
    eng = spme_gb300.Engine(n, L, xi, K, p, precision="fp64", max_nrhs=R, tile=tile,
                            terms=spme_gb300.TERM_RECIP)
    eng.set_positions(pos)
    u = eng.apply(f)
    eng.close()
    assert relerr(u, oracle.recip(pos, L, xi, K, p, f)) < 1e-12
