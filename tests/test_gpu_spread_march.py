"""The z-marching spread at the edges of its work split, against the tile kernel
(spread mode 0) and the oracle: the smallest mesh of each order, meshes that are
no multiple of its 8 x 2 / 8 x 4 columns or of its 8-plane groups, odd meshes, z
segments, one to four component chunks' widths, clusters (more visits than are
looked up together), a nearly empty mesh.

Tolerances relative L2 as for the other FP32 spread kernels: 2e-6 between the
kernels, 1e-5 against the oracle."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,p,R,n,cluster", [
    (19, 4, 3, 500, 0.06),
    (21, 6, 4, 500, 0.06),
    (23, 8, 5, 500, 0.06),     # 15 components: rows of no whole 16-byte pieces
    (24, 6, 4, 5000, 0.02),    # thousands of particles in a few cells
    (30, 6, 3, 3, 1.0),
    (45, 6, 4, 2000, 0.3),
    (50, 8, 5, 2000, 0.3),
    (101, 6, 6, 2000, 0.1),    # two components per lane
    (100, 4, 10, 2000, 0.1),
    (104, 8, 11, 2000, 0.1),   # three
    (100, 6, 17, 2000, 0.1),   # two chunks of 48 components
])
def test_march_spread(gpu_lib, K, p, R, n, cluster):
    L, xi = 40.0, 0.4
    rng = np.random.default_rng(K * p + R)
    pos = rng.uniform(0, L, (n, 3))
    pos[: n // 2] = cluster * pos[: n // 2] + 7.0
    f = rng.standard_normal((R, 3 * n)).astype(np.float32)
    out = {}
    for mode in (0, 1):
        eng = spme_gb300.Engine(n, L, xi, K, p, precision="fp32", max_nrhs=R,
                                terms=spme_gb300.TERM_RECIP)
        eng.set_spread_mode(mode)
        eng.set_positions(pos)
        out[mode] = eng.apply(f)
        eng.close()
    assert relerr(out[1], out[0]) < 2e-6
    assert relerr(out[1], oracle.recip(pos, L, xi, K, p, f.astype(np.float64))) < 1e-5
