"""The box spread at the edges of its work split, against the tile kernel
(spread mode 0) and the oracle: tile edges of p - 1 and below (up to four boxes
per coordinate), tiles that do not divide K, boxes wider than the mesh, empty
tiles, clustered particles, two and three right-hand sides.

Tolerances relative L2: FP64 1e-13 between the kernels (both round each product
and sum once, in another order) and 1e-12 against the oracle; FP32 2e-6 and 1e-5,
as the other spread kernels' tests have."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,K,p,tile,R,n", [
    ("fp64", 32, 6, None, 1, 800),
    ("fp64", 32, 4, None, 2, 800),
    ("fp64", 40, 8, None, 3, 800),
    ("fp64", 32, 6, (4, 4, 4), 1, 800),
    ("fp64", 33, 8, (4, 4, 4), 1, 800),
    ("fp64", 36, 8, (16, 8, 4), 2, 800),
    ("fp64", 30, 6, (7, 5, 4), 1, 800),
    ("fp64", 25, 8, (12, 12, 8), 1, 800),
    ("fp64", 9, 8, None, 1, 300),
    ("fp64", 48, 6, None, 1, 2),
    ("fp32", 96, 6, None, 1, 3000),
    ("fp32", 100, 6, (16, 8, 4), 1, 3000),
    ("fp32", 97, 4, (8, 4, 4), 2, 3000),
])
def test_box_spread(gpu_lib, prec, K, p, tile, R, n):
    L, xi = 40.0, 0.4
    dt, tol_k, tol_o = (np.float64, 1e-13, 1e-12) if prec == "fp64" else (np.float32, 2e-6, 1e-5)
    rng = np.random.default_rng(K * p + R)
    pos = rng.uniform(0, L, (n, 3))
    pos[: n // 4] = 0.06 * pos[: n // 4] + 7.0  # a cluster within a tile or two
    f = rng.standard_normal((R, 3 * n)).astype(dt)
    out = {}
    for mode in (0, 1):
        eng = spme_gb300.Engine(n, L, xi, K, p, precision=prec, max_nrhs=R, tile=tile,
                                terms=spme_gb300.TERM_RECIP)
        if mode == 0:
            eng.set_spread_mode(0)
        eng.set_positions(pos)
        out[mode] = eng.apply(f)
        eng.close()
    assert relerr(out[1], out[0]) < tol_k
    assert relerr(out[1], oracle.recip(pos, L, xi, K, p, f.astype(np.float64))) < tol_o
