"""The FP32 real-space sum at the edges of its two forms (up to 4 right-hand sides:
pairs split over the lanes; more: lanes of two right-hand sides), against the
FP64 oracle: odd counts (a padded column), one and two blocks of right-hand
sides, cells with more particles than are listed together, more pairs than a list
or a compensated run holds, more candidates than are staged, minimum images,
no pairs at all.  1e-5 relative L2, the repository's FP32 bound."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu

TERMS = spme_gb300.TERM_REAL | spme_gb300.TERM_SELF


def _run(pos, L, xi, rc, f, max_nrhs, a=1.0):
    eng = spme_gb300.Engine(pos.shape[0], L, xi, 16, 4, radius=a, rcut=rc, precision="fp32",
                            max_nrhs=max_nrhs, terms=TERMS)
    try:
        eng.set_positions(pos)
        return eng.apply(f).astype(np.float64)
    finally:
        eng.close()


@pytest.mark.parametrize("R,max_nrhs", [(1, 1), (2, 2), (3, 3), (4, 4), (5, 5), (6, 8), (9, 9),
                                        (16, 16), (17, 17), (37, 37), (7, 5)])
def test_right_hand_sides(gpu_lib, R, max_nrhs):
    n, L, rc, xi = 1500, 42.0, 10.0, 0.3
    rng = np.random.default_rng(R)
    pos, f = rng.uniform(0, L, (n, 3)), rng.standard_normal((R, 3 * n)).astype(np.float32)
    ref = oracle.real_self(pos, L, xi, rc, f.astype(np.float64))
    assert relerr(_run(pos, L, xi, rc, f, max_nrhs), ref) < 1e-5


@pytest.mark.parametrize("R", [1, 6])
@pytest.mark.parametrize("n,L,rc,xi", [
    (1, 30.0, 9.0, 0.4),
    (33, 90.0, 9.0, 0.4),     # mostly empty cells
    (900, 31.0, 10.0, 0.3),   # ~33 particles per cell, 900 candidates (not staged)
    (700, 25.0, 9.0, 0.35),   # one cell, minimum images
    (300, 12.0, 5.9, 0.5),    # ... nearly every pair within rc
])
def test_cells(gpu_lib, n, L, rc, xi, R):
    rng = np.random.default_rng(n)
    pos, f = rng.uniform(0, L, (n, 3)), rng.standard_normal((R, 3 * n)).astype(np.float32)
    ref = oracle.real_self(pos, L, xi, rc, f.astype(np.float64))
    assert relerr(_run(pos, L, xi, rc, f, R), ref) < 1e-5
