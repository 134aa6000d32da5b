"""The FP64 real-space sum at the edges of its work split, against the oracle:
right-hand sides around a sweep's width (4), cells with more particles than are
listed together (16), more pairs than a list holds, more candidates than are
staged (512), one cell of minimum images, single particles and empty cells.

Tolerance 1e-12 relative L2, the repository's FP64 bound (the table of the pair
functions is fitted to 2e-13 relative)."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu

TERMS = spme_gb300.TERM_REAL | spme_gb300.TERM_SELF


def _run(pos, L, xi, rc, f, a=1.0):
    eng = spme_gb300.Engine(pos.shape[0], L, xi, 16, 4, radius=a, rcut=rc, precision="fp64",
                            max_nrhs=f.shape[0], terms=TERMS)
    try:
        eng.set_positions(pos)
        return eng.apply(f)
    finally:
        eng.close()


@pytest.mark.parametrize("R", [1, 2, 3, 4, 5, 7, 9])
def test_right_hand_sides(gpu_lib, R):
    n, L, rc, xi = 1500, 42.0, 10.0, 0.3
    rng = np.random.default_rng(R)
    pos, f = rng.uniform(0, L, (n, 3)), rng.standard_normal((R, 3 * n))
    assert relerr(_run(pos, L, xi, rc, f), oracle.real_self(pos, L, xi, rc, f)) < 1e-12


@pytest.mark.parametrize("n,L,rc,xi,a", [
    (1, 30.0, 9.0, 0.4, 1.0),       # one particle, no pairs
    (2, 30.0, 9.0, 0.4, 1.0),
    (33, 90.0, 9.0, 0.4, 1.0),      # mostly empty cells
    (900, 31.0, 10.0, 0.3, 1.0),    # nc = 3: ~33 particles per cell, 900 candidates (not staged)
    (700, 25.0, 9.0, 0.35, 1.2),    # nc < 3: one cell, minimum images
    (300, 12.0, 5.9, 0.5, 1.0),     # ... nearly every pair within rc
    (1200, 40.0, 8.0, 1.0, 0.7),    # a steep kernel: finer table segments
    (4000, 60.0, 6.0, 0.8, 3.2),    # 2a beyond rc: the near form only
])
def test_cells(gpu_lib, n, L, rc, xi, a):
    rng = np.random.default_rng(n)
    pos, f = rng.uniform(0, L, (n, 3)), rng.standard_normal((2, 3 * n))
    assert relerr(_run(pos, L, xi, rc, f, a), oracle.real_self(pos, L, xi, rc, f, radius=a)) < 1e-12
