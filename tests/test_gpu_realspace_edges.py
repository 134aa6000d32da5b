"""The FP32 real-space part at the edges of the number range, against the FP64 oracle
(1e-5 relative L2, the repository's bound): particles closer than 1/r^2 can be held in
FP32, in either form of the sum, and infinite forces."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu

TERMS = spme_gb300.TERM_REAL | spme_gb300.TERM_SELF


@pytest.mark.parametrize("R", [1, 2, 4, 6, 17])
@pytest.mark.parametrize("gap", [1e-16, 1e-19, 1e-21, 1e-23])
def test_nearly_coincident(gpu_lib, gap, R):
    # near the corner of the first cell, where cell-relative positions keep such gaps
    L, rc, xi, n = 40.0, 10.0, 0.3, 40
    rng = np.random.default_rng(R)
    pos = rng.uniform(1.0, L, (n, 3))
    pos[0], pos[1] = 0.0, [gap, 0.5 * gap, 0.25 * gap]
    f = rng.standard_normal((R, 3 * n)).astype(np.float32)
    eng = spme_gb300.Engine(n, L, xi, 16, 4, rcut=rc, precision="fp32", max_nrhs=R, terms=TERMS)
    eng.set_positions(pos)
    u = eng.apply(f)
    eng.close()
    ref = oracle.real_self(pos, L, xi, rc, f.astype(np.float64))
    assert relerr(u, ref) < 1e-5


@pytest.mark.parametrize("R", [3, 5, 9, 17])
def test_infinite_force(gpu_lib, R):
    # what an infinite force component makes of the particle's own result: only that
    # component (its pairs act on the others)
    L, rc, xi, n = 40.0, 10.0, 0.3, 300
    rng = np.random.default_rng(R)
    pos = rng.uniform(0.0, L, (n, 3))
    f = rng.standard_normal((R, 3 * n)).astype(np.float32)
    f[:, 3 * np.arange(0, n, 37)] = np.inf
    eng = spme_gb300.Engine(n, L, xi, 16, 4, rcut=rc, precision="fp32", max_nrhs=R, terms=TERMS)
    eng.set_positions(pos)
    u = eng.apply(f)
    eng.close()
    ref = oracle.real_self(pos, L, xi, rc, f.astype(np.float64))
    assert np.array_equal(np.isfinite(u), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert relerr(u[ok], ref[ok]) < 1e-5
