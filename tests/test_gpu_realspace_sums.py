"""Sums of the FP32 real-space part that lose their small terms in plain FP32: of a
particle's partners two pull with forces 2^20 times the others' that cancel exactly
(mirrored positions, opposite forces), with a small term between them, so placed that
they meet it only in a compensated sum.  One cell, so the partners are listed in index
order; the others feel zero forces.  The error is that of the one particle's result
against the FP64 oracle, whose bound is the repository's 1e-5 (a sum that loses the
small term is off by 2^20 2^-24 or more)."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu

BIG = 2.0 ** 20


@pytest.mark.parametrize("R,n,who,plus,small,minus", [
    # up to 4: a lane's share of the 13 x 25 pairs that a warp lists, eleven of them
    (1, 26, 0, 1, 2, 3),
    (1, 26, 0, 1, 5, 9),
    (2, 26, 0, 1, 5, 9),
    (3, 26, 0, 1, 5, 9),
    (4, 26, 0, 1, 5, 9),
    # more than 4 right-hand sides: pair slots of 32 / 4, 32 / 8, 32 / 16 lanes
    (5, 26, 0, 1, 2, 3),      # three slots, summed across slots
    (12, 26, 0, 1, 2, 3),
    (17, 99, 1, 0, 41, 97),   # one slot: a run goes on in the next two windows of pairs
])
def test_cancelling_partners(gpu_lib, R, n, who, plus, small, minus):
    L, rc, xi = 40.0, 19.0, 0.3
    rng = np.random.default_rng(R)
    centre = np.full(3, 20.0)
    d = rng.standard_normal((n, 3))
    pos = centre + 9.0 * d / np.linalg.norm(d, axis=1)[:, None] * rng.uniform(0.4, 1.0, (n, 1))
    pos[who], pos[plus], pos[minus] = centre, centre + [2.0, 1.5, 0.5], centre - [2.0, 1.5, 0.5]
    f = np.zeros((R, n, 3), dtype=np.float32)
    f[:, who] = rng.standard_normal((R, 3))
    f[:, small] = rng.standard_normal((R, 3))
    f[:, plus] = BIG * rng.standard_normal((R, 3))
    f[:, minus] = -f[:, plus]
    f = f.reshape(R, 3 * n)
    eng = spme_gb300.Engine(n, L, xi, 16, 4, rcut=rc, precision="fp32", max_nrhs=R,
                            terms=spme_gb300.TERM_REAL | spme_gb300.TERM_SELF)
    eng.set_positions(pos)
    u = eng.apply(f).reshape(R, n, 3)[:, who]
    eng.close()
    ref = oracle.real_self(pos, L, xi, rc, f.astype(np.float64)).reshape(R, n, 3)[:, who]
    for r in range(R):
        assert relerr(u[r], ref[r]) < 1e-5, r
