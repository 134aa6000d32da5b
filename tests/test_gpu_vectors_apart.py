"""Right-hand sides, and the systems of a batch, stay apart: vectors of unlike size in
one call keep their own accuracy (the error is taken per vector), a zero vector gives
exact zeros, and a vector of NaN leaves the others bitwise as they are without it.
Odd mesh sizes among them: a mesh of an odd K has an odd number of rows, so the rows of
two components could share a transform.

FP32 1e-5 and FP64 1e-12 relative L2 against the oracle, the repository's bounds."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu

SCALES = [1.0, 1e-6, 0.0, 1.0]


@pytest.mark.parametrize("prec,K", [("fp32", 27), ("fp32", 32), ("fp32", 75), ("fp32", 135),
                                    ("fp64", 25), ("fp64", 27), ("fp64", 45), ("fp64", 75),
                                    ("fp64", 81), ("fp64", 135)])
def test_right_hand_sides(gpu_lib, prec, K):
    n, L, xi, p, R = 300, K / 0.6, 0.3, 4, len(SCALES)
    dt, tol = (np.float32, 1e-5) if prec == "fp32" else (np.float64, 1e-12)
    rng = np.random.default_rng(K)
    pos = rng.uniform(0, L, (n, 3))
    # some at the corner of the box: stencils in the first and the last rows of a mesh
    pos[:20] = rng.uniform(-0.5, 0.5, (20, 3)) * L / K
    f = (rng.standard_normal((R, 3 * n)) * np.array(SCALES)[:, None]).astype(dt)
    eng = spme_gb300.Engine(n, L, xi, K, p, precision=prec, max_nrhs=R,
                            terms=spme_gb300.TERM_RECIP)
    eng.set_fft_mode(1)
    eng.set_positions(pos)
    u = eng.apply(f)
    for r in range(R):
        if SCALES[r] == 0.0:
            assert not u[r].any()
        else:
            ref = oracle.recip(pos, L, xi, K, p, f[r:r + 1].astype(np.float64))
            assert relerr(u[r], ref[0]) < tol, r
    for bad in range(R):
        g = f.copy()
        g[bad] = np.nan
        v = eng.apply(g)
        assert np.isnan(v[bad]).all()
        for r in range(R):
            assert r == bad or np.array_equal(u[r], v[r]), (bad, r)
    eng.close()


@pytest.mark.parametrize("prec,tol", [("fp32", 1e-5), ("fp64", 1e-12)])
@pytest.mark.parametrize("R", [1, 3])
def test_systems(gpu_lib, prec, tol, R):
    import torch
    dt = torch.float32 if prec == "fp32" else torch.float64
    systems = [dict(N=200 + 50 * k, L=40.0 + k, K=27, p=4, xi=0.3, rc=10.0, radius=1.0)
               for k in range(len(SCALES))]
    rng = np.random.default_rng(R)
    pos = [rng.uniform(0, s["L"], (s["N"], 3)) for s in systems]
    for s, x in zip(systems, pos):
        x[:5] = rng.uniform(-0.5, 0.5, (5, 3)) * s["L"] / s["K"]
    f = [torch.tensor(rng.standard_normal((R, 3 * s["N"])) * c, device="cuda", dtype=dt)
         for s, c in zip(systems, SCALES)]
    b = spme_gb300.Batch(systems, nrhs=R, precision=prec)
    pos_d = b.pack([torch.tensor(x, device="cuda") for x in pos])

    def step(forces):
        f_d = b.pack(forces)
        u_d = torch.zeros_like(f_d)
        b.step(pos_d, f_d, u_d)
        torch.cuda.synchronize()
        return [x.cpu().numpy() for x in b.unpack(u_d)]

    u = step(f)
    for s, x, fk, uk, c in zip(systems, pos, f, u, SCALES):
        if c == 0.0:
            assert not uk.any()
            continue
        ref = oracle.full(x, s["L"], s["xi"], s["rc"], s["K"], s["p"],
                          fk.double().cpu().numpy())
        assert relerr(uk, ref) < tol, c
    for bad in range(len(systems)):
        v = step([torch.full_like(x, float("nan")) if k == bad else x for k, x in enumerate(f)])
        assert np.isnan(v[bad]).all()
        for k in range(len(systems)):
            assert k == bad or np.array_equal(u[k], v[k]), (bad, k)
    b.close()
