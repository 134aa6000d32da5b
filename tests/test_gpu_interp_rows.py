"""FP32 interpolation where TMA does not reach (mesh rows not a multiple of 16 bytes):
16-wide box rows at tiles of 8 columns or fewer, 24-wide ones above, copies of 8 bytes (even
K) and 4 bytes (odd K), engines and batches, against the oracle (FP32 1e-5, the
repository's bound)."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr, uniform_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [(8, 8, 8), (8, 4, 4), (5, 8, 4), (9, 8, 8), (16, 8, 4)])
@pytest.mark.parametrize("K,p", [(27, 4), (30, 6), (35, 8), (75, 4), (50, 6), (29, 8)])
def test_engine_rows(gpu_lib, tile, K, p):
    n, L, R = 500, 1.2 * K, 3
    pos, f = uniform_case(n, L, R, seed=K + p)
    eng = spme_gb300.Engine(n, L, 0.35, K, p, precision="fp32", max_nrhs=R,
                            terms=spme_gb300.TERM_RECIP)
    eng.set_tile(*tile)
    eng.set_positions(pos)
    u = eng.apply(f.astype(np.float32))
    eng.close()
    ref = oracle.recip(pos, L, 0.35, K, p, f.astype(np.float32).astype(np.float64), nthreads=4)
    assert relerr(u, ref) < 1e-5


@pytest.mark.parametrize("tile", [(8, 8, 8), (16, 8, 4)])
def test_batch_rows(gpu_lib, tile):
    import torch
    systems = [dict(N=400, L=36.0, K=27, p=4, xi=0.35, rc=9.0, radius=1.0),
               dict(N=500, L=40.0, K=30, p=6, xi=0.3, rc=10.0, radius=1.0),
               dict(N=450, L=38.0, K=36, p=8, xi=0.35, rc=9.0, radius=1.0),
               dict(N=600, L=42.0, K=29, p=8, xi=0.3, rc=10.0, radius=1.0)]
    R = 2
    rng = np.random.default_rng(5)
    pos = [rng.uniform(0, s["L"], (s["N"], 3)) for s in systems]
    f = [rng.standard_normal((R, 3 * s["N"])).astype(np.float32) for s in systems]
    b = spme_gb300.Batch(systems, nrhs=R, precision="fp32")
    b.set_tile(*tile)
    u_d = torch.zeros_like(f_d := b.pack([torch.tensor(x, device="cuda") for x in f]))
    b.step(b.pack([torch.tensor(x, device="cuda") for x in pos]), f_d, u_d)
    torch.cuda.synchronize()
    for s, x, fk, uk in zip(systems, pos, f, b.unpack(u_d)):
        ref = oracle.full(x, s["L"], s["xi"], s["rc"], s["K"], s["p"], fk.astype(np.float64))
        assert relerr(uk.cpu().numpy().astype(np.float64), ref) < 1e-5
    b.close()
