"""Native batches whose mesh sizes mix the two-factor transforms (several systems
of one size with boxes of their own) with cuFFT's (K = 28, and in FP32 K = 25, 45), in
one stream and with the groups on several.  FP32 1e-5 and FP64 1e-12 relative L2
against the oracle, the repository's bounds."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("fp64", 1e-12)])
@pytest.mark.parametrize("R", [1, 4])
def test_batch_mixed_transforms(gpu_lib, precision, tol, R):
    import torch
    systems = [dict(N=500, L=36.0, K=32, p=4, xi=0.35, rc=9.0, radius=1.0),
               dict(N=300, L=36.0, K=28, p=4, xi=0.3, rc=9.0, radius=1.0),
               dict(N=700, L=44.0, K=32, p=6, xi=0.3, rc=10.0, radius=1.0),
               dict(N=600, L=40.0, K=25, p=6, xi=0.3, rc=10.0, radius=1.0),
               dict(N=650, L=39.0, K=45, p=8, xi=0.35, rc=9.0, radius=1.0),
               dict(N=400, L=34.0, K=32, p=8, xi=0.4, rc=8.0, radius=1.0),
               dict(N=800, L=42.0, K=30, p=6, xi=0.3, rc=10.0, radius=1.0)]
    rng = np.random.default_rng(R)
    dt = torch.float32 if precision == "fp32" else torch.float64
    pos = [rng.uniform(0, s["L"], (s["N"], 3)) for s in systems]
    f = [rng.standard_normal((R, 3 * s["N"])) for s in systems]
    refs = [oracle.full(x, s["L"], s["xi"], s["rc"], s["K"], s["p"],
                        fk.astype(np.float32).astype(np.float64) if precision == "fp32" else fk)
            for s, x, fk in zip(systems, pos, f)]
    b = spme_gb300.Batch(systems, nrhs=R, precision=precision)
    pos_d = b.pack([torch.tensor(x, device="cuda") for x in pos])
    f_d = b.pack([torch.tensor(x, device="cuda", dtype=dt) for x in f])
    for overlap in (0, 2):
        b.set_overlap(overlap)
        u_d = torch.zeros_like(f_d)
        b.step(pos_d, f_d, u_d)
        torch.cuda.synchronize()
        for ref, uk in zip(refs, b.unpack(u_d)):
            assert relerr(uk.cpu().numpy().astype(np.float64), ref) < tol, overlap
    b.close()
