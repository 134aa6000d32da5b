"""Native batches whose packed meshes would leave the vector alignment: an odd
number of right-hand sides with odd and even mesh sizes in one batch (an odd K
holds an odd number of values, so the meshes packed after it would start on odd
elements).  FP32 1e-5 and FP64 1e-12 relative L2 against the oracle, the
repository's bounds."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("fp64", 1e-12)])
@pytest.mark.parametrize("R", [1, 3])
def test_batch_odd_mesh_before_even(gpu_lib, precision, tol, R):
    import torch
    systems = [dict(N=700, L=36.0, K=25, p=4, xi=0.35, rc=9.0, radius=1.0),
               dict(N=900, L=40.0, K=30, p=6, xi=0.3, rc=10.0, radius=1.0),
               dict(N=800, L=38.0, K=36, p=8, xi=0.35, rc=9.0, radius=1.0),
               dict(N=1100, L=44.0, K=32, p=8, xi=0.3, rc=10.0, radius=1.0)]
    rng = np.random.default_rng(R)
    dt = torch.float32 if precision == "fp32" else torch.float64
    pos = [rng.uniform(0, s["L"], (s["N"], 3)) for s in systems]
    f = [rng.standard_normal((R, 3 * s["N"])) for s in systems]
    b = spme_gb300.Batch(systems, nrhs=R, precision=precision)
    pos_d = b.pack([torch.tensor(x, device="cuda") for x in pos])
    f_d = b.pack([torch.tensor(x, device="cuda", dtype=dt) for x in f])
    u_d = torch.zeros_like(f_d)
    b.step(pos_d, f_d, u_d)
    torch.cuda.synchronize()
    for s, x, fk, uk in zip(systems, pos, f, b.unpack(u_d)):
        ref = oracle.full(x, s["L"], s["xi"], s["rc"], s["K"], s["p"],
                          fk.astype(np.float32).astype(np.float64) if precision == "fp32" else fk)
        assert relerr(uk.cpu().numpy().astype(np.float64), ref) < tol
    b.close()
