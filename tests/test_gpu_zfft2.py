"""Two-factor fused z transform (FP32): every supported mesh size and several
right-hand-side counts, against the same engine's 3D transforms and influence
pass."""
import pytest
import torch

import spme_gb300 as sp

pytestmark = pytest.mark.gpu

# Both paths round in FP32.  Per direction and axis at most 8 radix stages, each at
# most 2.5 roundings (a sum and a twiddle product), two directions, three axes: 120
# roundings of 2^-24 in the worst (linear) case.
TOL = 120 * 2.0 ** -24


@pytest.mark.parametrize("K,R", [
    (16, 1), (18, 2), (20, 3), (24, 5), (27, 4), (30, 1), (32, 16), (36, 2), (40, 3), (48, 1),
    (50, 5), (54, 2), (60, 3), (64, 9), (72, 4), (75, 8), (80, 1), (90, 3), (96, 2), (100, 5),
    (108, 1), (120, 7), (128, 1), (135, 2), (144, 3), (150, 1), (160, 5), (162, 2), (180, 1),
    (192, 2), (200, 3), (216, 1), (240, 2), (243, 1), (250, 1), (256, 3)])
def test_against_3d_path(K, R):
    n, L = 200, K / 0.55
    gen = torch.Generator(device="cuda").manual_seed(K)
    pos = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * L
    f = torch.randn((R, 3 * n), generator=gen, device="cuda", dtype=torch.float32)
    eng = sp.Engine(n, L, 0.3, K, 4, precision="fp32", max_nrhs=R, terms=sp.TERM_RECIP)
    eng.set_positions(pos)
    u = {}
    for mode in (1, 0):
        eng.set_fft_mode(mode)
        u[mode] = torch.zeros_like(f)
        eng.apply(f, u[mode])
        torch.cuda.synchronize()
    eng.close()
    assert torch.linalg.norm(u[1] - u[0]) <= TOL * torch.linalg.norm(u[0])
