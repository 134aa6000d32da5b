"""Two-factor x, y and fused z transforms in FP64 (the default there): every
supported mesh size, odd row counts among them, against cuFFT's 3D transforms
and the influence kernel."""
import pytest
import torch

import spme_gb300 as sp

pytestmark = pytest.mark.gpu

# Per direction and axis at most 8 radix stages, each at most 2.5 roundings (a sum and
# a twiddle product), two directions, three axes: 120 roundings of 2^-53 in the worst
# (linear) case.
TOL = 120 * 2.0 ** -53

SIZES = [16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96,
         100, 108, 120, 125, 128, 135, 144, 150, 160, 162, 180, 192, 200, 216, 225, 240, 243, 250,
         256]


@pytest.mark.parametrize("K,R", [(k, 1 + i % 3 if k <= 128 else 1) for i, k in enumerate(SIZES)])
def test_against_3d_path(K, R):
    n, L = 200, K / 0.55
    gen = torch.Generator(device="cuda").manual_seed(K)
    pos = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * L
    f = torch.randn((R, 3 * n), generator=gen, device="cuda", dtype=torch.float64)
    eng = sp.Engine(n, L, 0.3, K, 4, precision="fp64", max_nrhs=R, terms=sp.TERM_RECIP)
    eng.set_positions(pos)
    u = {}
    for mode in (1, 0):
        if mode == 0:
            eng.set_fft_mode(0)
        u[mode] = torch.zeros_like(f)
        eng.apply(f, u[mode])
        torch.cuda.synchronize()
    eng.close()
    assert torch.linalg.norm(u[1] - u[0]) <= TOL * torch.linalg.norm(u[0])
