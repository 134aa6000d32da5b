"""A caller's own stream capture of the position build and the pass right after a switch:
whatever the switch needs on the host or in device memory is made by it, not by the first
captured call.  The replay against the uncaptured engine, bitwise."""
import pytest

import spme_gb300

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,K,R,switch", [
    ("fp32", 32, 4, ("fft", 0)),
    ("fp32", 45, 2, ("fft", 0)),
    ("fp64", 32, 1, ("fft", 0)),
    ("fp64", 320, 1, ("fft", 1)),
    ("fp64", 48, 1, ("tile", (16, 16, 8))),   # boxes of another tile
    ("fp64", 48, 1, ("tile", (4, 4, 4))),     # ... more tiles
    ("fp64", 48, 4, ("tile", (16, 8, 8))),    # column gather
    ("fp64", 64, 3, ("tile", (4, 4, 4))),     # boxes to column gather
    ("fp32", 48, 8, ("tile", (8, 8, 4))),
])
def test_capture_after_switch(gpu_lib, prec, K, R, switch):
    import torch
    n, L = 3000, 60.0
    dt = torch.float32 if prec == "fp32" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(K)
    pos = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * L
    f = torch.randn((R, 3 * n), generator=gen, device="cuda", dtype=dt)
    u = [torch.zeros_like(f), torch.zeros_like(f)]
    for captured in (False, True):
        with spme_gb300.Engine(n, L, 0.3, K, 6, rcut=10.0, precision=prec, max_nrhs=R) as eng:
            if switch[0] == "fft":
                eng.set_fft_mode(switch[1])
            else:
                eng.set_tile(*switch[1])
            if captured:
                graph = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(graph):
                    eng.set_positions(pos)
                    eng.apply(f, u[1])
                graph.replay()
            else:
                eng.set_positions(pos)
                eng.apply(f, u[0])
            torch.cuda.synchronize()
    # (cuFFT's kernels are chosen by time: two engines may differ in rounding there)
    tol = 0.0 if switch[0] == "tile" else 1e-6 if prec == "fp32" else 1e-14
    assert torch.linalg.norm(u[1] - u[0]) <= tol * torch.linalg.norm(u[0])
    assert torch.linalg.norm(u[0]) > 0
