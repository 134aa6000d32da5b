"""Which kernels a call runs, and in which order: the transforms that are the default for
their sizes (told by the launches of a pass, as every transform gives the same result),
and the real-space sum beside the mesh pipeline in a replayed graph, whose kernels are
dependent launches on two streams: bitwise the serial result, again after new positions
and forces."""
import numpy as np
import pytest

import spme_gb300

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,K,own", [("fp64", k, True) for k in (16, 25, 45, 81, 96, 125)]
                         + [("fp32", k, True) for k in (16, 27, 75, 96, 128)]
                         + [("fp64", 28, False), ("fp32", 25, False), ("fp32", 45, False),
                            ("fp32", 28, False)])
def test_default_transforms(gpu_lib, prec, K, own):
    n, L = 50, 40.0
    rng = np.random.default_rng(K)
    pos = rng.uniform(0, L, (n, 3))
    f = rng.standard_normal((1, 3 * n)).astype(np.float32 if prec == "fp32" else np.float64)
    used = []
    with spme_gb300.Engine(n, L, 0.4, K, 4, precision=prec, terms=spme_gb300.TERM_RECIP) as eng:
        eng.set_positions(pos)
        for mode in (None, 0):
            if mode is not None:
                eng.set_fft_mode(mode)
            c = eng.launch_count()
            eng.apply(f)
            used.append(eng.launch_count() - c)
    # own transforms: two kernels each way and the z transform; else cuFFT (not counted) with
    # the influence's two or the z transform
    assert used[0] == used[1] + 3 if own else used[0] <= used[1]


@pytest.mark.parametrize("prec,R", [("fp32", 1), ("fp32", 4), ("fp32", 9), ("fp64", 1), ("fp64", 5)])
def test_overlap_in_graphs(gpu_lib, prec, R):
    import torch
    n, L = 5000, 75.0
    dt = torch.float32 if prec == "fp32" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(R)
    pos = torch.empty((n, 3), device="cuda", dtype=torch.float64)
    f = torch.empty((R, 3 * n), device="cuda", dtype=dt)
    engines = []
    for overlap in (False, True):
        e = spme_gb300.Engine(n, L, 0.3, 48, 6, rcut=10.0, precision=prec, max_nrhs=R)
        e.set_overlap(overlap)
        e.set_graphs(overlap)
        engines.append((e, torch.zeros_like(f)))
    for _ in range(4):
        pos.copy_(torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * L)
        f.copy_(torch.randn((R, 3 * n), generator=gen, device="cuda", dtype=dt))
        for e, u in engines:
            for _ in range(3):
                e.set_positions(pos)
                e.apply(f, u)
        torch.cuda.synchronize()
        assert torch.equal(engines[0][1], engines[1][1])
    for e, _ in engines:
        e.close()
