"""Engines and batches of unlike tiles in one process: one's captured graphs replay after
the other ran the same kernels with less shared memory, and two threads drive one engine
each."""
import threading

import numpy as np
import pytest

import spme_gb300

pytestmark = pytest.mark.gpu


def _engine(prec, K, p, R, tile, n, L):
    return spme_gb300.Engine(n, L, 0.3, K, p, rcut=10.0, precision=prec, max_nrhs=R, tile=tile)


@pytest.mark.parametrize("prec,p,R", [("fp64", 8, 1), ("fp64", 8, 4), ("fp32", 8, 1), ("fp32", 6, 8)])
def test_replay_after_smaller_tile(gpu_lib, prec, p, R):
    import torch
    n, L, K = 3000, 60.0, 48
    dt = torch.float32 if prec == "fp32" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(p)
    pos = torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) * L
    f = torch.randn((R, 3 * n), generator=gen, device="cuda", dtype=dt)
    u = torch.zeros_like(f)
    big, small = (_engine(prec, K, p, R, t, n, L) for t in ((16, 8, 8), (4, 4, 4)))
    big.set_graphs(True)
    first = None
    for _ in range(3):
        u.zero_()
        big.set_positions(pos)
        big.apply(f, u)
        torch.cuda.synchronize()
        if first is None:
            first = u.clone()
        assert torch.equal(u, first)
        small.set_positions(pos)
        small.apply(f)
        torch.cuda.synchronize()
    big.close()
    small.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_two_threads(gpu_lib, prec):
    n, L, K, R = 2000, 60.0, 48, 1
    rng = np.random.default_rng(3)
    pos = rng.uniform(0, L, (n, 3))
    f = rng.standard_normal((R, 3 * n)).astype(np.float32 if prec == "fp32" else np.float64)
    wrong = []

    def work(tile):
        try:
            with _engine(prec, K, 8, R, tile, n, L) as eng:
                eng.set_positions(pos)
                ref = eng.apply(f)
                for _ in range(60):
                    eng.set_positions(pos)
                    if not np.array_equal(eng.apply(f), ref):
                        wrong.append(tile)
        except Exception as e:  # noqa: BLE001 (told by the main thread)
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in ((16, 8, 8), (4, 4, 4))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
