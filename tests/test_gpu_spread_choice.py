"""The spread that an engine takes: the default (mode 1) can be had back after mode 0,
on meshes too small for the column gather too, and a tile whose boxes do not fit takes
the column gather; boxes above the line of particles per mesh point, against the other
kernels and the oracle (tolerances as the spread kernels' tests have them), and none below."""
import numpy as np
import pytest

import oracle
import spme_gb300
from conftest import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,K,p,R,n", [
    ("fp64", 9, 8, 1, 300),    # boxes, no column gather
    ("fp64", 12, 6, 2, 300),
    ("fp64", 48, 6, 1, 9000),  # boxes beside the column gather
    ("fp64", 40, 4, 4, 900),   # column gather
    ("fp32", 48, 6, 4, 9000),
])
def test_default_and_back(gpu_lib, prec, K, p, R, n):
    rng = np.random.default_rng(K)
    pos = rng.uniform(0, 40.0, (n, 3))
    f = rng.standard_normal((R, 3 * n)).astype(np.float32 if prec == "fp32" else np.float64)
    with spme_gb300.Engine(n, 40.0, 0.4, K, p, precision=prec, max_nrhs=R,
                           terms=spme_gb300.TERM_RECIP) as eng:
        eng.set_positions(pos)
        u = eng.apply(f)
        c = eng.launch_count()
        eng.apply(f)
        d = eng.launch_count()
        eng.set_spread_mode(0)
        eng.apply(f)
        assert eng.launch_count() - d < d - c  # the tile kernel alone
        eng.set_spread_mode(1)
        assert np.array_equal(eng.apply(f), u)


def test_no_other_spread(gpu_lib):
    # FP32, mesh too small for the column gather and no boxes: mode 1 stays refused
    with spme_gb300.Engine(100, 20.0, 0.4, 16, 6, precision="fp32", max_nrhs=4,
                           terms=spme_gb300.TERM_RECIP) as eng:
        with pytest.raises(spme_gb300.SpmeError) as err:
            eng.set_spread_mode(1)
        assert err.value.code == spme_gb300.ERR_UNSUPPORTED


def test_tile_without_boxes(gpu_lib):
    # 5x5x5 tiles at K = 410: over 4 GB of boxes for a component.  The column gather's two
    # kernels against the tile kernel's one (boxes: two per component); results as the
    # kernels' tests have them (FP64 1e-13 relative L2)
    n, L, K = 80_000, 700.0, 410
    rng = np.random.default_rng(K)
    pos, f = rng.uniform(0, L, (n, 3)), rng.standard_normal((1, 3 * n))
    out, used = {}, {}
    with spme_gb300.Engine(n, L, 0.3, K, 6, precision="fp64", max_nrhs=1,
                           terms=spme_gb300.TERM_RECIP) as eng:
        for name, tile, mode in (("default", (8, 8, 8), 1), ("small", (5, 5, 5), 1),
                                 ("tiles", (5, 5, 5), 0), ("again", (8, 8, 8), 1)):
            eng.set_spread_mode(mode)
            eng.set_tile(*tile)
            eng.set_positions(pos)
            c = eng.launch_count()
            out[name] = eng.apply(f)
            used[name] = eng.launch_count() - c
    assert used["small"] == used["tiles"] + 1
    assert np.array_equal(out["default"], out["again"])
    for name in ("small", "tiles"):
        assert np.linalg.norm(out[name] - out["default"]) < 1e-13 * np.linalg.norm(out["default"])


# Sizes at which boxes are taken (particles per mesh point above the line): tile edges of
# p - 1 and below on no, one (each) and several axes, tiles that do not divide K, a mesh
# smaller than a tile and its halo, nearly empty tiles.
@pytest.mark.parametrize("prec,K,p,tile,R,n", [
    ("fp64", 32, 6, None, 1, 800),
    ("fp64", 32, 4, None, 2, 2000),
    ("fp64", 40, 8, None, 3, 1200),
    ("fp64", 32, 6, (4, 8, 8), 1, 800),
    ("fp64", 32, 6, (8, 4, 8), 1, 800),
    ("fp64", 32, 6, (8, 8, 4), 2, 800),
    ("fp64", 32, 6, (4, 4, 4), 1, 1500),
    ("fp64", 33, 8, (4, 4, 4), 1, 800),
    ("fp64", 36, 8, (16, 8, 4), 2, 2500),
    ("fp64", 30, 6, (7, 5, 4), 1, 1200),
    ("fp64", 25, 8, (12, 12, 8), 1, 400),
    ("fp64", 48, 8, None, 1, 40),
    ("fp32", 96, 6, None, 1, 26_000),
    ("fp32", 96, 6, (16, 8, 4), 1, 31_000),
    ("fp32", 96, 6, (4, 4, 4), 1, 41_000),
    ("fp32", 100, 4, (8, 4, 4), 2, 45_000),
])
def test_boxes(gpu_lib, prec, K, p, tile, R, n):
    L, xi = 40.0, 0.4
    dt, tol_k, tol_o = (np.float64, 1e-13, 1e-12) if prec == "fp64" else (np.float32, 2e-6, 1e-5)
    rng = np.random.default_rng(K * p + R)
    pos = rng.uniform(0, L, (n, 3))
    pos[: n // 4] = 0.06 * pos[: n // 4] + 7.0  # a cluster within a tile or two
    f = rng.standard_normal((R, 3 * n)).astype(dt)
    out = {}
    # boxes; the tile kernel; an engine of more right-hand sides, which takes another spread
    for name, mode, most in (("box", 1, R), ("tile", 0, R), ("other", 1, 4)):
        with spme_gb300.Engine(n, L, xi, K, p, precision=prec, max_nrhs=most, tile=tile,
                               terms=spme_gb300.TERM_RECIP) as eng:
            eng.set_spread_mode(mode)
            eng.set_positions(pos)
            out[name] = eng.apply(f)
    assert not np.array_equal(out["box"], out["tile"])
    assert not np.array_equal(out["box"], out["other"])
    assert relerr(out["box"], out["tile"]) < tol_k
    assert relerr(out["box"], out["other"]) < tol_k
    assert relerr(out["box"], oracle.recip(pos, L, xi, K, p, f.astype(np.float64))) < tol_o


# Below the line: the column gather (FP64) or the tile kernel (FP32), as an engine of more
# right-hand sides takes them.
@pytest.mark.parametrize("prec,K,p,tile,R,n", [
    ("fp64", 48, 6, None, 1, 50),
    ("fp64", 48, 6, None, 2, 700),
    ("fp64", 32, 6, (4, 4, 4), 1, 800),
    ("fp64", 50, 6, None, 1, 2500),
    ("fp32", 96, 6, None, 1, 3000),
    ("fp32", 100, 6, None, 1, 60_000),
])
def test_no_boxes(gpu_lib, prec, K, p, tile, R, n):
    rng = np.random.default_rng(K * p + R)
    pos = rng.uniform(0, 40.0, (n, 3))
    f = rng.standard_normal((R, 3 * n)).astype(np.float64 if prec == "fp64" else np.float32)
    out = []
    for most in (R, 4 if prec == "fp64" else 2):
        with spme_gb300.Engine(n, 40.0, 0.4, K, p, precision=prec, max_nrhs=most, tile=tile,
                               terms=spme_gb300.TERM_RECIP) as eng:
            eng.set_positions(pos)
            out.append(eng.apply(f))
    assert np.array_equal(*out)
