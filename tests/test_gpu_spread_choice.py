"""The spread that an engine takes: the default (mode 1) can be had back after mode 0,
on meshes too small for the column gather too."""
import numpy as np
import pytest

import spme_gb300

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
