"""CPU: native batches whose packed 32-bit indexes would overflow are refused before any
device work."""
import ctypes

import pytest

import spme_gb300
from spme_gb300 import BatchSystem


@pytest.mark.parametrize("precision,R,systems", [
    # three meshes of 2^30 points: one sort key per point
    (spme_gb300.SPME_FP32, 1, [(10, 1024)] * 3),
    (spme_gb300.SPME_FP64, 1, [(10, 1024)] * 3),
    # vectors of 2^31 values
    (spme_gb300.SPME_FP32, 16, [(30_000_000, 64), (20_000_000, 64)]),
    # 40e6 particles: 1.9e9 values, but 2.6e9 in the padded rows of FP64
    (spme_gb300.SPME_FP64, 16, [(40_000_000, 64)]),
])
def test_refused(precision, R, systems):
    lib = spme_gb300.load()
    arr = (BatchSystem * len(systems))()
    for a, (n, K) in zip(arr, systems):
        a.np, a.dim, a.porder = n, K, 4
        a.box_size, a.xi, a.radius, a.rcut = 1000.0, 0.3, 1.0, 10.0
    out = ctypes.c_void_p()
    st = lib.spme_batch_create(arr, len(systems), R, precision, ctypes.byref(out))
    assert st == spme_gb300.ERR_UNSUPPORTED and not out.value
