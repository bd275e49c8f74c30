"""The allocation-free entry's limits by size: what it refuses, in which words, and what a set threshold opens."""
import ctypes

import numpy as np
import pytest

from helpers import A2B
from pm3_rs import _lib, native, workloads

pytestmark = pytest.mark.gpu
D, I = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int32)


@pytest.mark.parametrize("n_mol,threshold,words", [(32, 0, "fewer than 192"), (42, 0, "fewer than 192"), (32, 257, None), (42, 257, "scratch"),
                                                   (32, 150, "from 150"), (43, 0, "from 257")])
def test_limits(n_mol, threshold, words):
    z, xyz = workloads.water_cluster(n_mol, grid=(4, 4, 3))
    z, x, opts = np.ascontiguousarray(z, np.int32), np.ascontiguousarray(xyz * A2B), native.options(p_tol=1e-8)
    c = _lib.Context()
    try:
        if threshold:
            assert c.lib.pm3gpu_set_large_threshold(c.ptr, threshold) == 0
        res, q = _lib.Result(), np.zeros(len(z))
        rc = c.lib.pm3gpu_single_point_noalloc(c.ptr, len(z), z.ctypes.data_as(I), x.ctypes.data_as(D), ctypes.byref(opts),
                                               ctypes.byref(res), q.ctypes.data_as(D))
        if words:
            assert rc == _lib.RESOURCE_LIMIT and words in c.last_error()
        else:
            assert rc == _lib.OK
            ref = native.run(z, x, opts, context=c)
            assert abs(res.heat_of_formation_kcal - ref["heat_of_formation_kcal"]) < 1e-6
            assert np.abs(q - ref["charges"]).max() < 1e-5
    finally:
        c.close()
