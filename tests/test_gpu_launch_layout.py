"""pm3gpu_last_launch_layout: the reported size is one whose matrix the layout holds on chip."""
import ctypes

import pytest

from pm3_rs import _lib, native
from test_gpu_size_edges import cluster

pytestmark = pytest.mark.gpu


# One molecule, one CTA per SM: about 225 KB beside the carve-out, 25.7k doubles at 252 basis functions. The reduction takes 15
# doubles a frame row and 256 a block: 23072 for the 224 rows of n = 209 .. 224, 27152 for 240.
@pytest.mark.parametrize("unit,size", [(dict(w=35), 210), (dict(w=42), 224)])
def test_reported_size_fits(unit, size):
    z, xyz = cluster(**unit)
    c = _lib.Context()
    try:
        assert native.run(z, xyz, native.options(), context=c)["converged"]
        ctas, n = ctypes.c_int(), ctypes.c_int()
        assert c.lib.pm3gpu_last_launch_layout(c.ptr, ctypes.byref(ctas), ctypes.byref(n)) == _lib.OK
    finally:
        c.close()
    assert (ctas.value, n.value) == (1, size)
