"""The whole-GPU path's three Householder reductions: which one a tuned choice applies to, and that they agree at the odd sizes and
at the edges of 64-row stripes."""
import json

import numpy as np
import pytest

from helpers import A2B
from pm3_rs import _lib, native, workloads

pytestmark = pytest.mark.gpu


def _context(tuning=None):
    c = _lib.Context()
    assert c.lib.pm3gpu_set_large_threshold(c.ptr, 1) == 0
    if tuning is not None:
        assert c.lib.pm3gpu_load_tuning(c.ptr, str(tuning).encode()) == 0, c.last_error()
    return c


@pytest.mark.parametrize("entry,applies", [({"n_le": 2048, "coop": 0}, False),             # measured with panels, n = 1500 or so
                                           ({"n_le": 512, "coop": 0}, False),              # a file from before the tiles
                                           ({"n_le": 512, "tiles": 0, "coop": 0}, False),
                                           ({"n_le": 512, "tiles": 1, "coop": 0}, True),
                                           ({"n_le": 512, "tiles": 1, "coop": 1}, False)])
def test_a_tuned_choice_applies_to_the_form_it_was_measured_with(tmp_path, entry, applies):
    z, xyz = workloads.water_cluster(22, grid=(4, 3, 2))  # 132 basis functions
    path = tmp_path / "tuning.json"
    path.write_text(json.dumps({"large": [entry]}))
    runs = []
    for tuning in (None, path):
        c = _context(tuning)
        try:
            r = native.run(z, xyz * A2B, native.options(), context=c)
            runs.append((r["iterations"], c.lib.pm3gpu_last_kernel_launches(c.ptr), r["heat_of_formation_kcal"]))
            if tuning:
                assert c.lib.pm3gpu_tuning_choice(c.ptr, 1, 132) == (entry["coop"] if entry.get("tiles") else -1)
                assert c.lib.pm3gpu_tuning_choice(c.ptr, 1, 1473) == (0 if entry["n_le"] == 2048 else -1)
        finally:
            c.close()
    (ia, la, ha), (ib, lb, hb) = runs
    assert ia == ib and abs(ha - hb) < 1e-6
    assert (lb > la + 132 * ib) if applies else lb == la  # five launches a column against one launch


def test_tuning_file_keeps_the_form(tmp_path):
    bad = tmp_path / "bad.json"
    bad.write_text('{"large": [{"n_le": 512, "tiles": 2, "coop": 1}]}')
    assert _lib.load().pm3gpu_load_tuning(None, str(bad).encode()) == _lib.INVALID_INPUT
