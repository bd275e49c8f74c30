"""The whole-GPU path's three Householder reductions: which one a tuned choice applies to, and that they agree at the odd sizes and
at the edges of 64-row stripes."""
import ctypes
import json

import numpy as np
import pytest

from helpers import A2B
from pm3_rs import _lib, native, workloads
from test_gpu_size_edges import cluster

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


@pytest.mark.parametrize("unit", [dict(w=9, h=2, r=1), dict(w=20, r=1), dict(w=20, h=1, r=1), dict(w=42)])  # n = 65, 127, 129, 252
def test_tiles_panels_and_multi_launch_agree(monkeypatch, unit):
    """The same molecule on each form and on one CTA; the bars of the GPU suite, MO energies to first order in the density's 1e-8."""
    z, xyz = cluster(**unit)
    opts = native.options(p_tol=1e-8, multiplicity=2 if "r" in unit else 1)
    one = _lib.Context()
    try:
        assert one.lib.pm3gpu_set_large_threshold(one.ptr, 257) == 0
        ref = native.run(z, xyz, opts, context=one, want_mo_energies=True)
    finally:
        one.close()
    for tiles, coop in (("1", "1"), ("0", "1"), ("0", "0")):
        monkeypatch.setenv("PM3GPU_TILE_REDUCE", tiles)
        monkeypatch.setenv("PM3GPU_COOP_PANELS", coop)
        c = _context()
        try:
            got = native.run(z, xyz, opts, context=c, want_mo_energies=True)
        finally:
            c.close()
        assert got["converged"] and ref["converged"]
        assert abs(got["heat_of_formation_kcal"] - ref["heat_of_formation_kcal"]) < 1e-6
        assert np.abs(got["charges"] - ref["charges"]).max() < 1e-5
        assert np.abs(got["mo_energies"] - ref["mo_energies"]).max() < 1e-6


@pytest.mark.parametrize("waters,ammonias", [(244, 1), (242, 3), (245, 1)])  # 1471 functions: tiles; 1473 and 1477: panels, odd rows
def test_eigensolver_at_odd_sizes_around_the_last_tile(waters, ammonias):
    z, xyz = workloads.water_cluster(waters, grid=(7, 6, 6))
    z, xyz = list(z), list(np.asarray(xyz))
    top = np.max(xyz, axis=0)
    for k in range(ammonias):
        at = top + np.array([0.0, -4.0 * k, 4.0])
        z += [7, 1, 1, 1]
        xyz += [at, at + [0.94, 0.0, 0.38], at + [-0.47, 0.81, 0.38], at + [-0.47, -0.81, 0.38]]
    c = _context()
    try:
        assert c.lib.pm3gpu_set_large_checks(c.ptr, 1) == 0
        got = native.run(np.array(z, np.int32), np.array(xyz) * A2B, native.options(), context=c)
        rows = np.zeros((200, 6))
        k = c.lib.pm3gpu_last_large_checks(c.ptr, rows.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), 200)
    finally:
        c.close()
    assert got["converged"] and k >= got["iterations"]
    assert rows[:k, 3].max() < 1e-11
    assert rows[:k, 4].max() < 1e-9  # |F| about 150 eV, 1477 eps |F| = 5e-11 for one backward-stable pass, 20 of them
