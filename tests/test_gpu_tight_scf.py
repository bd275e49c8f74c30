"""Solves under the reference's second-derivative tolerances (pm3-rs src/hessian.rs:169-175), which run on the sums of
scf_tight.cuh: the Hessians they give stay what they were, and the solves agree with the oracle over the sizes at which that
kernel's matrices change place (packed triangle in shared or global memory, 2, 4 or 8 rows a lane)."""
import json
import os

import numpy as np
import pytest

import oracle as O
from helpers import A2B
from pm3_rs import _lib, native, workloads
from test_gpu_size_edges import cluster

pytestmark = pytest.mark.gpu
TIGHT = dict(e_tol=1e-12, p_tol=1e-11, max_scf=500)
HOF_TOL = 1e-6
Q_TOL = 1e-5
with open(os.path.join(os.path.dirname(__file__), "golden", "hessian_8_atoms.json")) as f:
    KEPT = json.load(f)["molecules"]


@pytest.mark.parametrize("k", range(len(KEPT)))
def test_hessians_keep_their_values(k):
    """What is left of the iteration when it stops, up to 1e-11 of the density, depends on the order of its sums and is 1e-9 of the
    Hessian. The bar is the rounding of the gradients: terms of up to 1e3 eV/Bohr, 1e-13 each, over 2e-3 Bohr, on a norm of
    1e2 eV/Bohr^2, with a margin."""
    m = KEPT[k]
    z, xyz = np.array(m["z"], np.int32), np.array(m["xyz_bohr"])
    nd = 3 * len(z)
    ref = np.zeros((nd, nd))
    ref[np.tril_indices(nd)] = m["lower"]
    ref = np.tril(ref) + np.tril(ref, -1).T
    got = native.numerical_hessian_batch(np.array([0, len(z)], np.int32), z, xyz)["hessians"][0]
    assert np.linalg.norm(got - ref) < 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("k", range(len(KEPT)))
def test_dipole_derivatives_keep_their_values(k):
    """The same for the dipole, whose rounding (charges of a few e Bohr, 1e-15 each) over 2e-3 Bohr is 1e-12."""
    z, xyz = np.array(KEPT[k]["z"], np.int32), np.array(KEPT[k]["xyz_bohr"])
    with open(os.path.join(os.path.dirname(__file__), "golden", "dipole_derivatives_8_atoms.json")) as f:
        ref = np.array(json.load(f)["derivatives"][k])
    got = native.dipole_derivatives_batch(np.array([0, len(z)], np.int32), z, xyz)["derivatives"][0]
    assert np.linalg.norm(got - ref) < 1e-10 * np.linalg.norm(ref)


def _check(res, m, z, xyz_bohr, **opts):
    ref = O.single_point(z, xyz_bohr, **opts)
    assert res.status[m] == 0 and res.unrestricted[m] == ref["unrestricted"]
    assert abs(res.heat_of_formation_kcal[m] - ref["heat_of_formation_kcal"]) < HOF_TOL
    assert np.abs(res.charges_of(m) - ref["charges"]).max() < Q_TOL


@pytest.mark.parametrize("units", [[dict(h=1), dict(w=10, h=2), dict(w=11), dict(w=21, h=1), dict(w=21, h=2)], [dict(w=27), dict(w=42)],
                                   [dict(h=57), dict(n=14)]])
def test_closed_shells_match_oracle(units):
    mols = [cluster(**u) for u in units]
    offs, z, xyz = workloads.pack(mols)
    res = native.batch(offs, z, xyz, native.options(**TIGHT))
    for m, (zm, xm) in enumerate(mols):
        _check(res, m, zm, xm, **TIGHT)


def test_two_spins_and_the_stability_search_match_oracle():
    mols = [cluster(r=1), cluster(w=4, h=1, r=1)]
    offs, z, xyz = workloads.pack(mols)
    opts = dict(TIGHT, multiplicity=2, max_scf=2000)
    res = native.batch(offs, z, xyz, native.options(**opts))
    for m, (zm, xm) in enumerate(mols):
        _check(res, m, zm, xm, **opts)
    z, xyz = workloads.organic(9, 709)
    offs, x = np.array([0, len(z), 2 * len(z)], np.int32), np.concatenate([xyz, xyz]) * A2B
    opts = dict(TIGHT, stability=2)
    res = native.batch(offs, np.concatenate([z, z]), x, native.options(**opts))
    assert res.scf_paths_tried[0] == O.single_point(z, xyz * A2B, **opts)["scf_paths_tried"] > 1
    _check(res, 1, z, xyz * A2B, **opts)


def test_a_launch_that_mixes_tolerances():
    """One launch with and without these tolerances runs the common kernel; the solves agree with those on their own."""
    a, b = workloads.organic(12, 5), workloads.organic(15, 6)
    offs, z, xyz = workloads.pack([a, b])
    both = native.batch(offs, z, xyz * A2B, [native.options(**TIGHT), native.options(p_tol=1e-8)])
    alone = native.batch(offs, z, xyz * A2B, native.options(**TIGHT))
    assert (both.status == 0).all() and (alone.status == 0).all()
    assert np.abs(both.heat_of_formation_kcal - alone.heat_of_formation_kcal).max() < HOF_TOL
    assert np.abs(both.charges - alone.charges).max() < Q_TOL


def test_a_lone_large_molecule_takes_the_whole_gpu():
    """From 192 basis functions on; the one CTA of this kernel would take 180 ms at 252."""
    z, xyz = workloads.water_cluster(32, grid=(4, 4, 2))
    c = _lib.Context()
    try:
        got = native.run(z, xyz * A2B, native.options(**TIGHT), context=c)
        assert c.lib.pm3gpu_last_kernel_launches(c.ptr) > 20
        ref = native.run(z, xyz * A2B, native.options(p_tol=1e-8), context=c)
    finally:
        c.close()
    assert abs(got["heat_of_formation_kcal"] - ref["heat_of_formation_kcal"]) < HOF_TOL
