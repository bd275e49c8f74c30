"""The device paths at the sizes where their splits change: 16-row blocks of the per-CTA eigensolver and products, the rows
it keeps in memory beyond 112, the two passes of the products beyond 128, molecules of one kind of atom only; 64-row stripes of
the whole-GPU reduction and its last size, 1472; the K slices of the FP64 product; the lone-molecule rule; and the pair
gradient over the shells and the orientations of its frame.

Bars as in the rest of the GPU suite: heat of formation 1e-6 kcal/mol, charges 1e-5 e, gradient components 1e-6 kcal/mol/A,
matrix products 2 K eps |A||B|.
"""
import ctypes

import numpy as np
import pytest

import oracle as O
from helpers import A2B, parse
from pm3_rs import _lib, native, workloads

pytestmark = pytest.mark.gpu
HOF_TOL = 1e-6
Q_TOL = 1e-5
GRAD_TOL = 1e-6 * 0.0433641043 / 1.8897261246
D = ctypes.POINTER(ctypes.c_double)
UNITS = {"w": ([8, 1, 1], [[0.0, 0.0, 0.0], [0.957, 0.0, 0.0], [-0.24, 0.927, 0.0]]),
         "h": ([1, 1], [[0.0, 0.0, 0.0], [0.74, 0.0, 0.0]]),
         "n": ([7, 7], [[0.0, 0.0, 0.0], [1.1, 0.0, 0.0]]),
         "r": ([6, 1, 1, 1], [[0.0, 0.0, 0.05], [1.12, 0.0, 0.0], [-0.55, 0.95, 0.0], [-0.55, -0.95, 0.0]])}


def cluster(w=0, h=0, n=0, r=0, seed=0):
    """Waters, H2, N2 and CH3 radicals (6, 2, 8 and 7 basis functions) on a shuffled, jittered grid."""
    rng = np.random.default_rng(seed + 100 * w + 10 * h + n)
    units = rng.permutation([*"w" * w, *"h" * h, *"n" * n, *"r" * r])
    side = int(np.ceil(len(units) ** (1.0 / 3.0)))
    z, xyz = [], []
    for k, u in enumerate(units):
        site = 3.3 * np.array([k % side, k // side % side, k // side // side]) + rng.uniform(-0.2, 0.2, 3)
        rot = workloads._random_rotation(rng)
        z += UNITS[u][0]
        xyz += [site + rot @ np.array(p) for p in UNITS[u][1]]
    return np.array(z, np.int32), np.array(xyz) * A2B


@pytest.fixture(scope="module")
def ctx():
    c = _lib.Context()
    yield c
    c.close()


@pytest.fixture(scope="module")
def whole():
    c = _lib.Context()
    assert c.lib.pm3gpu_set_large_threshold(c.ptr, 1) == 0
    yield c
    c.close()


def _close(got, ref):
    assert got["converged"] and ref["converged"]
    assert abs(got["heat_of_formation_kcal"] - ref["heat_of_formation_kcal"]) < HOF_TOL
    assert np.abs(np.asarray(got["charges"]) - np.asarray(ref["charges"])).max() < Q_TOL


@pytest.mark.parametrize("unit", [
    dict(h=1), dict(w=2, h=2), dict(w=3), dict(w=5, h=1), dict(w=18, h=2), dict(w=19), dict(w=21, h=1), dict(w=21, h=2), dict(w=26, h=2),
    dict(w=27), dict(w=29, h=1), dict(w=32), dict(w=32, h=1), dict(w=37, h=1), dict(w=37, h=2), dict(w=42, h=2),
    dict(h=9), dict(h=57), dict(n=2), dict(n=14), dict(n=8, h=25)])
def test_per_cta_sizes_match_oracle(ctx, unit):
    z, xyz = cluster(**unit)
    opts = dict(p_tol=1e-8)
    _close(native.run(z, xyz, native.options(**opts), context=ctx), O.single_point(z, xyz, **opts))


@pytest.mark.parametrize("unit", [dict(r=1), dict(w=1, h=1, r=1), dict(w=1, h=2, r=1), dict(w=4, h=1, r=1), dict(w=17, h=1, r=1), dict(w=17, h=2, r=1),
                                  dict(w=20, h=1, r=1)])
def test_per_cta_odd_sizes_with_two_spins_match_oracle(ctx, unit):
    z, xyz = cluster(**unit)
    opts = dict(multiplicity=2, p_tol=1e-8)
    _close(native.run(z, xyz, native.options(**opts), context=ctx), O.single_point(z, xyz, **opts))


@pytest.mark.parametrize("unit", [dict(h=1), dict(w=2, h=2), dict(w=10, h=2), dict(w=11), dict(w=21, h=1), dict(w=21, h=2), dict(w=32, h=1),
                                  dict(w=42, h=2), dict(h=33), dict(n=8)])
def test_whole_gpu_sizes_match_the_per_cta_path(ctx, whole, unit):
    z, xyz = cluster(**unit)
    opts = native.options(p_tol=1e-8)
    got = native.run(z, xyz, opts, context=whole, want_mo_energies=True)
    ref = native.run(z, xyz, opts, context=ctx, want_mo_energies=True)
    _close(got, ref)
    assert np.abs(got["mo_energies"] - ref["mo_energies"]).max() < 1e-6  # first order in the density's 1e-8


@pytest.mark.parametrize("n_mol", [245, 246])  # 1470 basis functions: in registers; 1476: panels
def test_eigensolver_on_both_sides_of_the_register_reduction(whole, n_mol):
    z, xyz = workloads.water_cluster(n_mol, grid=(7, 6, 6))
    assert whole.lib.pm3gpu_set_large_checks(whole.ptr, 1) == 0
    got = native.run(z, xyz * A2B, native.options(), context=whole)
    rows = np.zeros((200, 6))
    k = whole.lib.pm3gpu_last_large_checks(whole.ptr, rows.ctypes.data_as(D), 200)
    assert whole.lib.pm3gpu_set_large_checks(whole.ptr, 0) == 0
    assert got["converged"] and k >= got["iterations"]
    assert rows[:k, 3].max() < 1e-11
    assert rows[:k, 4].max() < 1e-9  # |F| about 150 eV, 1476 eps |F| = 5e-11 for one backward-stable pass, 20 of them


@pytest.mark.parametrize("k", [255, 256, 257, 300, 512, 1000])
@pytest.mark.parametrize("m,n", [(161, 97), (64, 64), (257, 33)])
def test_k_slices_of_small_products(ctx, m, n, k):
    rng = np.random.default_rng(k)
    a, b = np.asfortranarray(rng.standard_normal((k, m))), np.asfortranarray(rng.standard_normal((k, n)))
    c = np.zeros((m, n), order="F")
    rc = ctx.lib.pm3gpu_dgemm(ctx.ptr, 1, 0, m, n, k, 1.0, a.ctypes.data_as(D), k, b.ctypes.data_as(D), k, 0.0, c.ctypes.data_as(D), m)
    assert rc == _lib.OK, ctx.last_error()
    assert (np.abs(c - a.T @ b) <= 2 * k * np.finfo(np.float64).eps * (np.abs(a).T @ np.abs(b))).all()


@pytest.mark.parametrize("n_mol", [32, 42])  # 192 and 252 basis functions
def test_lone_molecule_route(whole, n_mol):
    z, xyz = workloads.water_cluster(n_mol, grid=(4, 4, 3))
    opts = native.options(p_tol=1e-8)
    c = _lib.Context()
    try:
        got = native.run(z, xyz * A2B, opts, context=c)
        assert c.lib.pm3gpu_last_kernel_launches(c.ptr) <= 4  # one CTA
        _close(got, native.run(z, xyz * A2B, opts, context=whole))
        assert c.lib.pm3gpu_set_large_checks(c.ptr, 1) == 0
        _close(native.run(z, xyz * A2B, opts, context=c), got)
        assert c.lib.pm3gpu_last_kernel_launches(c.ptr) > 20  # the checks belong to the whole-GPU path
        assert c.lib.pm3gpu_set_large_checks(c.ptr, 0) == 0
        res, q, x = _lib.Result(), np.zeros(len(z)), np.ascontiguousarray(xyz * A2B)
        rc = c.lib.pm3gpu_single_point_noalloc(c.ptr, len(z), z.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)), x.ctypes.data_as(D),
                                               ctypes.byref(opts), ctypes.byref(res), q.ctypes.data_as(D))
        assert rc != _lib.OK  # as before: the fixed scratch ends below 192
    finally:
        c.close()


PAIRS = {  # principal quantum numbers of the two shells, both orders, on axes of both signs
    "hcl": ("Cl 0 0 0; H -1.28 0 0", 1), "hcl_x": ("H 0 0 0; Cl -1.28 0 0", 1), "h2_z": ("H 0 0 0; H 0 0 0.74", 1),
    "acetylene_x": ("Cl 0 0 0; C 1.64 0 0; C 2.85 0 0; H 3.91 0 0", 1), "acetylene_y": ("H 0 3.91 0; C 0 2.85 0; C 0 1.64 0; Cl 0 0 0", 1),
    "silane": ("Si 0 0 0; P 2.2 0.1 0.2; Cl -0.9 1.8 0.1; H -0.6 -0.8 1.1; H -0.5 -0.7 -1.2; H 2.6 -0.6 1.3; H 2.7 1.2 0.6", 1),
    "sulfonyl": ("S 0 0 0; O 1.43 0 0; O -0.7 1.25 0; C -0.8 -0.9 1.3; H -1.8 -0.6 1.5; H -0.7 -1.9 1.0; H -0.2 -0.7 2.2; F -0.4 -0.7 -1.4", 1),
    "thiyl": ("C 0 0 0; S 0 0 -1.8; H 1.0 0 0.4; H -0.5 0.9 0.4; H -0.5 -0.9 0.4", 2)}


@pytest.mark.parametrize("name", sorted(PAIRS))
def test_pair_gradient_over_shells_and_orientations(ctx, name):
    z, xyz = parse(PAIRS[name][0])
    tight = dict(multiplicity=PAIRS[name][1], e_tol=1e-12, p_tol=1e-11, max_scf=2000)
    ref = O.single_point(z, xyz * A2B, want_gradient=True, **tight)
    got = native.run(z, xyz * A2B, native.options(**tight), want_gradient=True, context=ctx)
    assert np.abs(got["gradient"] - ref["gradient"]).max() < GRAD_TOL
