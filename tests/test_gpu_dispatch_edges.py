"""Both sides of the size rules that choose a kernel or its shape, against the
oracle at the same parameters.

Tolerance: 1e-10 of the largest value, the bound of the plain form: the splitting,
the modes and the window (converged to 1e-12) are the oracle's.  The point
potentials use another splitting than the oracle's stock sum, both converged to
1e-10: bounded at 1e-8 of the largest value."""

import math

import numpy as np
import pytest
from conftest import rel_max

import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-10
TOL_POINTS = 1e-8


@pytest.fixture(scope="module", params=["ik", "ad"])
def ctx(request, ewald_lib):
    c = ewald_lib.Context(0, ewald_lib.FP64)
    c.set_force_scheme(ewald_lib.FORCE_AD if request.param == "ad" else ewald_lib.FORCE_IK)
    yield c
    c.close()


def charges(rng, n):
    q = rng.normal(0.0, 0.4, size=n)
    return q - q.mean()


def compare(ctx, oracle, pos, q, lat, alpha, r_cut, k_cut, window):
    po, fo = oracle.fft_potential_force(pos, q, lat, 1e-8, alpha=alpha, r_cut=r_cut, k_cut=k_cut,
                                        window_cutoff=window)
    ov = dict(alpha_in=alpha, r_cut_in=r_cut, k_cut_in=k_cut, windowCutoff_in=window)
    pg, fg = ctx.potential_force(pos, q, lat, 1e-8, **ov)
    p_only = ctx.potential_force(pos, q, lat, 1e-8, want_force=False, **ov)
    assert rel_max(pg, po) < TOL
    assert rel_max(fg, fo) < TOL
    assert rel_max(p_only, po) < TOL


@pytest.mark.parametrize("n", [2047, 2048, 2049])
def test_box_sort_in_one_cta_and_in_several(ctx, oracle, n):
    rng = np.random.default_rng(n)
    lat = np.diag([30.0, 34.0, 32.0])
    compare(ctx, oracle, rng.uniform(size=(n, 3)) @ lat, charges(rng, n), lat, 0.5, 7.0, 2.0, 12)


@pytest.mark.parametrize("n,edge,k_cut", [
    (2800, 110.0, 0.9),  # 28 x 28 x 14 boxes
    (300, 80.0, 3.2),    # 21^3 tiles of 8 points
])
def test_scan_of_more_than_one_block_of_keys(ctx, oracle, n, edge, k_cut):
    rng = np.random.default_rng(n)
    lat = np.diag([edge, edge, edge])
    compare(ctx, oracle, rng.uniform(size=(n, 3)) @ lat, charges(rng, n), lat, 0.9, 4.0, k_cut, 12)


@pytest.mark.parametrize("n", [2, 15, 16, 17, 33, 127, 128, 129, 200, 400, 700])
def test_tile_lists_of_any_length(ctx, oracle, n):
    """Every atom reaches every tile of a small grid: lists of n entries, ordered in
    shared memory, in place, or by a kernel of their own."""
    rng = np.random.default_rng(n)
    lat = np.array([[9.0, 0.0, 0.0], [0.5, 10.0, 0.0], [0.3, -0.4, 9.5]])
    compare(ctx, oracle, rng.uniform(size=(n, 3)) @ lat, charges(rng, n), lat, 0.8, 4.0, 3.0, 12)


@pytest.mark.parametrize("window", [12, 13, 16, 17])
def test_weight_rows_beyond_shared_memory(ctx, oracle, window):
    """Half-widths whose rows do not fit the weights kernel's shared memory."""
    rng = np.random.default_rng(window)
    lat = np.diag([14.0, 13.0, 15.0])
    compare(ctx, oracle, rng.uniform(size=(70, 3)) @ lat, charges(rng, 70), lat, 0.8, 5.0, 4.5, window)


@pytest.mark.parametrize("alpha,r_cut", [(0.01, 9.0), (0.3, 9.0), (1.0, 9.0), (3.0, 9.0)])
def test_pair_term_over_its_range(ctx, oracle, alpha, r_cut):
    """alpha r from 1e-5 to 27, past which erfc has no double left."""
    rng = np.random.default_rng(5)
    lat = np.diag([20.0, 21.0, 19.5])
    d = np.geomspace(1e-3, 8.9, 40)
    u = rng.normal(size=(40, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    centre = rng.uniform(size=3) @ lat
    for r, w in zip(d[::4], u):  # a pair at a time: a near pair hides the others
        pos = np.stack([centre, centre + r * w])
        compare(ctx, oracle, pos, np.array([0.7, -0.7]), lat, alpha, r_cut, 1.5, 12)


@pytest.mark.parametrize("modes", [30, 50, 90])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_runtime_schedule_block_sizes(ewald_lib, oracle, modes, form):
    """Grids of 60, 100 and 180 points, no length of the register-radix passes: CTAs
    of 64, 128 and 256 threads.  The mixed form against its own result with four
    lines per CTA, which does the same arithmetic per line: 1e-6 of the largest
    value (FP32 grids)."""
    rng = np.random.default_rng(modes)
    k_cut = 2.0
    edge = 2 * math.pi / k_cut * (modes // 2 - 1.5)
    lat = np.diag([edge, edge, edge])
    pos, q = rng.uniform(size=(500, 3)) @ lat, charges(rng, 500)
    ov = dict(alpha_in=0.6, r_cut_in=5.0, k_cut_in=k_cut, windowCutoff_in=6)
    c = ewald_lib.Context(0, ewald_lib.MIXED if form == "mixed" else ewald_lib.FP64)
    try:
        pg, fg = c.potential_force(pos, q, lat, 1e-7, **ov)
        assert tuple(c.last_params()["n_modes"]) == (modes,) * 3
        if form == "mixed":
            c.set_kernel_shape({"fft_lines": 4})
            po, fo = c.potential_force(pos, q, lat, 1e-7, **ov)
            assert rel_max(pg, po) < 1e-6 and rel_max(fg, fo) < 1e-6
        else:
            po, fo = oracle.fft_potential_force(pos, q, lat, 1e-7, alpha=0.6, r_cut=5.0, k_cut=k_cut,
                                                window_cutoff=6)
            assert rel_max(pg, po) < TOL and rel_max(fg, fo) < TOL
    finally:
        c.close()


@pytest.mark.parametrize("edges", [(13.0, 15.0, 14.0), (2.6, 15.0, 2.9), (30.0, 3.0, 28.0)])
@pytest.mark.parametrize("targets", [1, 31, 65, 700])
def test_unblurred_points(ewald_lib, oracle, edges, targets):
    """Cells wide and narrow (more images of a box than the flat scan takes), with
    targets on sources and outside the cell.  The oracle's sum takes images around the
    plain difference vector, so it gets the targets folded into the cell."""
    rng = np.random.default_rng(targets)
    lat = W.triclinic_lattice(*edges, 82.0, 99.0, 93.0) * W.ANGSTROM_TO_BOHR
    src, q = rng.uniform(size=(120, 3)) @ lat, charges(rng, 120)
    tg = rng.uniform(-1, 2, size=(targets, 3)) @ lat
    tg[: min(5, targets)] = src[: min(5, targets)]
    folded = tg - np.floor(tg @ np.linalg.inv(lat) + 1e-14) @ lat
    folded[: min(5, targets)] = tg[: min(5, targets)]
    c = ewald_lib.Context(0, ewald_lib.FP64)
    c.set_point_engine(ewald_lib.POINTS_MESH)
    try:
        assert rel_max(c.potential_at(tg, src, q, lat.T, 1e-10),
                       oracle.potential_at(folded, src, q, lat.T, 1e-10)) < TOL_POINTS
        assert rel_max(c.potential_gradient_at(tg, src, q, lat.T, 1e-10),
                       oracle.potential_gradient_at(folded, src, q, lat.T, 1e-10)) < TOL_POINTS
    finally:
        c.close()


@pytest.mark.parametrize("n", [5, 20, 40, 90])
def test_gather_warps_by_list_length(ewald_lib, n):
    """Lists below and above the length from which the gather takes eight warps (48
    slots a tile; 3 x 3 x 3 tiles, of which each atom has a slot or more); the partials
    do not depend on it, so every shape agrees bitwise."""
    rng = np.random.default_rng(n)
    lat = np.diag([9.5, 9.0, 10.0])
    pos, q = rng.uniform(size=(n, 3)) @ lat, charges(rng, n)
    ov = dict(alpha_in=0.8, r_cut_in=4.0, k_cut_in=3.0, windowCutoff_in=12)
    c = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        results = [c.potential_force(pos, q, lat, 1e-8, **ov)]
        for warps in (2, 4, 8):
            c.set_kernel_shape({"gather_warps": warps})
            results.append(c.potential_force(pos, q, lat, 1e-8, **ov))
        for p, f in results[1:]:
            assert np.array_equal(p, results[0][0]) and np.array_equal(f, results[0][1])
    finally:
        c.close()
