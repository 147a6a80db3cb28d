"""The register-radix FP64 transform passes at every length they exist for,
against the oracle, and a batch that mixes their length classes against single
cells.

Tolerance: the bound of the plain form, 1e-10 of the largest value; the window
and the modes are the oracle's, so only rounding (1e-15 per transform) is left."""

import math

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-10
# every length the passes exist for: two radices of at most 24
LENGTHS = [16, 24, 32, 40, 48, 56, 64, 72, 80, 96, 112, 120, 128, 144, 160, 168, 192, 200, 216, 224,
           240, 256, 280, 288, 320, 336, 360, 384, 400, 432, 480, 576]


def rel_max(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


def skew_cell(n, edges, angles, seed):
    rng = np.random.default_rng(seed)
    lat = W.triclinic_lattice(*edges, *angles) * W.ANGSTROM_TO_BOHR
    q = rng.normal(0.0, 0.4, size=n)
    return rng.uniform(size=(n, 3)) @ lat, q - q.mean(), lat


@pytest.mark.parametrize("n", LENGTHS)
def test_pass_lengths_match_oracle(ewald_lib, oracle, n):
    """One axis of every pass length (Gaussian window, n = 2 modes), each of the
    three axes in turn; the other two stay short."""
    alpha, kc, m = 0.8, 3.0, 6
    # modes: next fast length of 2 (ceil(kc L / 2 pi) + 1); n / 2 is one
    highest = n // 4 - 1
    L = 2 * math.pi / kc * (highest - 0.5) if highest > 1 else 2 * math.pi / kc * 0.9
    short = 2 * math.pi / kc * 4.5
    rng = np.random.default_rng(n)
    ctx = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        for axis in range(3):
            edges = [short] * 3
            edges[axis] = L
            lat = np.diag(edges)
            lat[2, 0] = 0.3 * edges[2] if axis != 2 else 0.0  # skew where it keeps the lengths
            pos = rng.uniform(size=(40, 3)) @ lat
            q = rng.normal(size=40)
            q -= q.mean()
            ov = dict(alpha=alpha, r_cut=4.0, k_cut=kc, window_cutoff=m)
            po, fo = oracle.fft_potential_force(pos, q, lat, 1e-8, **ov)
            pg, fg = ctx.potential_force(pos, q, lat, 1e-8, alpha_in=alpha, r_cut_in=4.0, k_cut_in=kc,
                                         windowCutoff_in=m)
            assert rel_max(pg, po) < TOL
            assert rel_max(fg, fo) < TOL
            pots = ctx.potential_force(pos, q, lat, 1e-8, want_force=False, alpha_in=alpha, r_cut_in=4.0,
                                       k_cut_in=kc, windowCutoff_in=m)
            assert rel_max(pots, po) < TOL
    finally:
        ctx.close()


def test_batch_of_many_lengths_equals_single_cells(ewald_lib):
    """Cells of several length classes in one batch: bitwise the results of one call
    per cell."""
    edges = [(4, 5, 6), (9, 30, 12), (70, 8, 9), (18, 22, 26), (8, 8, 120), (35, 36, 37)]
    cells = [skew_cell(40 + 13 * i, e, (85, 95, 100), i) for i, e in enumerate(edges)]
    ctx = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        for scheme in (ewald_lib.FORCE_IK, ewald_lib.FORCE_AD):
            ctx.set_force_scheme(scheme)
            for tol in (1e-10, 1e-9):
                pots, forces = ctx.batch_potential_force(cells, tol)
                for (pos, q, lat), pb, fb in zip(cells, pots, forces):
                    ps, fs = ctx.potential_force(pos, q, lat, tol)
                    assert np.array_equal(ps, pb) and np.array_equal(fs, fb)
    finally:
        ctx.close()
