"""A batch whose cells take different windows: one Gaussian cell with rows wider than the
weights kernel's shared memory (window derivatives, five tiles of a stencil along an axis
that ends in a part tile) beside Kaiser-Bessel cells.

Tolerance: the single-cell calls take the same window and grid, so only the order of
the last sums differs: 1e-13 of the largest value, times ten."""

import math

import numpy as np
import pytest
from conftest import rel_max

import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-12
ALPHA, KC, M = 0.5, 3.7, 12


def damping(lib, pos, q, lat, ov):
    p = lib.ewald_parameters(pos, q, len(q), lat, 1e-8, **ov)
    edge = [math.pi * m / np.linalg.norm(lat[d]) for d, m in enumerate(p["n_modes"])]
    return max(math.exp(-(e * e) / (4 * p["alpha"] ** 2)) for e in edge), p["n_modes"]


@pytest.mark.parametrize("order", [(0, 1, 2), (1, 0, 2), (1, 2, 0)])
def test_wide_gaussian_rows_beside_kaiser_bessel(ewald_lib, oracle, order):
    rng = np.random.default_rng(4)
    cells = []
    for n, edges in ((60, (33.9, 9.0, 10.0)), (50, (12.0, 13.0, 14.0)), (33, (17.0, 9.0, 26.0))):
        lat = np.diag(edges)
        lat[1, 0] = 0.5
        q = rng.normal(0.0, 0.4, size=n)
        cells.append((rng.uniform(size=(n, 3)) @ lat, q - q.mean(), lat))
    ov = dict(alpha_in=ALPHA, r_cut_in=6.0, k_cut_in=KC, windowCutoff_in=M)
    d0, modes0 = damping(ewald_lib, *cells[0], ov)
    assert d0 > 2e-7 and 2 * modes0[0] % 8 != 0  # the Gaussian cell, part tiles along x
    assert all(damping(ewald_lib, *c, ov)[0] < 1e-8 for c in cells[1:])
    cells = [cells[i] for i in order]
    ctx = ewald_lib.Context(0, ewald_lib.FP64)
    ctx.set_force_scheme(ewald_lib.FORCE_AD)
    try:
        pots, forces = ctx.batch_potential_force(cells, 1e-8, **ov)
        for (pos, q, lat), pb, fb in zip(cells, pots, forces):
            ps, fs = ctx.potential_force(pos, q, lat, 1e-8, **ov)
            assert rel_max(pb, ps) < TOL and rel_max(fb, fs) < TOL
            po, fo = oracle.fft_potential_force(pos, q, lat, 1e-8, alpha=ALPHA, r_cut=6.0, k_cut=KC,
                                                window_cutoff=M)
            assert rel_max(pb, po) < 1e-10 and rel_max(fb, fo) < 1e-9
    finally:
        ctx.close()
