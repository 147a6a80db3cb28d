"""The Kaiser-Bessel window of the plain form (half-widths 11 and 12, damped
modes) against the oracle's Gaussian window on twice oversampled grids.

Tolerance: the bound of the plain form, 1e-10 of the largest value.  Both windows
are converged to 1e-12 or better at these parameters, so the results differ by
far less."""

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-10


def rel_max(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.fixture(scope="module", params=["ik", "ad"])
def ctx(request, ewald_lib):
    c = ewald_lib.Context(0, ewald_lib.FP64)
    c.set_force_scheme(ewald_lib.FORCE_AD if request.param == "ad" else ewald_lib.FORCE_IK)
    yield c
    c.close()


def skew_cell(n, edges, angles, seed):
    rng = np.random.default_rng(seed)
    lat = W.triclinic_lattice(*edges, *angles) * W.ANGSTROM_TO_BOHR
    q = rng.normal(0.0, 0.4, size=n)
    return rng.uniform(size=(n, 3)) @ lat, q - q.mean(), lat


# (atoms, edges in Angstrom, angles, tol): the smallest grids (one and two tiles per
# axis, stencils that come back into their first tile), axes of unequal length, one
# CTA of atoms and a remainder, both half-widths
CELLS = [
    (2, (4.0, 4.0, 4.0), (90, 90, 90), 1e-9),
    (31, (6.0, 7.0, 9.0), (80, 95, 100), 1e-10),
    (33, (14.0, 8.0, 30.0), (75, 105, 90), 1e-9),
    (500, (40.0, 9.0, 13.0), (100, 75, 80), 1e-10),
    (1601, (24.0, 25.0, 23.0), (90, 90, 90), 1e-10),
]


@pytest.mark.parametrize("n,edges,angles,tol", CELLS)
def test_kaiser_bessel_matches_oracle(ctx, oracle, n, edges, angles, tol):
    pos, q, lat = skew_cell(n, edges, angles, n)
    po, fo = oracle.fft_potential_force(pos, q, lat, tol)
    for _ in range(3):  # direct, recorded, replayed
        pg, fg = ctx.potential_force(pos, q, lat, tol)
        assert rel_max(pg, po) < TOL
        assert rel_max(fg, fo) < TOL
    assert ctx.last_params()["window_cutoff"] in (11, 12)
    # positions outside the cell, on its faces and on grid points
    frac = np.round(pos @ np.linalg.inv(lat) * 64) / 64
    frac = np.unique(frac % 1.0, axis=0)
    pos, q = (frac - 2.0) @ lat, q[: len(frac)] - q[: len(frac)].mean()
    po, fo = oracle.fft_potential_force(pos, q, lat, tol)
    pg, fg = ctx.potential_force(pos, q, lat, tol)
    assert rel_max(pg, po) < TOL
    assert rel_max(fg, fo) < TOL


def test_refused_mode_counts_stay_refused(ewald_lib):
    """Mode counts whose doubled length has no transform (a prime factor beyond 31,
    more than 4096 points) are refused whichever window would serve them."""
    pos, q, lat = W.c1_small_cubic()
    ctx = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        for modes in (74, 2 * 2050):
            with pytest.raises(ewald_lib.EwaldError) as e:
                ctx.potential_force(pos, q, lat, 1e-10, nModes_in=modes)
            assert e.value.code == 14  # EWG_ERR_GRID_TOO_LARGE
    finally:
        ctx.close()
