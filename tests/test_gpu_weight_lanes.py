"""Window weights with 8 and 32 atoms to a CTA: both sides of the sizes at which the
windows change from one to the other, remainders of either, and Gaussian stencils whose
points lanes share, among them some that are wider than the grid and reach points twice.

Tolerance: 1e-10 of the largest value against the oracle, the bound of the plain form."""

import numpy as np
import pytest
from conftest import rel_max

pytestmark = pytest.mark.gpu

TOL = 1e-10


def system(n, edges):
    rng = np.random.default_rng(n)
    lat = np.diag(edges)
    lat[1, 0], lat[2, 0] = 0.4, -0.3
    q = rng.normal(0.0, 0.4, size=n)
    return rng.uniform(size=(n, 3)) @ lat, q - q.mean(), lat


@pytest.fixture(scope="module", params=["ik", "ad"])
def ctx(request, ewald_lib):
    c = ewald_lib.Context(0, ewald_lib.FP64)
    c.set_force_scheme(ewald_lib.FORCE_AD if request.param == "ad" else ewald_lib.FORCE_IK)
    yield c, request.param
    c.close()


@pytest.mark.parametrize("n", [7, 8, 9, 1183, 1184, 1185, 4735, 4736, 4737])
@pytest.mark.parametrize("window", [9, 12])
def test_atoms_per_cta(ctx, oracle, n, window):
    ctx, scheme = ctx
    pos, q, lat = system(n, (20.0, 21.0, 19.0))
    po, fo = oracle.fft_potential_force(pos, q, lat, 1e-8, alpha=0.5, r_cut=3.0, k_cut=4.2, window_cutoff=window)
    ov = dict(alpha_in=0.5, r_cut_in=3.0, k_cut_in=4.2, windowCutoff_in=window)
    p, f = ctx.potential_force(pos, q, lat, 1e-8, **ov)
    assert rel_max(p, po) < TOL
    if scheme == "ik" or window == 12:  # the oracle's forces are i k, equal to 1e-10 at 12
        assert rel_max(f, fo) < TOL
    (pb,), (fb,) = ctx.batch_potential_force([(pos, q, lat)], 1e-8, **ov)
    assert rel_max(pb, p) < 1e-12 and rel_max(fb, f) < 1e-12


# modes 2 .. 16 and windows up to 33 points: 4 to 32 points along an axis
@pytest.mark.parametrize("modes", [2, 3, 4, 5, 8, 12, 16])
@pytest.mark.parametrize("window", [2, 4, 7, 9, 13, 16])
def test_stencils_wider_than_the_grid(ewald_lib, oracle, modes, window):
    pos, q, lat = system(45, (6.0, 7.0, 6.5))
    c = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        p, f = c.potential_force(pos, q, lat, 1e-6, alpha_in=0.7, r_cut_in=4.0, k_cut_in=2.0,
                                 nModes_in=modes, windowCutoff_in=window)
    finally:
        c.close()
    po, fo = oracle.fft_potential_force(pos, q, lat, 1e-6, alpha=0.7, r_cut=4.0, k_cut=2.0,
                                        n_modes=modes, window_cutoff=window)
    assert rel_max(p, po) < TOL and rel_max(f, fo) < TOL
