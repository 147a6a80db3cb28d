"""The Kaiser-Bessel window's own error, against the same sums with a Gaussian of
half-width 20 (converged), is no larger than the error of the Gaussian that it stands
in for: same half-width, same modes, on the twice oversampled grid.

The Gaussian's error does not depend on how far the outermost modes are damped (to 10%
between 2e-7 and 1e-10 from 24 modes on), so it is taken just above the damping of 2e-7 from
which the plain form keeps the Gaussian: a factor of 1.15 for that."""

import math

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

N = 1500
FACTOR = 1.15


def system(edges):
    rng = np.random.default_rng(7)
    site = np.stack(np.meshgrid(*(np.arange(12),) * 3, indexing="ij"), -1).reshape(-1, 3)
    frac = (site[rng.permutation(1728)[:N]] + rng.uniform(0.1, 0.9, size=(N, 3))) / 12
    q = rng.normal(0.0, 0.4, size=N)
    lat = np.diag(edges)
    lat[1, 0], lat[2, 1] = 3.0, -2.0
    return frac @ lat, q - q.mean(), lat


def errors(ctx, modes, damping, window, edges):
    """Errors of potential and force at half-width `window` with every axis's outermost
    modes damped to `damping` or less (the longest axis to it)."""
    pos, q, lat = system(edges)
    edge = math.pi * modes / np.max(np.linalg.norm(lat, axis=1))
    ov = dict(alpha_in=edge / (2.0 * math.sqrt(-math.log(damping))), r_cut_in=3.0, k_cut_in=edge,
              nModes_in=modes)
    want = ctx.potential_force(pos, q, lat, 1e-10, windowCutoff_in=20, **ov)
    got = ctx.potential_force(pos, q, lat, 1e-10, windowCutoff_in=window, **ov)
    return [np.linalg.norm(g - w) / np.linalg.norm(w) for g, w in zip(got, want)]


# three axes at the same damping; one, and two, that decide
@pytest.mark.parametrize("edges", [(40.0, 40.0, 40.0), (29.0, 40.0, 30.0), (40.0, 27.0, 39.5)])
@pytest.mark.parametrize("scheme", ["ik", "ad"])
@pytest.mark.parametrize("window", [11, 12])
@pytest.mark.parametrize("modes", [24, 40, 50, 100, 125, 135, 150, 160])
def test_error_no_larger_than_the_gaussians(ewald_lib, edges, scheme, window, modes):
    ctx = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        ctx.set_force_scheme(ewald_lib.FORCE_AD if scheme == "ad" else ewald_lib.FORCE_IK)
        gauss = errors(ctx, modes, 2.2e-7, window, edges)
        for damping in (1.9e-7, 9e-8, 3e-8, 1e-8, 3e-9, 1e-9, 1e-11):
            kaiser = errors(ctx, modes, damping, window, edges)
            assert kaiser[0] <= FACTOR * gauss[0], (damping, kaiser, gauss)
            assert kaiser[1] <= FACTOR * gauss[1], (damping, kaiser, gauss)
    finally:
        ctx.close()
