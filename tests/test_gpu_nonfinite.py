"""Positions that are not numbers go through every index that is made of a position, as the
first box and grid point, and come out as results that are not numbers; the context's next
call is as good as a fresh one's."""

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu


def system(n, edge):
    rng = np.random.default_rng(n)
    lat = W.triclinic_lattice(edge, 1.1 * edge, 0.95 * edge, 85.0, 94.0, 99.0)
    q = rng.normal(0.0, 0.4, size=n)
    return rng.uniform(size=(n, 3)) @ lat, q - q.mean(), lat


# one CTA's box sort and the one of several; a cell narrower than the cutoff
@pytest.mark.parametrize("n,edge", [(40, 8.0), (600, 24.0), (2500, 38.0)])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("form,tol", [("fp64", 1e-10), ("fp64", 1e-7), ("mixed", 1e-7)])
@pytest.mark.parametrize("scheme", ["ik", "ad"])
def test_positions_that_are_not_numbers(ewald_lib, n, edge, value, form, tol, scheme):
    pos, q, lat = system(n, edge)
    bad = pos.copy()
    bad[n // 2, 1] = value
    ctx = ewald_lib.Context(0, ewald_lib.MIXED if form == "mixed" else ewald_lib.FP64)
    ctx.set_force_scheme(ewald_lib.FORCE_AD if scheme == "ad" else ewald_lib.FORCE_IK)
    try:
        want = ctx.potential_force(pos, q, lat, tol)
        p, f = ctx.potential_force(bad, q, lat, tol)
        assert np.isnan(p).any() and np.isnan(f).any()
        ctx.batch_potential_force([(pos, q, lat), (bad, q, lat)], tol)
        ctx.potential_force_stress(bad, q, lat, tol)
        ctx.set_lattice(lat.T)
        ctx.set_coords(bad)
        ctx.set_charges(q)
        assert np.isnan(ctx.shift(tol, n)).any()
        if form == "fp64":
            ctx.set_point_engine(ewald_lib.POINTS_MESH)
            for blur in (None, np.full(n, 0.5)):
                assert np.isnan(ctx.potential_at(bad, pos, q, lat.T, tol, blur=blur)).any()
        again = ctx.potential_force(pos, q, lat, tol)
        assert np.array_equal(again[0], want[0]) and np.array_equal(again[1], want[1])
    finally:
        ctx.close()
