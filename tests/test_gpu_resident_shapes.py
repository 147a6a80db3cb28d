"""Calls on a resident geometry whose kernel shape changes between them: each spread
finds the tile lists in order, whichever spread the geometry was binned for.

A fresh context with the same shape bins, weights and sums in the same order, so the
results agree bitwise."""

import numpy as np
import pytest

import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-7


def fresh(lib, lat, pos, q, stencil, scheme, force):
    ctx = lib.Context(0, lib.MIXED)
    try:
        ctx.set_force_scheme(scheme)
        ctx.set_kernel_shape({"stencil": stencil})
        ctx.set_lattice(lat.T)
        ctx.set_coords(pos)
        ctx.set_charges(q)
        return ctx.shift_force(TOL, len(q)) if force else (ctx.shift(TOL, len(q)), None)
    finally:
        ctx.close()


# tile lists that the tensor-core spread orders in shared memory (33), in place (1500) and
# by a kernel of its own (402 atoms that reach every tile)
@pytest.mark.parametrize("n,edge", [(1500, 32.0), (402, 14.0), (33, 14.0)])
@pytest.mark.parametrize("engines", [(1, 2, 1), (2, 1, 2)])
@pytest.mark.parametrize("scheme", ["ik", "ad"])
def test_stencil_engine_changes_on_a_resident_geometry(ewald_lib, n, edge, engines, scheme):
    rng = np.random.default_rng(n)
    lat = W.triclinic_lattice(edge, 0.9 * edge, 1.1 * edge, 85.0, 95.0, 99.0)
    s = ewald_lib.FORCE_AD if scheme == "ad" else ewald_lib.FORCE_IK
    ctx = ewald_lib.Context(0, ewald_lib.MIXED)
    ctx.set_force_scheme(s)
    try:
        for _ in range(2):  # the second geometry finds the first one's lists in the buffers
            pos = rng.uniform(size=(n, 3)) @ lat
            ctx.set_lattice(lat.T)
            ctx.set_coords(pos)
            for engine in engines:
                for force in (False, True, False):
                    q = rng.normal(0.0, 0.4, size=n)
                    q -= q.mean()
                    ctx.set_charges(q)
                    ctx.set_kernel_shape({"stencil": engine})
                    got = ctx.shift_force(TOL, n) if force else (ctx.shift(TOL, n), None)
                    want = fresh(ewald_lib, lat, pos, q, engine, s, force)
                    assert np.array_equal(got[0], want[0])
                    assert not force or np.array_equal(got[1], want[1])
    finally:
        ctx.close()
