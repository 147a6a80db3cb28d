"""Charges that fill a small part of their cell: most mesh tiles hold no atom and a few
hold most of them, so tile lists run from none to all the atoms.

Tolerance: 1e-10 of the largest value against the oracle, the bound of the plain form;
calls on a resident geometry repeat the first call's sums in the same order: bitwise."""

import numpy as np
import pytest
from conftest import rel_max, rel_rms

import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-10


def ball(n, fill, seed):
    """n charges, one to each of the nearest sites of a cubic lattice around the cell's
    centre, jittered, in the order of a random permutation."""
    rng = np.random.default_rng(seed)
    lat = W.triclinic_lattice(30.0, 31.0, 29.0, 88.0, 93.0, 97.0)
    d = (fill * 30.0**3 / n) ** (1.0 / 3.0)
    k = int(np.ceil((3.0 * n / (4.0 * np.pi)) ** (1.0 / 3.0))) + 1
    g = np.stack(np.meshgrid(*(np.arange(-k, k + 1),) * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g[np.argsort((g**2).sum(1), kind="stable")][:n]
    pos = (g + rng.uniform(-0.25, 0.25, size=(n, 3))) * d + lat.sum(0) / 2
    q = rng.normal(0.0, 0.4, size=n)
    return pos[rng.permutation(n)], q - q.mean(), lat


# the lists' edges: 128 entries in shared memory, one or more windows of 16,384 atoms
@pytest.mark.parametrize("n,fill", [(128, 0.01), (129, 0.01), (700, 0.02), (3000, 0.05), (17000, 0.05)])
@pytest.mark.parametrize("scheme", ["ik", "ad"])
def test_cluster_matches_oracle_and_repeats(ewald_lib, oracle, n, fill, scheme):
    pos, q, lat = ball(n, fill, n)
    ov = dict(alpha=0.35, r_cut=2.5, k_cut=2.4, window_cutoff=12)
    po, fo = oracle.fft_potential_force(pos, q, lat, 1e-8, **ov)
    ctx = ewald_lib.Context(0, ewald_lib.FP64)
    try:
        ctx.set_force_scheme(ewald_lib.FORCE_AD if scheme == "ad" else ewald_lib.FORCE_IK)
        gpu = dict(alpha_in=0.35, r_cut_in=2.5, k_cut_in=2.4, windowCutoff_in=12)
        for _ in range(2):
            pg, fg = ctx.potential_force(pos, q, lat, 1e-8, **gpu)
            assert rel_max(pg, po) < TOL and rel_max(fg, fo) < TOL
        (p2,), (f2,) = ctx.batch_potential_force([(pos, q, lat)], 1e-8, **gpu)
        assert rel_max(p2, pg) < 1e-12 and rel_max(f2, fg) < 1e-12
        ctx.set_lattice(lat.T)
        ctx.set_coords(pos)
        ctx.set_charges(q)
        first = ctx.shift_force(1e-9, n)
        for _ in range(2):
            again = ctx.shift_force(1e-9, n)
            assert np.array_equal(again[0], first[0]) and np.array_equal(again[1], first[1])
    finally:
        ctx.close()


def test_cluster_mixed_form(ewald_lib):
    """The mixed form's spread orders its lists in the same way: both its engines within the
    form's bound of the plain one with the same window, 1e-6 in the root mean square."""
    pos, q, lat = ball(3000, 0.05, 1)
    gpu = dict(alpha_in=0.35, r_cut_in=2.5, k_cut_in=2.2, windowCutoff_in=9)
    ref = ewald_lib.Context(0, ewald_lib.FP64)
    p0, f0 = ref.potential_force(pos, q, lat, 1e-7, **gpu)
    ref.close()
    ctx = ewald_lib.Context(0, ewald_lib.MIXED)
    try:
        for stencil in (1, 2):
            ctx.set_kernel_shape({"stencil": stencil})
            p, f = ctx.potential_force(pos, q, lat, 1e-7, **gpu)
            assert rel_rms(p, p0) < 1e-6 and rel_rms(f, f0) < 1e-6
    finally:
        ctx.close()
