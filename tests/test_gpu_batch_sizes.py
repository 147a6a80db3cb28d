"""Batches on both sides of the size up to which the real-space sum runs beside the mesh
stages, against single cells: the same sums, the last ones in the order of the batch's
common shape (1e-12 of the largest value), and bitwise the same when repeated, recorded and
replayed."""

import numpy as np
import pytest
from conftest import rel_max

import workloads as W

pytestmark = pytest.mark.gpu


def cell(n, seed):
    rng = np.random.default_rng(seed)
    edge = (10.5 * n) ** (1.0 / 3.0)
    lat = W.triclinic_lattice(edge, 1.1 * edge, 0.9 * edge, 84.0, 93.0, 98.0) * W.ANGSTROM_TO_BOHR
    k = int(np.ceil(n ** (1.0 / 3.0)))
    site = np.stack(np.meshgrid(*(np.arange(k),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    q = rng.normal(0.0, 0.4, size=n)
    return (site + rng.uniform(0.1, 0.9, size=(n, 3))) / k @ lat, q - q.mean(), lat


@pytest.mark.parametrize("sizes", [(40,), (40, 300, 77), (4000,) * 5 + (3999, 1), (6000,) * 4, (6000,) * 4 + (2,)])
@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_batch_equals_single_cells(ewald_lib, sizes, form):
    tol = 1e-9 if form == "fp64" else 1e-6
    sizes = [max(2, n) for n in sizes]
    cells = [cell(n, i) for i, n in enumerate(sizes)]
    ctx = ewald_lib.Context(0, ewald_lib.MIXED if form == "mixed" else ewald_lib.FP64)
    try:
        first = ctx.batch_potential_force(cells, tol)
        for _ in range(3):
            again = ctx.batch_potential_force(cells, tol)
            assert all(np.array_equal(a, b) for x, y in zip(first, again) for a, b in zip(x, y))
        for i in (0, len(cells) - 1):
            p, f = ctx.potential_force(*cells[i], tol)
            assert rel_max(first[0][i], p) < 1e-12 and rel_max(first[1][i], f) < 1e-12
    finally:
        ctx.close()
