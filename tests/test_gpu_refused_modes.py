"""Mode counts that no transform serves are refused before any work that grows with them."""

import time

import pytest

import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_huge_mode_counts_are_refused_at_once(ewald_lib, form):
    pos, q, lat = W.c1_small_cubic()
    ctx = ewald_lib.Context(0, ewald_lib.MIXED if form == "mixed" else ewald_lib.FP64)
    try:
        ctx.potential_force(pos, q, lat, 1e-7)
        begin = time.perf_counter()
        with pytest.raises(ewald_lib.EwaldError) as e:  # 1e9 + 2 points an axis, a part tile at its end
            ctx.potential_force(pos, q, lat, 1e-7, nModes_in=500000001)
        assert e.value.code == 14  # EWG_ERR_GRID_TOO_LARGE
        assert time.perf_counter() - begin < 1.0
    finally:
        ctx.close()
