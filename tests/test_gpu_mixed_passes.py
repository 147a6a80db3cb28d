"""The mixed form's transform passes at lengths of the runtime radix schedule, in CTAs of
64, 128 and 256 threads, and at a compile-time length, against the plain form with the
same window and modes: the mixed form's bound, 1e-6 in the root mean square."""

import math

import numpy as np
import pytest
from conftest import rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modes", [15, 30, 50, 70, 90])
@pytest.mark.parametrize("batched", [False, True])
def test_mixed_passes_match_the_plain_form(ewald_lib, modes, batched):
    rng = np.random.default_rng(modes)
    k_cut = 2.0
    edge = 2 * math.pi / k_cut * (modes // 2 - 1.5)
    lat = np.diag([edge, edge, edge])
    n = 500
    site = np.stack(np.meshgrid(*(np.arange(8),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (site + rng.uniform(0.15, 0.85, size=(n, 3))) / 8 @ lat
    q = rng.normal(0.0, 0.4, size=n)
    q -= q.mean()
    ov = dict(alpha_in=0.6, r_cut_in=5.0, k_cut_in=k_cut, windowCutoff_in=6, nModes_in=modes)
    out = {}
    for form in (ewald_lib.FP64, ewald_lib.MIXED):
        ctx = ewald_lib.Context(0, form)
        try:
            if batched:
                p, f = ctx.batch_potential_force([(pos, q, lat)] * 3, 1e-7, **ov)
                out[form] = np.concatenate(p), np.concatenate(f)
            else:
                out[form] = ctx.potential_force(pos, q, lat, 1e-7, **ov)
        finally:
            ctx.close()
    for plain, mixed in zip(out[ewald_lib.FP64], out[ewald_lib.MIXED]):
        assert rel_rms(mixed, plain) < 1e-6
