"""One context per host thread: transform kernels of one length launched with different
shared-memory sizes at the same time (the z pass holds the modes, more of them under
the Kaiser-Bessel window than under the Gaussian at the same 336 points).

The results do not depend on what other threads do: bitwise those of serial calls."""

import math
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LZ = 60.0


def column(seed):
    rng = np.random.default_rng(seed)
    lat = np.diag([3.0, 3.2, LZ])
    z = (np.arange(40) + rng.uniform(0.2, 0.8, size=40)) / 40
    q = rng.normal(0.0, 0.4, size=40)
    return np.column_stack([rng.uniform(size=(40, 2)), z]) @ lat, q - q.mean(), lat


def overrides(modes, window):
    return dict(alpha_in=1.2, r_cut_in=5.0, k_cut_in=2 * math.pi * (modes / 2 - 1.5) / LZ, windowCutoff_in=window)


@pytest.mark.parametrize("batched", [False, True])
def test_threads_share_a_transform_length(ewald_lib, batched):
    jobs = [(column(1), overrides(252, 12)), (column(2), overrides(168, 6))]

    def call(ctx, job):
        (pos, q, lat), ov = job
        if not batched:
            return ctx.potential_force(pos, q, lat, 1e-8, **ov)
        p, f = ctx.batch_potential_force([(pos, q, lat)], 1e-8, **ov)
        return p[0], f[0]

    want, bad = [], []
    for job, modes in zip(jobs, (252, 168)):
        ctx = ewald_lib.Context(0, ewald_lib.FP64)
        ctx.set_graphs(False)
        want.append(call(ctx, job))
        ctx.close()
        p = ewald_lib.ewald_parameters(*job[0][:2], 40, job[0][2], 1e-8, **job[1])
        assert p["n_modes"][2] == modes

    def work(i):
        try:
            ctx = ewald_lib.Context(0, ewald_lib.FP64)
            ctx.set_graphs(False)
            for _ in range(1000):
                p, f = call(ctx, jobs[i % 2])
                if not (np.array_equal(p, want[i % 2][0]) and np.array_equal(f, want[i % 2][1])):
                    bad.append((i, "other values"))
                    break
            ctx.close()
        except Exception as e:
            bad.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
