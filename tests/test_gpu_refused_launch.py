"""Launches that the runtime refuses are reported by every entry point that queues them,
and the caller's arrays stay as they were.  The refusal is made on the host: a preloaded
stand-in for the runtime's launch calls returns an error and launches nothing."""

import os
import subprocess
import sys

import pytest
from conftest import PKG

pytestmark = pytest.mark.gpu

SHIM = r"""
static __thread int last;
int cudaLaunchKernel() { return last = 1; }      /* cudaErrorInvalidValue */
int cudaLaunchKernelExC() { return last = 1; }
int cudaGetLastError() { int e = last; last = 0; return e; }
"""

SCRIPT = r"""
import sys
import numpy as np
import ewald_b200 as eb
import workloads as W

kind, precision = sys.argv[1], eb.MIXED if sys.argv[2] == "mixed" else eb.FP64
pos, q, lat = W.c1_small_cubic()
ctx = eb.Context(0, precision)
ctx.set_graphs(False)
try:
    if kind == "batch":
        cells = eb.PackedCells([(pos, q, lat)] * 3)
        cells.pot[:] = 7.0
        cells.force[:] = 7.0
        try:
            cells.evaluate(ctx, 1e-8)
        finally:
            assert np.all(cells.pot == 7.0) and np.all(cells.force == 7.0), "outputs written"
    else:
        ctx.potential_force(pos, q, lat, 1e-8)
except eb.EwaldError as e:
    print("refused", e.code)
"""


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["single", "batch"])
def test_refused_launches_are_reported(ewald_lib, tmp_path, kind, form):
    src, shim = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", str(shim), str(src)], check=True)
    env = dict(os.environ, LD_PRELOAD=str(shim), PYTHONPATH=PKG)
    r = subprocess.run([sys.executable, "-c", SCRIPT, kind, form], env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["refused", "12"]  # EWG_ERR_CUDA
