"""Kernel attributes (dynamic shared memory above the default) are set for the device a launch goes to, not
once per process.  One device is enough to see it: after cudaDeviceReset, in a process of its own, the
device is as new, and a context made then must step like the first."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, "tests")
from conftest import load_package
wt = load_package()
rt = ctypes.CDLL("libcudart.so.12")


def solve(prec, form, eps, n):
    ctx = wt.Context(0)
    g = wt.Mesh.uniform_hex(ctx, n, 2, outer_tag=7, warp_A=0.05, precision=prec)
    if form is not None:
        g.set_fp32_form(form)
    c, ws = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, wt.workloads.adm_params(3)), wt.make_wave3d_workspace(g)
    x = np.linspace(0.0, 1.0, g.nn).astype(np.float32 if prec else np.float64)
    P, Q, E = np.sin(9 * x), np.cos(7 * x), np.zeros(2)
    wt.evolve_curved_host(P, Q, c, ws, 1e-4, 1, 2, eps, wt.make_bc3d([2] * 6), True, E)
    for h in (ws, c, g, ctx):
        h.close()
    return P, Q, E


cases = [(0, None, 0.0, 8), (0, None, 0.1, 8), (1, None, 0.0, 8), (1, wt.FP32_CUDA_CORES, 0.0, 8), (1, wt.FP32_BF16X3, 0.0, 8),
         (0, None, 0.1, 7)]
first = [solve(*c) for c in cases]
assert rt.cudaDeviceReset() == 0
for c, a in zip(cases, first):
    assert all(np.array_equal(x, y) for x, y in zip(a, solve(*c))), c
print("same")
"""


def test_attributes_after_a_device_reset(ctx):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, CUDA_MODULE_LOADING="LAZY"))
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout + r.stderr
