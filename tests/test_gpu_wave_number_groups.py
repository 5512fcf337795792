"""First-order sums of grid columns where many components share a wave number:
a wave of one frequency from n directions that comes together at a point, at the
seabed and at the surface, against FP64.  Whole grid, listed columns, short list."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

# RMS error over the RMS.  A chain of 128 FP32 terms in phase between two Kahan
# steps, FP32 profiles and phases good to 4e-7: 4.1e-7 measured
TOL = 4e-7
D, H, MTH = 3.9, 40.0, 20.0


@pytest.fixture(scope="module")
def wm(tmp_path_factory):
    import os
    cwd = os.getcwd()
    os.chdir(tmp_path_factory.mktemp("run"))
    m = cw.CFDwavemaker()
    yield m
    m.cleanup()
    os.chdir(cwd)


@pytest.mark.parametrize("n", [63, 64, 65, 300, 1000])
@pytest.mark.parametrize("nx,ny,ignore", [(200, 230, False), (200, 230, True), (11, 21, False)])
def test_one_frequency_many_directions(wm, n, nx, ny, ignore):
    o = np.full(n, 0.9)
    k = o * o / 9.81
    for _ in range(200):
        k = o * o / (9.81 * np.tanh(k * H))
    th = np.linspace(-1.2, 1.2, n)
    a = th + MTH * 3.1415926535897 / 180.0
    x0, t0 = 10.0 * D, 19.0                     # they meet here, at the time of the newest slot
    phase = -(k * np.cos(a) * x0 + k * np.sin(a) * x0 - o * t0)
    A = np.full(n, 1e-6)                        # (the second order is 1e-5 of the first)
    grid = {"bounds": (0.0, D * (nx - 1), 0.0, D * (ny - 1)), "nx": nx, "ny": ny, "nl": 4, "t0": 17.5, "dt": 0.5,
            "stretch": (0.7, 1.5)}
    if ignore:
        grid["ignore"] = (-0.5, 0.5, -1.0, 5000.0)          # the first row of columns
    comps = {"omega": o, "A": A, "k": k, "phase": phase, "theta": th}
    assert wm.initialize_text(ss.write_irregular(None, comps, H, extrap=2, mtheta=MTH, lsgrid=grid)) == 0
    wm.sgrid_method(1)
    wm.force_update(wm.sgrid_state()[0] + 0.75)
    assert wm.sgrid_state()[0] + 1.0 == t0
    rng = np.random.default_rng(0)
    i, j = rng.integers(1, nx, 1500), rng.integers(0, ny, 1500)
    P = np.outer(D * i, k * np.cos(a)) + np.outer(D * j, k * np.sin(a)) - o * t0 + phase
    bed = A * 9.81 * k / o / np.cosh(k * H)
    want = [np.cos(P) @ A, np.cos(P) @ (bed * np.cos(a)), np.cos(P) @ (bed * np.sin(a))]
    for f, w in enumerate(want):
        g = np.zeros((nx, ny, 1 if f == 0 else 4), np.float32)
        assert wm.lib.cfdwm_sgrid_block_export(f, 0, nx, cw._ptr(g)) == 0, cw.last_error()
        e = np.sqrt(np.mean((g[i, j, 0] - w) ** 2) / np.mean(w ** 2))
        assert e <= TOL, (f, e)
