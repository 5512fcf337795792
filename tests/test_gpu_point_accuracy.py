"""Accuracy of the point API's vertical velocity near the seabed, where
w = sum q sinh(k (z + h)) ... is what is left of two nearly equal exponentials:
one point at a time, short batches and a batch for the per-thread kernels."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
import oracle
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

# RMS error of w over its maximum.  FP32 profiles e1 (1 - e2), e2 = exp(-2 k (z + h)),
# at the FP32 height z: 2.0e-7 (128 components, 50 m); E - Y, Y = exp(-k (z + 2 h)): 3.1e-7
TOL = 2.0e-7


@pytest.fixture(scope="module")
def wm(tmp_path_factory):
    import os
    cwd = os.getcwd()
    os.chdir(tmp_path_factory.mktemp("run"))
    m = cw.CFDwavemaker()
    yield m
    m.cleanup()
    os.chdir(cwd)


@pytest.mark.parametrize("individual", [False, True])
def test_vertical_velocity_near_the_bed(wm, individual):
    depth, n = 50.0, 128
    comps = ss.irregular_components(4.0, 10.0, 3.3, n, 0.3, 2.0, depth, 12345)
    rng = np.random.default_rng(3)
    ramps = [np.full(n, 4.0), rng.uniform(0, 3, n), np.full(n, 500.0)] if individual else None
    txt = ss.write_irregular(None, comps, depth, extrap=2, rho=1025.0, mtheta=20.0, ramp_columns=ramps)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    m = 300
    x, y = rng.uniform(0, 500, m), rng.uniform(-100, 100, m)
    z, t = rng.uniform(-depth, -depth + 3.0, m), rng.uniform(10, 60, m)
    ref = oracle.Model(oracle.waveinput.read_text(txt)).api(x, y, z, t)[:, 3]
    top = np.max(np.abs(ref))
    one = np.array([wm.velocity(*p)[2] for p in zip(x, y, z, t)])
    reps = 17                                    # 5100 points: the kernels of 128 points a block
    got = {"one by one": one, "short batch": wm.velocity_batch(x, y, z, t)[2],
           "batch": wm.velocity_batch(*(np.tile(a, reps) for a in (x, y, z, t)))[2][:m]}
    for what, w in got.items():
        e = np.sqrt(np.mean((w - ref) ** 2)) / top
        assert e <= TOL, (what, e)
