"""The point API on both sides of its few-point limit, at component counts around the
16- and 32-component tiles, against the FP64 oracle: the kernels of 128 points a
block have batches of their own here (the limit is 4096 points for up to 32
components, 1943 for 33 to 64, 116 for 257 to 288)."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
import oracle
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

TOL = 1e-5      # FP32 sums, normwise per field (the bar of test_gpu_parity.py)


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
@pytest.mark.parametrize("nfreq,ndir,batches", [(1, 1, (4096, 4097, 4225)), (15, 1, (4096, 4097, 4225)),
                                                (16, 2, (4097, 4225)), (11, 3, (1940, 1945, 2177)),
                                                (257, 1, (100, 513))])
def test_both_sides_of_the_limit(wm, nfreq, ndir, batches, individual):
    depth = 35.0
    comps = ss.irregular_components(3.5, 9.0, 2.0, nfreq, 0.4, 1.9, depth, 8, ndir=ndir, spreading_s=5.0)
    n = nfreq * ndir
    rng = np.random.default_rng(n)
    ramps = [np.full(n, 4.0), rng.uniform(0, 3, n), np.full(n, 500.0)] if individual else None
    txt = ss.write_irregular(None, comps, depth, extrap=2, swl=0.4, rho=1025.0, mtheta=25.0, ramp_columns=ramps)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    cfg = oracle.waveinput.read_text(txt)
    model, sea = oracle.Model(cfg), oracle.Sea(cfg)
    m = max(batches)
    x, y = rng.uniform(-50, 300, m), rng.uniform(-80, 80, m)
    z, t = rng.uniform(-depth - 2.0, 3.0, m), rng.uniform(0.5, 30, m)
    ref, zc = model.api(x, y, z, t), np.maximum(z, -depth)
    rf = sea.fields(x, y, zc, t)
    rf = rf if rf.shape[0] == 5 else rf.T
    for b in batches:
        p = x[:b], y[:b], z[:b], t[:b]
        got = [wm.surface_elevation_batch(p[0], p[1], p[3]), *wm.velocity_batch(*p), wm.dynamic_pressure_batch(*p),
               wm.nonhydrostatic_pressure_batch(*p)]
        for q, a in enumerate(got):
            assert np.max(np.abs(a - ref[:b, q])) <= TOL * np.max(np.abs(ref[:, q])), (q, b)
        f = wm.irregular_fields(p[0], p[1], zc[:b], p[3])          # the unclamped sums
        for q in range(5):
            assert np.max(np.abs(f[q] - rf[q][:b])) <= TOL * np.max(np.abs(rf[q])), (q, b)
