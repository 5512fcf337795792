"""The point API's pair sums at the edges of their tiles and batches: component
counts around the 16- and 32-component tiles, batches around the few-point
limit and the blocks of 128, the phase-free pressure terms from the height
table (wave_* calls with one ramp for all components) and summed per point
(individual ramps, unclamped fields), against the FP64 oracle."""
import os

import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
import oracle
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

TOL = 1e-5      # FP32 sums, normwise per field (the bar of test_gpu_parity.py)


@pytest.fixture(scope="module")
def wm(tmp_path_factory):
    from cfdwavemaker_gb300 import build
    build.build()
    d = tmp_path_factory.mktemp("run")
    cwd = os.getcwd()
    os.chdir(d)
    m = cw.CFDwavemaker()
    yield m
    m.cleanup()
    os.chdir(cwd)


@pytest.mark.parametrize("individual", [False, True])
@pytest.mark.parametrize("nfreq,ndir", [(1, 1), (15, 1), (11, 3), (65, 2)])
def test_points_vs_oracle(wm, nfreq, ndir, individual):
    depth, swl = 35.0, 0.4
    comps = ss.irregular_components(3.5, 9.0, 2.0, nfreq, 0.4, 1.9, depth, 8, ndir=ndir, spreading_s=5.0)
    n = nfreq * ndir
    rng = np.random.default_rng(n)
    ramps = [np.full(n, 4.0), rng.uniform(0, 3, n), np.full(n, 500.0)] if individual else None
    txt = ss.write_irregular(None, comps, depth, extrap=2, swl=swl, rho=1025.0, mtheta=25.0, ramp_columns=ramps)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    cfg = oracle.waveinput.read_text(txt)
    model, sea = oracle.Model(cfg), oracle.Sea(cfg)
    for m in (513, 641, 1025):
        x, y = rng.uniform(-50, 300, m), rng.uniform(-80, 80, m)
        z, t = rng.uniform(-depth - 2.0, 3.0, m), rng.uniform(0.5, 30, m)
        ref = model.api(x, y, z, t)
        eta = wm.surface_elevation_batch(x, y, t)
        u, v, w = wm.velocity_batch(x, y, z, t)
        p, nh = wm.dynamic_pressure_batch(x, y, z, t), wm.nonhydrostatic_pressure_batch(x, y, z, t)
        for q, a in enumerate((eta, u, v, w, p, nh)):
            assert np.max(np.abs(a - ref[:, q])) <= TOL * np.max(np.abs(ref[:, q])), (q, m, n)
        # the unclamped sums of the same points, clamped here
        zc = np.maximum(z, -depth)
        f = wm.irregular_fields(x, y, zc, t)
        rf = sea.fields(x, y, zc, t)
        rf = rf if rf.shape[0] == 5 else rf.T
        for q in range(5):
            assert np.max(np.abs(f[q] - rf[q])) <= TOL * np.max(np.abs(rf[q])), (q, m, n)


@pytest.mark.parametrize("nfreq,ndir", [(1, 1), (33, 1), (43, 3), (130, 2)])
def test_few_points_match_a_large_batch(wm, nfreq, ndir):
    """The one-kernel evaluation of a short batch gives the rows that the same
    points have in a batch too large for it (each within TOL of the sums, so
    2 TOL apart at most), call after call."""
    comps = ss.irregular_components(3.5, 9.0, 2.0, nfreq, 0.4, 1.9, 35.0, 8, ndir=ndir, spreading_s=5.0)
    txt = ss.write_irregular(None, comps, 35.0, extrap=2, swl=0.4, rho=1025.0, mtheta=25.0)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    rng = np.random.default_rng(nfreq)
    m = 4200
    x, y = rng.uniform(-50, 300, m), rng.uniform(-80, 80, m)
    z, t = rng.uniform(-37.0, 3.0, m), rng.uniform(0.5, 30, m)

    def rows(k):
        p = x[:k], y[:k], z[:k], t[:k]
        return np.array([wm.surface_elevation_batch(*p[:2], p[3]), *wm.velocity_batch(*p),
                         wm.dynamic_pressure_batch(*p), wm.nonhydrostatic_pressure_batch(*p)])

    ref = rows(m)
    top = np.max(np.abs(ref), axis=1, keepdims=True)
    for k in (1, 2, 17, 130, 1, 20, 400):
        assert np.all(np.abs(rows(k) - ref[:, :k]) <= 2 * TOL * top), k


@pytest.mark.parametrize("individual", [False, True])
@pytest.mark.parametrize("nfreq,ndir", [(1, 1), (15, 1), (17, 1), (11, 3)])
def test_smit_tiles_and_batches(wm, nfreq, ndir, individual):
    """The Smit theory's sums at the edges of its 16-component tiles, in batches
    for the kernel of 128 points a block against the FP64 oracle, and in short
    ones, a block per point, against those."""
    depth = 35.0
    comps = ss.irregular_components(3.0, 9.0, 2.0, nfreq, 0.4, 1.9, depth, 8, ndir=ndir, spreading_s=5.0)
    n = nfreq * ndir
    rng = np.random.default_rng(n)
    ramps = [np.full(n, 4.0), rng.uniform(0, 3, n), np.full(n, 500.0)] if individual else None
    txt = ss.write_irregular(None, comps, depth, extrap=2, swl=0.4, rho=1025.0, mtheta=25.0, ramp_columns=ramps,
                             vertical_theory="smit")
    assert wm.initialize_text(txt) == 0, cw.last_error()
    model = oracle.Model(oracle.waveinput.read_text(txt))
    for m in (513, 1100):
        x, y = rng.uniform(-50, 300, m), rng.uniform(-80, 80, m)
        z, t = rng.uniform(-depth - 2.0, 1.0, m), rng.uniform(5.0, 30, m)
        ref = model.api(x, y, z, t)
        u, v, w = wm.velocity_batch(x, y, z, t)
        p = wm.dynamic_pressure_batch(x, y, z, t)
        for q, a in ((1, u), (2, v), (3, w), (4, p)):
            assert np.max(np.abs(a - ref[:, q])) <= TOL * np.max(np.abs(ref[:, q])), (q, m, n)
        for k in (1, 9):
            part = [*wm.velocity_batch(x[:k], y[:k], z[:k], t[:k]), wm.dynamic_pressure_batch(x[:k], y[:k], z[:k], t[:k])]
            for a, b in zip(part, (u, v, w, p)):
                assert np.max(np.abs(a - b[:k])) <= 2 * TOL * np.max(np.abs(b)), (m, n, k)
