"""The s-grid column sums where frequencies lie close together.  The potential
form's terms are larger than the sums there by k / |k_i - k_m|; the columns have to
be as exact as the triangular blocks make them, which a sea with individual (here
equal) ramps takes.  The first order of the two is the same, so only the second
order's rounding can differ."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

# of a field's maximum: two units in the last place of the stored FP32 values (up to
# 1.2e-7 each; the forms' sums are atomic, in no fixed order) and of the second-order
# sums, a fifth of it at most, 3e-7 of their own maximum in either form
TOL = 3e-7
NX, NY, NL = 13, 17, 10


@pytest.fixture()
def wm(tmp_path, monkeypatch):
    monkeypatch.chdir(tmp_path)
    m = cw.CFDwavemaker()
    yield m
    m.cleanup()


def _sea(kind):
    rng = np.random.default_rng(5)
    if kind == "dense":                       # long-crested, shallow
        return ss.irregular_components(1.5, 9.0, 2.0, 256, 0.4, 1.8, 12.0, 3), 12.0
    if kind == "denser":
        return ss.irregular_components(1.5, 9.0, 2.0, 1024, 0.4, 1.8, 12.0, 3), 12.0
    if kind == "crests":                      # directional, shallow
        return ss.irregular_components(1.5, 9.0, 2.0, 128, 0.4, 1.8, 20.0, 3, ndir=4, spreading_s=6.0), 20.0
    if kind == "random":                      # frequencies at random
        n, h = 300, 45.0
        o = np.sort(rng.uniform(0.4, 1.8, n))
    else:                                     # two of them this close
        n, h = 64, 45.0
        o = np.linspace(0.4, 1.8, n)
        o[31] = o[30] * (1.0 + float(kind))
    k = o * o / 9.81
    for _ in range(100):
        k = o * o / (9.81 * np.tanh(k * h))
    a = 0.4 * np.exp(-((o - 0.8) / 0.25) ** 2) / np.sqrt(n / 64.0) + 1e-4
    return {"omega": o, "A": a, "k": k, "phase": rng.uniform(0, 2 * np.pi, n), "theta": np.full(n, 0.2)}, h


def _newest(wm, comps, depth, pressure, ramps):
    grid = {"bounds": (-40.0, 20.0, 10.0, 80.0), "nx": NX, "ny": NY, "nl": NL, "t0": 17.5, "dt": 0.5,
            "stretch": (0.7, 1.5)}
    txt = ss.write_irregular(None, comps, depth, extrap=2, mtheta=20.0, lsgrid=grid, ramp_columns=ramps)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    wm.sgrid_method(1)
    if pressure:
        wm.sgrid_pressure(True)
    wm.force_update(wm.sgrid_state()[0] + 0.75)
    out = []
    for f in range(5 if pressure else 4):
        a = np.zeros((NX, NY, 1 if f == 0 else NL), np.float32)
        assert wm.lib.cfdwm_sgrid_block_export(f, 0, NX, cw._ptr(a)) == 0, cw.last_error()
        out.append(a)
    return out


@pytest.mark.parametrize("pressure", [False, True])
@pytest.mark.parametrize("kind", ["dense", "denser", "crests", "random", "1e-4", "1e-5", "1e-6", "1e-7"])
def test_close_frequencies(wm, kind, pressure):
    comps, depth = _sea(kind)
    n = len(comps["omega"])
    got = _newest(wm, comps, depth, pressure, None)
    ref = _newest(wm, comps, depth, pressure, [np.full(n, 4.0), np.zeros(n), 500.0 + np.arange(n) / n])
    for f, (a, b) in enumerate(zip(got, ref)):
        e = np.max(np.abs(a - b)) / np.max(np.abs(b))
        assert np.isfinite(b).all() and e <= TOL, (kind, f, e)


def test_no_density(wm):
    """The pressure of a sea without density is zero, and its velocities are those of
    the same sea without the pressure."""
    comps = ss.irregular_components(3.0, 9.0, 2.0, 24, 0.4, 1.8, 45.0, 3, ndir=4, spreading_s=6.0)
    grid = {"bounds": (-40.0, 20.0, 10.0, 80.0), "nx": NX, "ny": NY, "nl": NL, "t0": 17.5, "dt": 0.5,
            "stretch": (0.7, 1.5)}
    txt = ss.write_irregular(None, comps, 45.0, extrap=2, mtheta=20.0, rho=0.0, lsgrid=grid)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    wm.sgrid_method(1)
    ref = np.zeros((2, 3, NX, NY, NL), np.float32)
    p = np.ones((NX, NY, NL), np.float32)
    for on in (0, 1):
        wm.sgrid_pressure(bool(on))
        for f in range(3):
            assert wm.lib.cfdwm_sgrid_block_export(1 + f, 0, NX, cw._ptr(ref[on, f])) == 0, cw.last_error()
    assert wm.lib.cfdwm_sgrid_block_export(4, 0, NX, cw._ptr(p)) == 0, cw.last_error()
    assert not p.any()
    assert np.max(np.abs(ref[1] - ref[0])) <= TOL * np.max(np.abs(ref[0]))
