"""First-order sums over the s-grid's columns: the kernels for whole grids (tiles
of rows), for long lists of columns and for short ones give the same columns.
Rings that share an origin and a spacing share the phasor tables, so only the
order of the FP32 sums differs (chunks of at most 128 terms, then compensated)."""
import ctypes

import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

TOL = 2e-6
D = 3.7


@pytest.fixture(scope="module")
def wm(tmp_path_factory):
    import os
    cwd = os.getcwd()
    os.chdir(tmp_path_factory.mktemp("run"))
    m = cw.CFDwavemaker()
    yield m
    m.cleanup()
    os.chdir(cwd)


def _load(wm, comps, nx, ny, nl, ignore=None, ramps=None):
    grid = {"bounds": (-40.0, -40.0 + D * (nx - 1), 10.0, 10.0 + D * (ny - 1)), "nx": nx, "ny": ny, "nl": nl,
            "t0": 7.5, "dt": 0.5, "stretch": (0.7, 1.5)}
    if ignore:
        grid["ignore"] = ignore
    txt = ss.write_irregular(None, comps, 45.0, extrap=2, swl=0.3, mtheta=20.0, lsgrid=grid, ramp_columns=ramps)
    assert wm.initialize_text(txt) == 0, cw.last_error()
    wm.sgrid_method(1)


def _newest(wm, nx, ny, nl):
    wm.force_update(wm.sgrid_state()[0] + 0.75)
    out = []
    for f, m in enumerate((1, nl, nl, nl)):
        a = np.zeros((nx, ny, m), np.float32)
        assert wm.lib.cfdwm_sgrid_block_export(f, 0, nx, cw._ptr(a)) == 0, cw.last_error()
        out.append(a)
    return out


@pytest.mark.parametrize("nl,nfreq,ndir,individual", [(16, 33, 1, False), (16, 20, 4, True), (5, 12, 3, False),
                                                      (21, 9, 5, False)])
def test_whole_grids_lists_and_short_lists(wm, nl, nfreq, ndir, individual):
    comps = ss.irregular_components(4.0, 9.0, 2.0, nfreq, 0.4, 1.8, 45.0, 3, ndir=ndir, spreading_s=6.0)
    n = nfreq * ndir
    rng = np.random.default_rng(n)
    ramps = [np.full(n, 4.0), rng.uniform(0, 3, n), np.full(n, 500.0)] if individual else None
    big, small = (200, 230), (11, 21)
    _load(wm, comps, *big, nl, ramps=ramps)
    ref = _newest(wm, *big, nl)
    top = [np.max(np.abs(a)) for a in ref]
    # without its first row of columns: a long list
    _load(wm, comps, *big, nl, ignore=(-40.5, -39.5, 0.0, 5000.0), ramps=ramps)
    got = _newest(wm, *big, nl)
    for a, b, t in zip(got, ref, top):
        assert np.max(np.abs(a[1:] - b[1:])) <= TOL * t
    # narrow: tiles would leave most lanes empty
    _load(wm, comps, 1500, 33, nl, ramps=ramps)
    got = _newest(wm, 1500, 33, nl)
    for a, b, t in zip(got, ref, top):
        assert np.max(np.abs(a[:200] - b[:, :33])) <= TOL * t
    # the corner: a short list
    _load(wm, comps, *small, nl, ramps=ramps)
    got = _newest(wm, *small, nl)
    for a, b, t in zip(got, ref, top):
        assert np.max(np.abs(a - b[:11, :21])) <= TOL * t


def test_first_order_channels(wm):
    torch = pytest.importorskip("torch")
    nl = 16
    comps = ss.irregular_components(4.0, 9.0, 2.0, 20, 0.4, 1.8, 45.0, 3, ndir=4, spreading_s=6.0)
    lib = wm.lib
    out = {}
    for nx, ny in ((200, 230), (1500, 30), (11, 21)):
        _load(wm, comps, nx, ny, nl)
        assert lib.cfdwm_surrogate_create(nl, 1) == 0
        feat = torch.zeros(8 * nl, nx + 8, ny + 8, device="cuda")
        base, eta = torch.zeros(3, nx, ny, nl, device="cuda"), torch.zeros(nx, ny, device="cuda")
        assert lib.cfdwm_surrogate_features(ctypes.c_double(9.25), cw._ptr(feat), cw._ptr(base), cw._ptr(eta)) == 0
        out[nx, ny] = [a.cpu().numpy() for a in (feat, base, eta)]
    ref = out[200, 230]
    for (nx, ny), got in out.items():
        i, j = min(nx, 200), min(ny, 230)
        for q in range(8):
            d = got[0][q::8, :i + 8, :j + 8] - ref[0][q::8, :i + 8, :j + 8]
            assert np.max(np.abs(d)) <= TOL * np.max(np.abs(ref[0][q::8]))
        for f in range(3):
            assert np.max(np.abs(got[1][f, :i, :j] - ref[1][f, :i, :j])) <= TOL * np.max(np.abs(ref[1][f]))
        assert np.max(np.abs(got[2][:i, :j] - ref[2][:i, :j])) <= TOL * np.max(np.abs(ref[2]))


@pytest.mark.parametrize("pressure", [False, True])
@pytest.mark.parametrize("nfreq,ndir", [(1, 1), (31, 1), (257, 1), (43, 3)])
def test_potential_form(wm, monkeypatch, nfreq, ndir, pressure):
    """One ramp for all components: the potential form's three full blocks per
    depth function against the plain pair sums and against the triangular blocks.
    Each tensor-core form is within 1e-5 of the second-order sums, a few per cent
    of the fields."""
    comps = ss.irregular_components(4.0, 9.0, 2.0, nfreq, 0.4, 1.8, 45.0, 3, ndir=ndir, spreading_s=6.0)
    nx, ny, nl = 13, 17, 10
    got = {}
    for form in ("plain", "potential", "triangular"):
        if form == "triangular":
            monkeypatch.setenv("CFDWM_DF_TWO_ACC", "1")
        grid = {"bounds": (-40.0, -40.0 + D * (nx - 1), 10.0, 10.0 + D * (ny - 1)), "nx": nx, "ny": ny, "nl": nl,
                "t0": 7.5, "dt": 0.5, "stretch": (0.7, 1.5)}
        txt = ss.write_irregular(None, comps, 45.0, extrap=2, swl=0.3, mtheta=20.0, lsgrid=grid)
        assert wm.initialize_text(txt) == 0, cw.last_error()
        wm.sgrid_method(0 if form == "plain" else 1)
        if pressure:
            wm.sgrid_pressure(True)
        got[form] = _newest(wm, nx, ny, nl)
        if pressure:
            p = np.zeros((nx, ny, nl), np.float32)
            assert wm.lib.cfdwm_sgrid_block_export(4, 0, nx, cw._ptr(p)) == 0, cw.last_error()
            got[form].append(p)
    for form in ("potential", "triangular"):
        for f, (a, b) in enumerate(zip(got[form], got["plain"])):
            assert np.max(np.abs(a - b)) <= 2e-6 * np.max(np.abs(b)), (form, f, np.max(np.abs(a - b)) / np.max(np.abs(b)))
