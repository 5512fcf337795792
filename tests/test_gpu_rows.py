"""The API rows that the evaluation's last kernel writes into the caller's own
arrays, and the s-grid query's cooperative gather, at the sizes where they can
go wrong: odd batches, grids of one column or level, outputs that alias inputs
or one another, overlap them or are not aligned."""
import os

import numpy as np
import pytest

from conftest import load_golden

import cfdwavemaker_gb300 as cw
import oracle
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

TOL = 1e-5      # FP32 arithmetic, normwise (the bar of test_gpu_parity.py)


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


@pytest.mark.parametrize("pressure", [False, True])
@pytest.mark.parametrize("nx,ny,nl", [(9, 7, 6), (5, 1, 4), (1, 6, 3), (4, 3, 2), (33, 2, 5)])
def test_sgrid_query_shapes(wm, nx, ny, nl, pressure):
    comps = ss.irregular_components(3.0, 9.0, 2.0, 12, 0.4, 1.8, 30.0, 5, ndir=3, spreading_s=6.0)
    grid = {"bounds": (0.0, 60.0, -20.0, 20.0), "nx": nx, "ny": ny, "nl": nl, "t0": 4.0, "dt": 0.4,
            "stretch": (0.7, 1.5)}
    txt = ss.write_irregular(None, comps, 30.0, extrap=2, lsgrid=grid, ramps={"time_rampup": (0.0, 9.0)})
    assert wm.initialize_text(txt) == 0, cw.last_error()
    wm.sgrid_pressure(pressure)
    wm.force_update(4.6)
    cfg = oracle.waveinput.read_text(txt)
    og = oracle.Sgrid(cfg, oracle.Sea(cfg), pressure=pressure)
    og.force_update(4.6)
    rng = np.random.default_rng(nx * 100 + nl)
    N = 257
    X, Y = rng.uniform(-3, 63, N), rng.uniform(-22, 22, N)
    Z, T = rng.uniform(-31, 2.5, N), rng.uniform(4.4, 4.8, N)
    full = og.query(X, Y, np.maximum(Z, -30.0), T) * oracle.ramp(cfg, X, Y, T)[:, None]
    scale = np.max(np.abs(full), axis=0)
    for n in (1, 31, 33, N):
        x, y, z, t, ref = X[:n], Y[:n], Z[:n], T[:n], full[:n]
        kin = wm.kinematics_batch(x, y, z, t)
        assert np.all(np.abs(kin - ref[:, :4]) <= TOL * scale[:4]), (n, nx, ny, nl)
        assert np.array_equal(wm.surface_elevation_batch(x, y, t), kin[:, 0])
        u, v, w = wm.velocity_batch(x, y, z, t)
        assert np.array_equal(np.stack([u, v, w], 1), kin[:, 1:])
        p = wm.dynamic_pressure_batch(x, y, z, t)
        if pressure:
            assert np.all(np.abs(p - ref[:, 4]) <= TOL * scale[4])
        else:
            assert not p.any()


@pytest.mark.parametrize("case", ["config1_point", "smit_spread", "fenton24", "stokes5", "sgrid_small"])
@pytest.mark.parametrize("n", [1, 127, 600])
def test_rows_in_awkward_arrays(wm, case, n):
    """u, v, w written over inputs, over one another, into overlapping and
    unaligned device arrays: the values of a call with arrays of their own."""
    import ctypes as C
    import torch
    g = load_golden(case)
    assert wm.initialize_text(str(g["waveinput"])) == 0, cw.last_error()
    rng = np.random.default_rng(n)
    t0 = 0.0 if case != "sgrid_small" else wm.sgrid_state()[0]
    host = [rng.uniform(0, 5, n), rng.uniform(-2, 2, n), rng.uniform(-3, 0.5, n), t0 + rng.uniform(0, 0.2, n)]
    lib = wm.lib
    fresh = lambda: [torch.as_tensor(a, device="cuda") for a in host]  # noqa: E731
    p = cw._ptr
    x, y, z, t = fresh()
    want = torch.empty(3, n, device="cuda", dtype=torch.float64)
    assert lib.wave_VeloXYZ_batch(p(x), p(y), p(z), p(t), n, p(want[0]), p(want[1]), p(want[2])) == 0
    assert torch.isfinite(want).all()
    # over the inputs themselves
    x, y, z, t = fresh()
    assert lib.wave_VeloXYZ_batch(p(x), p(y), p(z), p(t), n, p(z), p(t), p(x)) == 0
    assert torch.equal(torch.stack([z, t, x]), want)
    # the same array for every row: the last one stays
    x, y, z, t = fresh()
    one = torch.empty(n, device="cuda", dtype=torch.float64)
    assert lib.wave_VeloXYZ_batch(p(x), p(y), p(z), p(t), n, p(one), p(one), p(one)) == 0
    assert torch.equal(one, want[2])
    # an output that begins inside an input
    buf = torch.empty(n + 5, device="cuda", dtype=torch.float64)
    buf[:n] = fresh()[2]
    assert lib.wave_VeloXYZ_batch(p(x), p(y), p(buf), p(t), n, C.c_void_p(buf.data_ptr() + 40), None, None) == 0
    assert torch.equal(buf[5:], want[0])
    # rows that overlap: copied in row order, so the later one stays whole
    buf = torch.empty(n + 3, device="cuda", dtype=torch.float64)
    z = fresh()[2]
    assert lib.wave_VeloXYZ_batch(p(x), p(y), p(z), p(t), n, p(buf), C.c_void_p(buf.data_ptr() + 24), None) == 0
    assert torch.equal(buf[3:], want[1]) and torch.equal(buf[:min(3, n)], want[0][:3])
    # not aligned for an FP64 store
    raw = torch.zeros(8 * n + 8, device="cuda", dtype=torch.uint8)
    assert lib.wave_VeloXYZ_batch(p(x), p(y), p(z), p(t), n, None, C.c_void_p(raw.data_ptr() + 4), None) == 0
    got = np.frombuffer(raw.cpu().numpy()[4:4 + 8 * n].tobytes(), np.float64)
    assert np.array_equal(got, want[1].cpu().numpy())
    # host arrays give the same
    h = wm.velocity_batch(*host)
    assert all(np.array_equal(a, b.cpu().numpy()) for a, b in zip(h, want))
