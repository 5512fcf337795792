"""Short batches (one block per point and slice of the sums) leave nothing in the
thread's workspace that the next one depends on: the same rows come back after
the workspace has grown into memory full of other values, between large batches,
on other streams and from a captured graph."""
import ctypes

import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu


@pytest.fixture()
def wm(tmp_path, monkeypatch):
    monkeypatch.chdir(tmp_path)
    m = cw.CFDwavemaker()
    comps = ss.irregular_components(4.0, 10.0, 3.3, 128, 0.3, 2.0, 50.0, 12345)
    assert m.initialize_text(ss.write_irregular(None, comps, 50.0, extrap=2, rho=1025.0, mtheta=20.0)) == 0
    yield m
    m.lib.cfdwm_set_stream(None)
    m.cleanup()


def _points(torch, n):
    rng = np.random.default_rng(1)
    host = rng.uniform(0, 500, n), rng.uniform(-100, 100, n), rng.uniform(-50, 3, n), rng.uniform(5, 60, n)
    return [torch.as_tensor(a, device="cuda") for a in host]


def test_after_other_use_of_the_memory(wm):
    torch = pytest.importorskip("torch")
    few, many = _points(torch, 7), _points(torch, 70000)
    k = torch.zeros(7, 4, device="cuda", dtype=torch.float64)
    big = torch.zeros(70000, 4, device="cuda", dtype=torch.float64)

    def short():
        k.fill_(-777.0)
        torch.cuda.synchronize()
        assert wm.lib.wave_Kinematics_batch(*map(cw._ptr, few), 7, cw._ptr(k)) == 0
        torch.cuda.synchronize()
        return k.clone()

    def scalars():
        p = [float(a[0]) for a in few]
        return [*wm.velocity(*p), wm.surface_elevation(p[0], p[1], p[3])]

    ref, ref1 = short(), scalars()
    assert (ref != -777.0).all()
    for n in (1500, 3000, 9000, 20000, 40000, 70000):
        # memory that is freed with every bit set, then a larger workspace
        junk = [torch.full((m << 18,), float("nan"), device="cuda") for m in (1, 4, 16, 64, 256)]
        for j in junk:
            j.view(torch.int32).fill_(-1)
        torch.cuda.synchronize()
        del junk, j
        torch.cuda.empty_cache()
        assert wm.lib.wave_Kinematics_batch(*map(cw._ptr, many), n, cw._ptr(big)) == 0
        assert torch.equal(short(), ref) and scalars() == ref1, n


def test_streams_and_graph(wm):
    torch = pytest.importorskip("torch")
    few = _points(torch, 13)
    out = [torch.zeros(13, 4, device="cuda", dtype=torch.float64) for _ in range(4)]
    assert wm.lib.wave_Kinematics_batch(*map(cw._ptr, few), 13, cw._ptr(out[0])) == 0
    torch.cuda.synchronize()
    for i in (1, 2):
        st = torch.cuda.Stream()
        wm.lib.cfdwm_set_stream(ctypes.c_void_p(st.cuda_stream))
        for n in (1, 5, 13):
            assert wm.lib.wave_Kinematics_batch(*map(cw._ptr, few), n, cw._ptr(out[i])) == 0
        st.synchronize()
        assert torch.equal(out[i], out[0])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        assert wm.lib.wave_Kinematics_batch(*map(cw._ptr, few), 13, cw._ptr(out[3])) == 0
    for _ in range(3):
        out[3].zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[3], out[0])


def test_allocation_free_batch_limit(wm):
    """The allocation-free entry's 32 MiB hold phasors, ramps, sums and the slices of
    18246 points of a 128-component sea, and of less than 100 more."""
    torch = pytest.importorskip("torch")
    n = 18246
    p = _points(torch, n + 100)
    out = torch.zeros(5, n + 100, device="cuda", dtype=torch.float64)
    ref = wm.irregular_fields(*(a[:n].cpu().numpy() for a in p))
    torch.cuda.synchronize()
    fields = wm.lib.cfdwm_irregular_fields_noalloc
    assert fields(*map(cw._ptr, p), n, 31, cw._ptr(out)) == 0, cw.last_error()
    got = out.flatten()[:5 * n].view(5, n).cpu().numpy()
    for q in range(5):
        assert np.max(np.abs(got[q] - ref[q])) <= 1e-6 * np.max(np.abs(ref[q]))
    assert fields(*map(cw._ptr, p), n + 100, 31, cw._ptr(out)) == -8
