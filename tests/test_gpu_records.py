"""wave_Kinematics records written over the call's own inputs (x, y, z, t in the
quarters of the record array, whole or in part) and to an address that is not
aligned for an FP64 store: the records of a call with arrays of their own."""
import ctypes

import numpy as np
import pytest
from conftest import load_golden

import cfdwavemaker_gb300 as cw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wm(tmp_path_factory):
    import os
    cwd = os.getcwd()
    os.chdir(tmp_path_factory.mktemp("run"))
    m = cw.CFDwavemaker()
    yield m
    m.cleanup()
    os.chdir(cwd)


@pytest.mark.parametrize("case", ["config1_point", "smit_spread", "fenton24", "sgrid_small"])
@pytest.mark.parametrize("n", [1, 2, 127, 600, 5001])
def test_records_over_the_inputs(wm, case, n):
    torch = pytest.importorskip("torch")
    assert wm.initialize_text(str(load_golden(case)["waveinput"])) == 0, cw.last_error()
    rng = np.random.default_rng(n)
    t0 = 0.0 if case != "sgrid_small" else wm.sgrid_state()[0]
    host = np.stack([rng.uniform(0, 5, n), rng.uniform(-2, 2, n), rng.uniform(-3, 0.5, n),
                     t0 + rng.uniform(0, 0.2, n)])
    call, p = wm.lib.wave_Kinematics_batch, cw._ptr
    ins = torch.as_tensor(host, device="cuda")
    want = torch.full((n, 4), -777.0, device="cuda", dtype=torch.float64)
    assert call(*map(p, ins), n, p(want)) == 0, cw.last_error()
    torch.cuda.synchronize()
    assert not (want == -777.0).any()
    # the inputs are the quarters of the output
    ins = torch.as_tensor(host, device="cuda")
    assert call(*map(p, ins), n, p(ins)) == 0
    torch.cuda.synchronize()
    assert torch.equal(ins.view(n, 4), want)
    # the output begins inside the last input
    buf = torch.zeros(8 * n, device="cuda", dtype=torch.float64)
    buf[:4 * n] = torch.as_tensor(host, device="cuda").flatten()
    at = 4 * n - (n + 1) // 2
    assert call(*(p(buf[q * n:]) for q in range(4)), n, p(buf[at:])) == 0
    torch.cuda.synchronize()
    assert torch.equal(buf[at:at + 4 * n].view(n, 4), want)
    # not aligned
    ins = torch.as_tensor(host, device="cuda")
    raw = torch.zeros(32 * n + 8, device="cuda", dtype=torch.uint8)
    assert call(*map(p, ins), n, ctypes.c_void_p(raw.data_ptr() + 4)) == 0
    torch.cuda.synchronize()
    got = np.frombuffer(raw.cpu().numpy()[4:4 + 32 * n].tobytes(), np.float64).reshape(n, 4)
    assert np.array_equal(got, want.cpu().numpy())
    # host arrays
    over = host.copy()
    assert call(*map(p, over), n, p(over)) == 0
    assert np.array_equal(over.reshape(n, 4), want.cpu().numpy())
