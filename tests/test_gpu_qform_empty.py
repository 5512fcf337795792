"""The precision form of a sea without components: zeros from both methods."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env", [{}, {"CFDWM_QFORM_TWO_ACC": "1"}])
@pytest.mark.parametrize("fp16", [0, 1])
def test_no_components(tmp_path, monkeypatch, fp16, env):
    torch = pytest.importorskip("torch")
    monkeypatch.chdir(tmp_path)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    none = {k: np.zeros(0) for k in ("omega", "A", "k", "phase", "theta")}
    wm = cw.CFDwavemaker()
    assert wm.initialize_text(ss.write_irregular(None, none, 50.0, extrap=2)) == 0, cw.last_error()
    assert wm.lib.cfdwm_qform_build(fp16) == 0, cw.last_error()
    for n in (1, 300, 70000):
        d = [torch.rand(n, device="cuda", dtype=torch.float64) for _ in range(3)]
        for m in (0, 1):
            out = torch.full((n, 4), float("nan"), device="cuda")
            torch.cuda.synchronize()
            assert wm.lib.cfdwm_qform_eval(*[cw._ptr(a) for a in d], n, m, cw._ptr(out)) == 0, cw.last_error()
            torch.cuda.synchronize()
            assert not out.any()
    wm.cleanup()
