"""The precision form's GEMM on component counts that do not fill its tiles of
256: the last column tile's columns (by 32), the K blocks past the last component
left out, and segments of one K block, in one accumulator and in two."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss
from conftest import norm_rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5          # fp16 split against the plain FP32 form (the bar of test_gpu_qform.py)


@pytest.mark.parametrize("env", [{}, {"CFDWM_QFORM_KSEG": "1"}, {"CFDWM_QFORM_TWO_ACC": "1"}, {"CFDWM_TC_PAIR": "0"}])
@pytest.mark.parametrize("nf,nd", [(31, 1), (65, 1), (43, 6), (97, 3), (128, 4)])
def test_partial_tiles(tmp_path, monkeypatch, env, nf, nd):
    torch = pytest.importorskip("torch")
    monkeypatch.chdir(tmp_path)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    comps = ss.irregular_components(6.0, 12.0, 2.0, nf, 0.25, 1.6, 100.0, 17, ndir=nd, spreading_s=10.0)
    wm = cw.CFDwavemaker()
    assert wm.initialize_text(ss.write_irregular(None, comps, 100.0, extrap=2)) == 0, cw.last_error()
    assert wm.lib.cfdwm_qform_build(1) == 0, cw.last_error()
    n = 300
    rng = np.random.default_rng(nf)
    d = [torch.tensor(rng.uniform(0, s, n), device="cuda", dtype=torch.float64) for s in (1000, 1000, 100)]
    out = [torch.zeros((n, 4), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    for m in (0, 1):
        assert wm.lib.cfdwm_qform_eval(*[cw._ptr(a) for a in d], n, m, cw._ptr(out[m])) == 0, cw.last_error()
    plain, got = (o.cpu().numpy().astype(np.float64) for o in out)
    wm.cleanup()
    for f in range(4):
        assert norm_rel_err(got[:, f], plain[:, f]) <= TOL, (f, norm_rel_err(got[:, f], plain[:, f]))
