"""An s-grid of more rows of columns than a launch has blocks in y: its first rows
are those of a small grid of the same origin and spacing."""
import numpy as np
import pytest

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

pytestmark = pytest.mark.gpu

TOL = 2e-6          # the same tables, another order of the FP32 sums (the bar of test_gpu_columns.py)
D, NY = 3.7, 22


@pytest.mark.parametrize("nx,nl", [(131070, 2), (131090, 2), (131090, 17), (262150, 2)])
def test_many_rows(tmp_path, monkeypatch, nx, nl):
    monkeypatch.chdir(tmp_path)
    wm = cw.CFDwavemaker()
    comps = ss.irregular_components(3.0, 9.0, 2.0, 5, 0.4, 1.8, 45.0, 3)

    def columns(rows):
        grid = {"bounds": (0.0, D * (rows - 1), 0.0, D * (NY - 1)), "nx": rows, "ny": NY, "nl": nl, "t0": 7.5, "dt": 0.5,
                "stretch": (0.7, 1.5)}
        assert wm.initialize_text(ss.write_irregular(None, comps, 45.0, extrap=2, lsgrid=grid)) == 0, cw.last_error()
        wm.sgrid_method(1)
        wm.force_update(wm.sgrid_state()[0] + 0.75)
        out = []
        for f, m in enumerate((1, nl, nl, nl)):
            a = np.zeros((16, NY, m), np.float32)
            assert wm.lib.cfdwm_sgrid_block_export(f, 0, 16, cw._ptr(a)) == 0, cw.last_error()
            out.append(a)
        return out

    ref = columns(40)
    assert ref[0].any() and ref[1].any()
    for a, b in zip(columns(nx), ref):                   # (v is zero: one direction)
        assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b))
    wm.cleanup()
