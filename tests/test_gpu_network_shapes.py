"""The learned update's network at the edges of its kernels' tiles: planes
smaller than a tile, one more and one less than whole tiles, several images,
level counts whose channels are not whole groups of 16, need one or several
blocks of the weight gradient, or fill the output's 64; planes that take the
wide tiles."""
import ctypes

import numpy as np
import pytest
from conftest import norm_rel_err

import cfdwavemaker_gb300 as cw
from oracle import surrogate_ref as sr

pytestmark = pytest.mark.gpu

TOL_NET, TOL_GRAD = 1e-5, 1e-4          # the bars of test_gpu_surrogate.py


@pytest.mark.parametrize("nl,b,h,w", [(1, 1, 9, 9), (2, 3, 10, 23), (3, 2, 16, 15), (5, 1, 17, 38), (6, 2, 25, 24),
                                      (10, 1, 24, 64), (11, 1, 31, 22), (16, 2, 22, 37), (21, 1, 18, 30),
                                      (2, 2, 250, 62), (11, 2, 247, 61)])
def test_network_and_gradient(nl, b, h, w):
    torch = pytest.importorskip("torch")
    lib = cw.load()
    assert lib.cfdwm_surrogate_create(nl, 3) == 0
    ch, offw, offb, n = sr.layout(nl)
    rng = np.random.default_rng(100 * nl + h)
    prm = np.zeros(n, np.float32)
    for l in range(4):
        k = ch[l + 1] * ch[l] * 9
        prm[offw[l]:offw[l] + k] = rng.normal(size=k) * np.sqrt(2.0 / (9 * ch[l]))
        prm[offb[l]:offb[l] + ch[l + 1]] = 0.1 * rng.normal(size=ch[l + 1])
    assert lib.cfdwm_surrogate_set_params(cw._ptr(prm), n) == 0
    x = rng.normal(size=(b, ch[0], h, w)).astype(np.float32)
    t = (0.5 * rng.normal(size=(b, ch[4], h - 8, w - 8))).astype(np.float32)
    dx, dt = torch.as_tensor(x, device="cuda"), torch.as_tensor(t, device="cuda")
    dy = torch.zeros(b, ch[4], h - 8, w - 8, device="cuda")
    dg = torch.zeros(n, device="cuda")
    loss = ctypes.c_double(0.0)
    torch.cuda.synchronize()
    for _ in range(2):                   # and again over the workspaces of the first pass
        assert lib.cfdwm_surrogate_forward(cw._ptr(dx), b, h, w, cw._ptr(dy)) == 0
        assert lib.cfdwm_surrogate_loss_grad(cw._ptr(dx), cw._ptr(dt), b, h, w, ctypes.byref(loss),
                                             cw._ptr(dg)) == 0
        y, g = dy.cpu().numpy(), dg.cpu().numpy()
        ref, _ = sr.forward(prm, nl, x.astype(np.float64))
        l_ref, g_ref = sr.loss_grad(prm, nl, x.astype(np.float64), t.astype(np.float64))
        assert norm_rel_err(y.ravel(), ref.ravel()) <= TOL_NET
        assert abs(loss.value - l_ref) <= TOL_NET * abs(l_ref)
        for l in range(4):
            k = ch[l + 1] * ch[l] * 9
            for sl in (slice(offw[l], offw[l] + k), slice(offb[l], offb[l] + ch[l + 1])):
                assert norm_rel_err(g[sl].astype(np.float64), g_ref[sl]) <= TOL_GRAD, (l, sl)
