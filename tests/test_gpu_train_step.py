"""One training step around its tile edges: 1 to 129 rows (a 128-row forward tile, 64-row weight-gradient
tiles) and more K-tiles than CTAs, against the numpy restatement (BF16 at the same points: the
tolerances of the gradient test), and the same bits from every run."""
import ctypes as C

import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi
from oracle import guide_oracle as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 74 * 64, 74 * 64 + 1, 19001])
def test_step_matches_oracle_and_repeats(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    params = rng.normal(0, 0.15, G.NP).astype(np.float32)
    x = G.bf16(rng.normal(0.0, 1.0, (n, 64)).astype(np.float32))
    x[:, 46:] = 0.0
    dirs = rng.normal(size=(n, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    w = (rng.random(n) + 0.05).astype(np.float32)
    xd = torch.from_numpy(G.to_bf16_bits(x).view(np.int16)).cuda()
    dd, wd = torch.from_numpy(dirs.astype(np.float32)).cuda(), torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
    L, got = _abi.lib(), []
    for _ in range(2):
        h = C.c_void_p()
        _abi.check(L.tr_guide_create(0, 1, C.byref(h)))
        try:
            _abi.check(L.tr_guide_set_params(h, params.ctypes.data))
            loss = C.c_float()
            _abi.check(L.tr_guide_train_step(h, C.c_void_p(xd.data_ptr()), C.c_void_p(dd.data_ptr()),
                                             C.c_void_p(wd.data_ptr()), n, 1e-3, C.byref(loss), None))
            g, p = np.zeros(G.NP, np.float32), np.zeros(G.NP, np.float32)
            _abi.check(L.tr_guide_get_grads(h, g.ctypes.data))
            _abi.check(L.tr_guide_get_params(h, p.ctypes.data))
        finally:
            L.tr_guide_destroy(h)
        got.append((loss.value, g, p))
    assert got[0][0] == got[1][0] and (got[0][1] == got[1][1]).all() and (got[0][2] == got[1][2]).all()
    ref_loss, ref = G.gradients(params, x, dirs, w)
    assert abs(got[0][0] - ref_loss) <= 1e-3 * abs(ref_loss) + 1e-4
    g = got[0][1]
    for a, b in [(l * 4096, (l + 1) * 4096) for l in range(4)] + [(4 * 4096, G.NP)]:
        assert np.linalg.norm(g[a:b] - ref[a:b]) <= 0.05 * np.linalg.norm(ref[a:b]) + 1e-12
    exp, _, _ = G.adam(params, g, np.zeros(G.NP), np.zeros(G.NP), 1, 1e-3)
    assert np.allclose(got[0][2], exp, atol=1e-6, rtol=1e-5)
