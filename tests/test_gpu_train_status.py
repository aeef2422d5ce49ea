"""A training step whose tensor-core wait gives up (a wait limit of no polls) is reported and changes nothing:
parameters, moments and step count stay, so the next step is the one a guide that never failed takes."""
import ctypes as C

import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi
from oracle import guide_oracle as G

pytestmark = pytest.mark.gpu

TIMEOUT = 5


@pytest.mark.parametrize("before,failed", [(0, 1), (1, 3)])
def test_a_timed_out_step_is_not_counted(gpu, before, failed):
    import torch
    L, n = _abi.lib(), 1000
    rng = np.random.default_rng(3)
    params = rng.normal(0, 0.15, G.NP).astype(np.float32)
    x = G.bf16(rng.normal(0.0, 1.0, (n, 64)).astype(np.float32))
    dirs = rng.normal(size=(n, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    xd = torch.from_numpy(G.to_bf16_bits(x).view(np.int16)).cuda()
    dd = torch.from_numpy(dirs.astype(np.float32)).cuda()
    wd = torch.from_numpy((rng.random(n) + 0.05).astype(np.float32)).cuda()
    torch.cuda.synchronize()

    def step(g):
        return L.tr_guide_train_step(g, C.c_void_p(xd.data_ptr()), C.c_void_p(dd.data_ptr()), C.c_void_p(wd.data_ptr()),
                                     n, 1e-3, None, None)

    def read(g):
        p = np.zeros(G.NP, np.float32)
        _abi.check(L.tr_guide_get_params(g, p.ctypes.data))
        return p

    got = []
    for fails in (0, failed):
        g = C.c_void_p()
        _abi.check(L.tr_guide_create(0, 1, C.byref(g)))
        try:
            _abi.check(L.tr_guide_set_params(g, params.ctypes.data))
            for _ in range(before):
                _abi.check(step(g))
            p = read(g)
            _abi.check(L.tr_guide_set_wait_limit(g, 0))
            for _ in range(fails):
                assert step(g) == TIMEOUT
                assert (read(g) == p).all()
            _abi.check(L.tr_guide_set_wait_limit(g, 1 << 24))
            for _ in range(2):
                _abi.check(step(g))
                got.append(read(g))
        finally:
            L.tr_guide_destroy(g)
    assert (got[0] == got[2]).all() and (got[1] == got[3]).all()
