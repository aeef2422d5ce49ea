"""tr_get_film_device into tensors at 16-byte and at 8-byte offsets, with odd array lengths and with arrays left
out: the values tr_get_film delivers, and nothing beyond the arrays."""
import ctypes as C

import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi, scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,bins,offset", [(1, 1, 1, 0), (3, 1, 5, 1), (33, 17, 31, 0), (33, 17, 31, 1),
                                                      (256, 256, 91, 0)])
def test_device_film_equals_host_film(gpu, width, height, bins, offset):
    import torch
    sc = S.cornell(width=width, height=height, time_bins=bins, exposure=5.12 / bins, sqrt_spp=2, max_bounces=3)
    shapes = [(height, width, bins, 3), (height, width, 3), (height, width)]
    with gpu.Context(sc) as ctx:
        ctx.render(0, sc.spp)
        host = ctx.film()
        for skip in (None, 0, 2):
            dev = [torch.full((int(np.prod(s)) + offset + 4,), -7.0, dtype=torch.float64, device="cuda") for s in shapes]
            torch.cuda.synchronize()
            ptr = [None if k == skip else C.c_void_p(d.data_ptr() + 8 * offset) for k, d in enumerate(dev)]
            _abi.check(_abi.lib().tr_get_film_device(ctx.h, *ptr))
            for k, (d, s, name) in enumerate(zip(dev, shapes, ("streak", "steady", "weight"))):
                d = d.cpu().numpy()
                n = int(np.prod(s))
                want = np.full(n, -7.0) if k == skip else host[name].reshape(-1)
                assert (d[offset:offset + n] == want).all()
                assert (d[:offset] == -7.0).all() and (d[offset + n:] == -7.0).all()
