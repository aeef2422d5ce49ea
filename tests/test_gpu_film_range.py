"""tr_get_film_device checks on the host that each array it is given holds the film's: the kernel that copies
it checks no bounds.  Arrays that begin in an allocation and reach beyond its end are refused and stay untouched."""
import ctypes as C

import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi, scenes as S

pytestmark = pytest.mark.gpu


class _Attributes(C.Structure):
    _fields_ = [("type", C.c_int), ("device", C.c_int), ("device_ptr", C.c_void_p), ("host_ptr", C.c_void_p),
                ("reserved", C.c_long * 8)]


def _allocation(rt, size):
    """An allocation of ``size`` bytes with nothing mapped behind it, and all that were made to find it."""
    made = []
    for _ in range(8):
        p, at = C.c_void_p(), _Attributes()
        assert rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0
        made.append(p)
        assert rt.cudaPointerGetAttributes(C.byref(at), C.c_void_p(p.value + size)) == 0
        if at.type == 0:
            return p.value, made
    pytest.skip("every allocation has another behind it")


@pytest.mark.parametrize("short", ["streak", "steady", "weight"])
def test_array_that_ends_too_soon_is_refused(gpu, short):
    import torch
    sc = S.cornell(width=33, height=17, time_bins=64, exposure=0.08, sqrt_spp=1, max_bounces=3)
    npix = sc.width * sc.height
    size = {"streak": npix * sc.time_bins * 3, "steady": npix * 3, "weight": npix}
    rt = C.CDLL("libcudart.so.12")
    end, made = _allocation(rt, 4 << 20)
    end += 4 << 20
    try:
        with gpu.Context(sc) as ctx:
            ctx.render(0, 1)
            host = ctx.film()
            good = {k: torch.full((n,), -7.0, dtype=torch.float64, device="cuda") for k, n in size.items()}
            torch.cuda.synchronize()

            def get(offset):
                ptr = {k: t.data_ptr() for k, t in good.items()}
                ptr[short] = end - 8 * offset
                return _abi.lib().tr_get_film_device(ctx.h, *(C.c_void_p(ptr[k]) for k in size))

            assert get(size[short] - 1) == 1
            assert all((t == -7.0).all() for t in good.values())
            assert get(size[short]) == 0
            got = np.empty(size[short])
            assert rt.cudaMemcpy(got.ctypes.data_as(C.c_void_p), C.c_void_p(end - 8 * size[short]),
                                 C.c_size_t(8 * size[short]), 2) == 0
            assert (got == host[short].reshape(-1)).all()
    finally:
        for p in made:
            assert rt.cudaFree(p) == 0
