"""Renders of at least 8.4 M paths take larger wavefront batches.  The same pixels rendered as two windows
below that size take the small ones: the same paths, so the same film up to the FP32 group sums at
the windows' seam (relative 1e-6) and the same weights and ray counts."""
import numpy as np
import pytest

from jarabotransientrendering_b200 import scenes as S

pytestmark = pytest.mark.gpu


# samples per pixel that fill splat blocks evenly, unevenly (5 pixels of 100 slots) and one pixel per block
@pytest.mark.parametrize("width,height,sqrt_spp,inc", [(363, 364, 8, 1), (301, 290, 10, 1), (97, 92, 18, 3)])
def test_large_batches_equal_small_ones(gpu, width, height, sqrt_spp, inc):
    sc = S.cornell(width=width, height=height, time_bins=8, exposure=0.64, max_bounces=3, sqrt_spp=sqrt_spp,
                   incoming_samples=inc)
    assert sc.paths_per_frame() >= 1 << 23
    with gpu.Context(sc) as ctx:
        ctx.render(0, sc.spp)
        a, ca = ctx.film(), ctx.stats()
    with gpu.Context(sc) as ctx:
        ctx.render(0, sc.spp, window=(0, 0, width, height // 2))
        ctx.render(0, sc.spp, window=(0, height // 2, width, height))
        b, cb = ctx.film(), ctx.stats()
    for k in ("paths", "closest_rays", "shadow_rays", "splats"):
        assert ca[k] == cb[k]
    assert (a["weight"] == b["weight"]).all()
    assert np.allclose(a["streak"], b["streak"], rtol=1e-6, atol=0.0)
    assert np.allclose(a["steady"], b["steady"], rtol=1e-6, atol=0.0)


def test_large_render_falls_back_when_its_batches_do_not_fit(gpu):
    """With too little free memory for the large batches the render takes the small ones."""
    import torch
    sc = S.cornell(width=512, height=512, time_bins=4, exposure=1.28, max_bounces=3, sqrt_spp=8)
    with gpu.Context(sc) as ctx:
        ctx.render(0, 2)
        from jarabotransientrendering_b200 import _abi
        _abi.check(_abi.lib().tr_release_cached_memory(0))
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(max(0, free - (2300 << 20)), dtype=torch.uint8, device="cuda")
        try:
            ctx.render(2, 62)
        finally:
            del hold
            torch.cuda.empty_cache()
        f = ctx.film()
    assert (f["weight"] == 64).all() and f["streak"].sum() > 0
