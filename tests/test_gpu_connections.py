"""Connection rays are set up from per-warp lists of eye-light pairs.  Sizes around a warp and a block, one
slot, more slots than the grid has threads (lists carried from one run of slots to the next), depths without
pairs up to the limit of 16, and films short enough that the delay tests cut the lists.  Against the CPU
oracle: equal ray counts, films per bin up to the FP32 rounding of warp-group sums."""
import numpy as np
import pytest

from jarabotransientrendering_b200 import scenes as S

pytestmark = pytest.mark.gpu

RTOL = 2e-5      # a group of up to 32 FP32 samples: 32 * 2^-24 = 1.9e-6, and the device's FP32 functions


@pytest.mark.parametrize("width,height,sqrt_spp,inc,depth,bins", [
    (1, 1, 1, 1, 6, 96), (31, 1, 1, 1, 6, 96), (11, 3, 1, 1, 16, 96), (257, 1, 1, 1, 5, 96), (13, 7, 2, 3, 12, 40),
    (24, 20, 2, 1, 1, 96), (24, 20, 2, 1, 2, 96), (24, 20, 2, 1, 3, 24), (205, 197, 2, 1, 3, 64)])
def test_connections_match_oracle(gpu, oracle_lib, width, height, sqrt_spp, inc, depth, bins):
    sc = S.cornell(width=width, height=height, time_bins=bins, exposure=0.05, sqrt_spp=sqrt_spp, max_bounces=depth,
                   incoming_samples=inc)
    sc.flags |= S.FLAG_TIME_SAMPLING | S.FLAG_BIDIRECTIONAL
    n = sqrt_spp * sqrt_spp
    with gpu.Context(sc) as c:
        c.render(0, n)
        f, st = c.film(), c.stats()
    o = oracle_lib.Oracle(sc).render(sample_count=n, nthreads=8)
    assert st["closest_rays"] == o["stats"]["closest_rays"] and st["shadow_rays"] == o["stats"]["shadow_rays"]
    for k in ("streak", "steady"):
        assert ((f[k] != 0) == (o[k] != 0)).all()
        assert np.allclose(f[k], o[k], rtol=RTOL, atol=1e-12)
