"""A batch that has the GPU to itself walks its last depths in one launch, from the first depth that few
paths reach; per-kernel timing keeps the wavefront kernels.  Same rays, vertices and records, so films agree
up to the order of the FP64 additions (relative 1e-12) and the ray counters are equal."""
import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi, scenes as S

pytestmark = pytest.mark.gpu


def _scene(name, width, height, sqrt_spp, inc, depth):
    kw = dict(width=width, height=height, time_bins=64, exposure=0.08, max_bounces=depth, sqrt_spp=sqrt_spp,
              incoming_samples=inc)
    if name == "mesh":
        return S.icosphere(subdiv=3, **kw)
    sc = {"room": S.cornell, "options": S.cornell, "medium": S.medium, "ggx": S.guided}[name](**kw)
    if name == "options":
        sc.camera_unwarp, sc.bounce_films = 1, 2
        sc.components = S.COMP_DEPTH | S.COMP_POSITIONS | S.COMP_NORMALS
    return sc


def _render(gpu, sc, wavefront):
    with gpu.Context(sc) as ctx:
        if wavefront:
            _abi.check(_abi.lib().tr_set_profiling(ctx.h, 1))
        ctx.render(0, sc.spp)
        films = [ctx.film()] + [ctx.bounce_film(b) for b in range(sc.bounce_films)]
        films.append(ctx.components() if sc.components else {})
        st = ctx.stats()
    return films, {k: st[k] for k in ("paths", "closest_rays", "shadow_rays", "splats")}


# more paths than one launch walks whole; six bounces (never), seven (the first with it), the deepest; about
# 106 thousand paths (few left early) to 1.4 million (few left late)
@pytest.mark.parametrize("name,width,height,sqrt_spp,inc,depth", [
    ("room", 131, 90, 3, 1, 6), ("room", 131, 90, 3, 1, 7), ("room", 131, 90, 3, 1, 8), ("room", 300, 291, 4, 1, 12),
    ("room", 131, 90, 3, 1, 63), ("mesh", 173, 160, 4, 1, 9), ("medium", 97, 70, 4, 2, 12), ("ggx", 127, 101, 4, 1, 8),
    ("options", 113, 67, 4, 1, 10)])
def test_last_depths_equal_the_wavefront(gpu, name, width, height, sqrt_spp, inc, depth):
    sc = _scene(name, width, height, sqrt_spp, inc, depth)
    a, ca = _render(gpu, sc, False)
    b, cb = _render(gpu, sc, True)
    assert ca == cb
    for fa, fb in zip(a, b):
        for k in fa:
            if fa[k] is not None:
                assert np.allclose(fa[k], fb[k], rtol=1e-12, atol=0.0), k
