"""Small batches render whole paths in one launch; per-kernel timing keeps the wavefront kernels apart.
Both walk the same paths and leave the same splat records, so films agree up to the order of the
FP64 additions (relative 1e-12) and the ray counters are equal."""
import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi, scenes as S

pytestmark = pytest.mark.gpu


def _scene(name, width, height, sqrt_spp, inc):
    kw = dict(width=width, height=height, time_bins=64, exposure=0.08, max_bounces=5, sqrt_spp=sqrt_spp,
              incoming_samples=inc)
    if name == "mesh":
        return S.icosphere(subdiv=3, **kw)
    if name == "medium":
        return S.medium(**kw)
    if name == "arealight":
        sc = S.guided(lambertian_floor=True, **kw)
        sc.lights = [S.rect_light((0.6, 0.8, 0.6), (0.6, 0.0, 0.6), (0.2, 0.2), 4.0)]
        return sc
    sc = S.guided(**kw) if name == "ggx" else S.medium(**kw) if name == "timesampling" else S.cornell(**kw)
    if name == "timesampling":
        sc.flags = S.FLAG_TIME_SAMPLING
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


# path counts: one, around a warp's sixteen, one per resident warp and one more (2,960), above that
@pytest.mark.parametrize("name,width,height,sqrt_spp,inc", [
    ("room", 1, 1, 1, 1), ("room", 5, 3, 1, 1), ("room", 17, 1, 1, 1), ("room", 80, 37, 1, 1), ("room", 47, 63, 1, 1),
    ("mesh", 37, 29, 4, 1), ("medium", 24, 24, 4, 2), ("arealight", 23, 19, 3, 3), ("ggx", 24, 24, 3, 1),
    ("timesampling", 24, 24, 3, 1), ("options", 31, 17, 3, 2)])
def test_whole_paths_equal_the_wavefront(gpu, name, width, height, sqrt_spp, inc):
    sc = _scene(name, width, height, sqrt_spp, inc)
    a, ca = _render(gpu, sc, False)
    b, cb = _render(gpu, sc, True)
    assert ca == cb
    for fa, fb in zip(a, b):
        for k in fa:
            if fa[k] is not None:
                assert np.allclose(fa[k], fb[k], rtol=1e-12, atol=0.0), k


def test_no_bounces_leave_an_empty_film(gpu):
    sc = _scene("room", 8, 8, 2, 1)
    sc.max_bounces = 0
    (f, _), _ = _render(gpu, sc, False)
    assert f["streak"].sum() == 0 and (f["weight"] == sc.spp).all()
