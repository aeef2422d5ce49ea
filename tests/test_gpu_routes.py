"""Which launches a render takes, by its count of kernels: whole paths in one launch (and the splat) up to 32,768
paths per level of the tree, else a ray generation, three kernels per depth and a splat per batch; one more
for the last depths of a lone batch of at least seven bounces; fewer, larger batches from 8.4 M paths on."""
import pytest

from jarabotransientrendering_b200 import _abi, scenes as S

pytestmark = pytest.mark.gpu


def _room(width, height, sqrt_spp, depth, **kw):
    return S.cornell(width=width, height=height, time_bins=8, exposure=0.64, max_bounces=depth, sqrt_spp=sqrt_spp, **kw)


def _launches(ctx, first, count):
    ctx.render(first, count)
    return ctx.stats()["kernel_launches"]


@pytest.mark.parametrize("depth", [1, 6, 7, 12])
def test_whole_paths_up_to_the_trees_line(gpu, depth):
    with gpu.Context(_room(128, 128, 16, depth)) as ctx:
        levels = ctx.stats()["bvh_depth"]
        wave, tail = 2 + 3 * depth, 1 if depth >= 7 else 0
        assert _launches(ctx, 0, 2 * levels) == 2             # 32,768 paths per level
        assert _launches(ctx, 0, 2 * levels + 1) == wave + tail
        _abi.check(_abi.lib().tr_set_profiling(ctx.h, 1))     # per-kernel times: the kernels apart
        assert _launches(ctx, 0, 1) == wave
        assert _launches(ctx, 0, 2 * levels + 1) == wave


@pytest.mark.parametrize("flags,more", [(S.FLAG_TIME_SAMPLING, 0), (0, 1)])
def test_last_depths_of_a_lone_batch(gpu, flags, more):
    sc = _room(256, 256, 8, 8)
    sc.flags = flags
    wave = 2 + 3 * 8
    with gpu.Context(sc) as ctx:
        assert _launches(ctx, 0, 32) == wave + more           # one batch of 2 M slots
        assert _launches(ctx, 0, 64) == 2 * wave              # two, on two lanes


def test_large_batches_from_their_line_on(gpu):
    sc = _room(512, 512, 8, 3)
    wave = 2 + 3 * 3
    with gpu.Context(sc) as ctx:
        assert _launches(ctx, 0, 31) == 4 * wave              # 8.1 M paths: four of 2 M slots
        assert _launches(ctx, 0, 32) == 2 * wave              # 8.4 M: two of 4 M
        assert _launches(ctx, 0, 64) == 2 * wave              # 16.8 M: two of 8 M
