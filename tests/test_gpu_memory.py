"""Device memory of a context's renders: what a render loses, refuses or keeps when its buffers grow, do not
fit or are no longer needed."""
import contextlib

import numpy as np
import pytest

from jarabotransientrendering_b200 import _abi, renderer as R, scenes as S

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@contextlib.contextmanager
def _only(free_bytes, release=True):
    """Leaves the device about ``free_bytes`` of free memory (``release``: with the library's pool emptied)."""
    import torch
    if release:
        _abi.check(_abi.lib().tr_release_cached_memory(0))
    torch.cuda.empty_cache()
    hold = torch.empty(max(0, _free() - int(free_bytes)), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def test_render_after_a_failed_one(gpu):
    """An allocation that failed is reported by its own call only: the next render, with memory there again,
    succeeds."""
    sc = S.cornell(width=512, height=512, time_bins=8, exposure=0.64, max_bounces=3, sqrt_spp=4)
    with gpu.Context(sc) as ctx:
        ctx.render(0, 1)
        with _only(300 * MB):
            with pytest.raises(gpu.TransientError, match="memory"):
                ctx.render(1, 15)
        ctx.render(1, 15)
        assert (ctx.film()["weight"] == 16).all()


def _bidirectional():
    sc = S.cornell(width=256, height=256, time_bins=16, exposure=0.4, max_bounces=16, sqrt_spp=4)     # 1 M paths
    sc.flags |= S.FLAG_TIME_SAMPLING | S.FLAG_BIDIRECTIONAL
    return sc


def _connections(gpu, spare):
    """The film and counters of ``_bidirectional``, rendered with ``spare`` bytes of device memory to take (0: all)."""
    with gpu.Context(_bidirectional()) as ctx:
        with _only(spare) if spare else contextlib.nullcontext():
            ctx.render(0, 16)
        return ctx.film(), ctx.stats()


def test_connections_with_room_for_one_queue(gpu):
    """Light subpaths set up the next depth's connections while this one's are traced where two queues fit, one
    after the other where one fits, also when it is the record flags that do not: the same film and rays."""
    full, cf = _connections(gpu, 0)
    with gpu.Context(_bidirectional()) as ctx:
        base = ctx.stats()["device_bytes"]
    queue = 15 * 3 * 16 << 20                                # 15 rays of 48 bytes in each of 1 M slots
    flags = (16 + 120) << 20                                 # one per record
    for spare in (cf["device_bytes"] - base - queue // 2, cf["device_bytes"] - base - flags // 2):
        one, co = _connections(gpu, spare)
        assert co["device_bytes"] == cf["device_bytes"] - queue
        for k in ("paths", "closest_rays", "shadow_rays", "splats"):
            assert co[k] == cf[k]
        for k in full:
            assert np.allclose(one[k], full[k], rtol=1e-12, atol=0.0), k


def test_context_renders_after_running_out_of_memory(gpu):
    """A render that found no memory leaves its context as it was: nothing of it stays held, and with memory
    there again the same context renders the same film."""
    full, cf = _connections(gpu, 0)
    with gpu.Context(_bidirectional()) as ctx:
        for share in (0.2, 0.5, 0.8):                        # of what the render takes with one queue
            with _only(share * (cf["device_bytes"] - (720 << 20))):
                with pytest.raises(gpu.TransientError, match="memory"):
                    ctx.render(0, 16)
                assert ctx.stats()["device_bytes"] < 256 * MB
        ctx.render(0, 16)
        f, c = ctx.film(), ctx.stats()
    assert c["device_bytes"] == cf["device_bytes"] and c["shadow_rays"] == cf["shadow_rays"]
    for k in full:
        assert np.allclose(f[k], full[k], rtol=1e-12, atol=0.0), k


# from one batch of half a million slots to one of two million; to the large batches of at least 8.4 M paths
@pytest.mark.parametrize("first,second", [(2, 8), (8, 32)])
def test_pending_training_samples_survive_larger_batches(gpu, first, second):
    """The samples a guided pass collected train the proposal during the next pass, of whatever size."""
    sc = S.guided(width=512, height=512, time_bins=8, exposure=0.64, sqrt_spp=8, max_bounces=3)
    sc.flags = S.FLAG_ORTHONORMAL_FRAME
    g = R.Guide(device=0, seed=1)
    try:
        with gpu.Context(sc) as ctx:
            ctx.set_guide(g, mix_prob=0.5, learning_rate=1e-3, train_pool=16384)
            ctx.render(0, first)
            before = g.params()
            ctx.render(first, second)
            assert ctx.stats()["train_steps"] == 1
            assert (g.params() != before).any()
    finally:
        g.close()


def test_rgbe_images_do_not_cost_a_large_render_its_fallback(gpu):
    """A frame whose large batches fit but not beside its RGBE images takes the small ones."""
    sc = S.cornell(width=512, height=512, time_bins=1023, exposure=0.005, max_bounces=3, sqrt_spp=8)
    steady = np.zeros((512, 512, 4), np.uint8)
    with gpu.Context(sc) as ctx:
        ctx.render(0, 1)
        # three batches of 4 M slots take 2.2 GB, the images 1.1 GB, four batches of 2 M slots 1.5 GB
        with _only(2850 * MB):
            ctx.render_film(1, 63, steady=steady)
        f = ctx.film(streak=False)
    assert (f["weight"] == 64).all() and steady.any()


def test_freed_memory_counts_as_free(gpu):
    """What destroyed contexts left in the library's pool counts as free memory for the next one."""
    def scene(bins):
        return S.cornell(width=256, height=256, time_bins=bins, exposure=0.01, sqrt_spp=1, max_bounces=2)
    _abi.check(_abi.lib().tr_release_cached_memory(0))
    gpu.Context(scene(2040)).close()                         # 3.2 GB
    with _only(1000 * MB, release=False):
        before = _free()
        for _ in range(3):                                   # 1.1 GB of the 3.2, of which 2.1 and 1.0 beside are left
            gpu.Context(scene(680)).close()
        assert abs(_free() - before) < 64 * MB
def test_large_batches_are_given_back(gpu):
    """Between its calls a context holds no more than small batches take, however large its renders were,
    and contexts that render in turn share the memory of the large ones."""
    sc = S.cornell(width=512, height=512, time_bins=8, exposure=0.64, max_bounces=6, sqrt_spp=8)
    _abi.check(_abi.lib().tr_release_cached_memory(0))
    with gpu.Context(sc) as a, gpu.Context(sc) as b, gpu.Context(sc) as c:
        a.render(0, 31)                                      # 8.1 M paths: four batches of 2 M slots
        small = a.stats()["device_bytes"]
        b.render(0, 64)
        free1 = _free()
        assert b.stats()["device_bytes"] <= small
        c.render(0, 64)
        assert free1 - _free() < 256 * MB
        for k in range(1, 4):
            b.render(64 * k, 64)
        assert b.stats()["device_bytes"] <= small
        assert free1 - _free() < 256 * MB
        assert (b.film()["weight"] == 256).all()


def test_refused_film_is_not_taken_first(gpu):
    """A film that would leave less than 2 GiB is refused before anything is allocated: the memory that
    destroyed contexts left in the pool stays there."""
    small = S.cornell(width=256, height=256, time_bins=680, exposure=0.01, sqrt_spp=1, max_bounces=2)    # 1.07 GB
    big = S.cornell(width=256, height=256, time_bins=1400, exposure=0.01, sqrt_spp=1, max_bounces=2)     # 2.2 GB
    _abi.check(_abi.lib().tr_release_cached_memory(0))
    gpu.Context(small).close()
    with _only(2600 * MB, release=False):
        before = _free()
        with pytest.raises(gpu.TransientError, match="does not fit"):
            gpu.Context(big)
        assert abs(_free() - before) < 64 * MB
        gpu.Context(small).close()                           # 1 GB of the pool, 2.6 GB beside it
        assert abs(_free() - before) < 64 * MB


def test_small_batches_where_the_large_ones_do_not_fit(gpu):
    """With too little free memory for the two large batches of a render, eight small ones, and the large ones
    again with memory there."""
    sc = S.cornell(width=512, height=512, time_bins=4, exposure=1.28, max_bounces=3, sqrt_spp=8)
    wave = 2 + 3 * 3
    with gpu.Context(sc) as ctx:
        ctx.render(0, 1)
        # two batches of 8 M slots take 2.9 GB, four of 2 M slots 1.5 GB
        for free, batches in ((2300, 8), (4000, 8), (6000, 2)):
            with _only(free * MB):
                ctx.render(0, 64)
            assert ctx.stats()["kernel_launches"] == batches * wave
        assert (ctx.film()["weight"] == 193).all()


def test_large_batches_are_not_carved_up(gpu):
    """What other contexts keep is not taken out of the large batches' memory while that is idle: a large render
    after them maps nothing new."""
    sc = S.cornell(width=512, height=512, time_bins=8, exposure=0.64, max_bounces=6, sqrt_spp=8)
    _abi.check(_abi.lib().tr_release_cached_memory(0))
    with gpu.Context(sc) as a, gpu.Context(sc) as b, gpu.Context(sc) as c:
        a.render(0, 64)
        for x in (b, c):
            x.render(0, 31)                                  # four batches of 2 M slots each, kept
        before = _free()
        a.render(64, 64)
        assert before - _free() < 64 * MB


def test_idle_large_batches_count_as_free(gpu):
    """Memory that large renders left idle is there for a film that needs it."""
    sc = S.cornell(width=512, height=512, time_bins=8, exposure=0.64, max_bounces=6, sqrt_spp=8)
    film = S.cornell(width=256, height=256, time_bins=1400, exposure=0.01, sqrt_spp=1, max_bounces=2)    # 2.2 GB
    _abi.check(_abi.lib().tr_release_cached_memory(0))
    with gpu.Context(sc) as a:
        a.render(0, 64)                                      # two batches of 8 M slots: 3.7 GB
        with _only(1000 * MB, release=False):
            with gpu.Context(film) as ctx:
                ctx.render(0, 1)
                assert (ctx.film(streak=False)["weight"] == 1).all()
        a.render(64, 64)
        assert (a.film()["weight"] == 128).all()


def test_contexts_are_destroyed_while_another_thread_captures(gpu):
    """Giving memory back waits for the device without disturbing a graph that another thread is capturing."""
    import threading
    import torch
    sc = S.cornell(width=64, height=64, time_bins=64, exposure=0.08, max_bounces=3, sqrt_spp=4)
    g, x = R.Guide(device=0, seed=1), torch.zeros(1024, device="cuda")
    ctx = gpu.Context(sc)
    ctx.render(0, sc.spp)
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()

    def destroy():
        ctx.close()
        g.close()

    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="thread_local")
        x += 1
        t = threading.Thread(target=destroy)
        t.start()
        t.join()
        x += 1
        graph.capture_end()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert (x == 6).all()


def test_large_renders_of_several_threads(gpu):
    """Threads whose contexts take and return large batches at once, one on a stream of its caller's, with small
    renders between: the films of the same renders one after another."""
    import threading
    import torch
    scenes = [S.cornell(width=512, height=512, time_bins=8, exposure=0.64, max_bounces=3, sqrt_spp=8, seed=k + 1)
              for k in range(3)]

    def work(k, films, stream=None):
        with gpu.Context(scenes[k]) as ctx:
            if stream is not None:
                _abi.check(_abi.lib().tr_set_stream(ctx.h, stream.cuda_stream))
            for first, count in ((0, 32), (32, 2), (34, 64), (98, 1)):
                ctx.render(first, count)
            films[k] = ctx.film()

    one, many = [None] * 3, [None] * 3
    for k in range(3):
        work(k, one)
    side = torch.cuda.Stream()
    threads = [threading.Thread(target=work, args=(k, many, side if k == 1 else None)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(one, many):
        assert (a["weight"] == 99).all() and (b["weight"] == 99).all()
        for k in a:
            assert np.allclose(a[k], b[k], rtol=1e-12, atol=0.0), k
