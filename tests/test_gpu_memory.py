"""Device memory of a context's renders: what a render loses, refuses or keeps when its buffers grow, do not
fit or are no longer needed."""
import contextlib

import pytest

from jarabotransientrendering_b200 import _abi, scenes as S

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
