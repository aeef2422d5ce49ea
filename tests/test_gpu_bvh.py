"""The device BVH build at the edges of its phases: one node, the eight- and sixteen-lane node sizes, the
largest subtree one block finishes and the first ones that take level launches, coincident triangles
(no axis can be binned) and a mesh stretched over nine orders of magnitude (deep, unbalanced tree).
The tree decides only what is visited, so the hits of every build equal the oracle's."""
import numpy as np
import pytest

from jarabotransientrendering_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _mesh(kind, n):
    rng = np.random.default_rng(n)
    c = rng.random((n, 1, 3))
    if kind == "same":
        c[:] = 0.5
    if kind == "stretched":
        c *= 10.0 ** rng.uniform(-9.0, 0.0, (n, 1, 1))
    size = 0.5 if kind == "same" else 0.1
    p = c + size * (rng.random((n, 3, 3)) - 0.5) * (1.0 if kind != "stretched" else np.maximum(c, 1e-9))
    if kind == "same":                       # one triangle, n times
        p = np.repeat(p[:1], n, axis=0)
    return p.astype(np.float32).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("kind,n", [("random", 1), ("random", 3), ("random", 8), ("random", 9), ("random", 17),
                                    ("random", 511), ("random", 512), ("random", 513), ("random", 1030),
                                    ("random", 20011), ("same", 5), ("same", 600), ("same", 2500), ("stretched", 400),
                                    ("stretched", 30000)])
def test_hits_over_device_built_trees_match_oracle(gpu, oracle_lib, kind, n):
    v, t = _mesh(kind, n)
    sc = S.cornell(width=4, height=4, time_bins=8, exposure=1.0, sqrt_spp=1)
    sc.meshes = [S.Mesh("soup", v, t, 0)]
    rays = S.random_rays(4000, seed=n)
    with gpu.Context(sc) as ctx:
        hits = ctx.trace(rays)
        blocked = ctx.trace(rays, any_hit=True)
        st = ctx.stats()
    assert 1 <= st["bvh_nodes"] <= max(1, n - 1)
    ref = oracle_lib.Oracle(sc).trace(rays)
    assert (hits["prim_id"] == ref["prim_id"]).all()
    assert (hits["t"].view(np.uint32) == ref["t"].view(np.uint32)).all()
    assert ((blocked["prim_id"] != 0xFFFFFFFF) == (ref["prim_id"] != 0xFFFFFFFF)).all()
