"""Ray queries at the traversal's edges: directions with zero or vanishing components, origins far
outside the scene, rays with a negative start, and ray counts around the warps' queue runs.  The
oracle evaluates the same triangle test, so ids and distances are equal bit for bit; its own box
test drops hits behind the origin, so rays with a negative start are compared with every triangle
in 64 bits."""
import numpy as np
import pytest

from jarabotransientrendering_b200 import scenes as S

pytestmark = pytest.mark.gpu

SCENE = dict(subdiv=4, width=8, height=8, time_bins=16, exposure=0.4, sqrt_spp=1)


def _rays(kind, n):
    rays = S.random_rays(n, seed=len(kind) + n)
    rng = np.random.default_rng(n)
    d = rays[:, 4:7]
    if kind == "axis":                       # one or two components exactly zero, of either sign
        k = rng.integers(0, 3, n)
        d[np.arange(n), k] = np.where(rng.random(n) < 0.5, 0.0, -0.0)
        two = rng.random(n) < 0.5
        d[two, (k[two] + 1) % 3] = 0.0
        d /= np.linalg.norm(d, axis=1, keepdims=True)
    elif kind == "tiny":                     # components down to where the reciprocal is capped
        k = rng.integers(0, 3, n)
        d[np.arange(n), k] = rng.choice((1e-8, -1e-12, 1e-20, -1e-31, 1e-38), n)
    elif kind == "far":                      # from up to 1,000 scene sizes away, aimed at the room
        target = rays[:, 0:3].copy()
        dist = np.exp(rng.uniform(0.0, np.log(1000.0), n)).astype(np.float32)
        rays[:, 0:3] = target - d * dist[:, None]
    return np.ascontiguousarray(rays, np.float32)


@pytest.mark.parametrize("kind,n", [("axis", 20000), ("tiny", 20000), ("far", 20000), ("uniform", 1),
                                    ("uniform", 31), ("uniform", 33), ("uniform", 113665)])
def test_edge_rays_match_oracle(gpu, oracle_lib, kind, n):
    sc = S.icosphere(**SCENE)
    rays = _rays(kind, n)
    with gpu.Context(sc) as ctx:
        hits = ctx.trace(rays)
        anyhit = ctx.trace(rays, any_hit=True)
    ref = oracle_lib.Oracle(sc).trace(rays)
    assert (hits["prim_id"] == ref["prim_id"]).all()
    assert (hits["t"].view(np.uint32) == ref["t"].view(np.uint32)).all()
    hit = ref["prim_id"] != 0xFFFFFFFF
    assert (hits["u"][hit].view(np.uint32) == ref["u"][hit].view(np.uint32)).all()
    assert (hits["v"][hit].view(np.uint32) == ref["v"][hit].view(np.uint32)).all()
    assert ((anyhit["prim_id"] != 0xFFFFFFFF) == hit).all()


def test_negative_start_finds_hits_behind_the_origin(gpu):
    """Closest hit in (tnear, inf] with tnear < 0 against all triangles in float64 (Moeller &
    Trumbore 1997).  A float32 plane distance over coordinates below 2 is off by at most
    8 * 2^-24 / |cos|; rays meeting their triangle at |cos| < 0.01 are left out: 5e-5."""
    sc = S.icosphere(**SCENE)
    rays = S.random_rays(1000, seed=5)
    rays[:, 3] = -0.75
    with gpu.Context(sc) as ctx:
        hits = ctx.trace(rays)
    v, t, _ = sc.flatten()
    p = v.astype(np.float64)[t]
    p0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    ng = np.cross(e1, e2)
    ng /= np.linalg.norm(ng, axis=1, keepdims=True)
    compared = 0
    with np.errstate(divide="ignore", invalid="ignore"):
        for r, h in zip(rays.astype(np.float64), hits):
            o, d = r[0:3], r[4:7]
            x = np.cross(d, e2)
            det = np.einsum("ij,ij->i", x, e1)
            s = o - p0
            u = np.einsum("ij,ij->i", x, s) / det
            q = np.cross(s, e1)
            w = q @ d / det
            dist = np.einsum("ij,ij->i", q, e2) / det
            ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (dist > r[3])
            dist = np.where(ok, dist, np.inf)
            k = int(dist.argmin())
            if not np.isfinite(dist[k]):
                assert h["prim_id"] == 0xFFFFFFFF
            elif abs(ng[k] @ d) >= 0.01:
                assert abs(h["t"] - dist[k]) <= 5e-5
                compared += 1
    assert compared > 900
