"""Performance cases: what programs that use this renderer have it do, each through its public
entry points (the Python classes of ``renderer`` and the C ABI below them).

A case names a kind of call (``kind``), the scene it works on and its sizes:

* ``preview``  - ``Context.render`` + ``Context.film`` of a few pixels: an interactive preview or a
  unit test's render, where launches and host work are all there is;
* ``window``   - ``tr_render_region_noalloc`` of a pixel window, the frame loop of a program that may
  not allocate, its film read on the device;
* ``pass``     - one progressive pass (``Context.render`` of the next samples), the film copied to a
  device tensor as ``convergence.film_device`` does;
* ``frame``    - a whole frame from scratch: scene upload and BVH, ``Context.render_film`` into pinned
  host memory (RGBE images, FP32 or FP64 sums), release;
* ``modes``    - a film with its options on: per-bounce films, camera unwarp, component images;
* ``guided``   - a pass with the learned proposal attached, the network frozen (the long phase of a
  guided render, after its training budget is spent);
* ``train``    - one training step of the proposal on a pool of path samples;
* ``batch``    - several scenes rendered together by ``Batch.render``;
* ``rays``     - a new mesh uploaded and a batch of rays cast against it.

Rendered films are sums of radiance samples of seeded paths, so a pass has the same outputs every
time, up to the order of the FP64 additions.  Passes add to the film, as progressive renders do.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from jarabotransientrendering_b200 import _abi
from jarabotransientrendering_b200 import renderer as R
from jarabotransientrendering_b200 import scenes as S

ROOM_TRIANGLES = 34                  # the Cornell room and its two boxes
FILM_TYPES = {"rgbe": (torch.uint8, 4), "f32": (torch.float32, 3), "f64": (torch.float64, 3)}


def _case(kind, scene="room", subdiv=0, width=64, height=64, bins=256, sqrt_spp=4, inc=1, depth=8, **more):
    return dict(kind=kind, scene=scene, subdiv=subdiv, width=width, height=height, bins=bins, sqrt_spp=sqrt_spp,
                inc=inc, depth=depth, **more)


def listed():
    return [
        # the smoke test's and an editor preview's size: 1,024 paths, latency only
        dict(_case("preview", width=16, height=16, bins=128, sqrt_spp=2, depth=4), name="preview"),
        # an engine's frame loop on a mid-size mesh: an odd window just below the entry point's limit
        dict(_case("window", "mesh", 5, 160, 120, 512, win_w=61, win_h=47), name="window"),
        # the Cornell workload as configured: 128 x 128, 1024 bins, 64 samples, depth 6
        dict(_case("pass", width=128, height=128, bins=1024, sqrt_spp=8, depth=6), name="room_pass"),
        # a progressive pass over the 327,714-triangle mesh at a ragged size (several pixel batches)
        dict(_case("pass", "mesh", 7, 317, 243, 256, sqrt_spp=8), name="mesh_pass"),
        # the headline workload's frame (67.1 M paths) from host arrays to images in host memory
        dict(_case("frame", "mesh", 7, 512, 512, 1024, sqrt_spp=16, film="rgbe"), name="image_frame"),
        # the participating-medium workload's options (depth 12, two paths per camera sample)
        dict(_case("pass", "medium", 0, 192, 160, 1024, sqrt_spp=8, inc=2, depth=12), name="medium_pass"),
        # light subpaths and vertex connections (time sampling comes with them)
        dict(_case("pass", "mesh", 5, 200, 150, 512, flags=6), name="subpath_pass"),
        # area light, per-bounce films, unwarped time, component images; odd film
        dict(_case("modes", "arealight", 0, 61, 47, 128, sqrt_spp=6, depth=5, bounce_films=3), name="film_modes"),
        # the guided workload (glossy floor, occluded area light) after training
        dict(_case("guided", "guided", 0, 256, 256, 512), name="guided_pass"),
        # one step of the proposal's training: a full batch of 65,536 samples
        dict(_case("train", samples=65536), name="train_step"),
        # sixteen small scenes of uneven meshes, half with media, 32 paths per pixel
        dict(_case("batch", "batch", 0, 64, 64, 256, sqrt_spp=4, inc=2, scenes=16), name="scene_batch"),
        # line-of-sight queries on a mesh that has just changed: upload, BVH build, 262,144 rays
        dict(_case("rays", "mesh", 7, 1, 1, 1, sqrt_spp=1, rays=262144, any_hit=False), name="mesh_rays"),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))

    kind = rng.choice(("preview", "window", "pass", "pass", "pass", "pass", "frame", "modes", "guided", "train", "batch",
                       "rays"))
    subdiv = rng.randint(2, 7)
    width, height, bins = log(24, 400), log(24, 400), log(64, 2048)
    inc = rng.choice((1, 1, 2, 3))
    depth = rng.randint(2, 12)
    sqrt_spp = rng.randint(2, 10)
    if kind == "train":
        return _case(kind, samples=log(1024, 65536))
    if kind == "rays":
        return _case(kind, "mesh", subdiv, 1, 1, 1, sqrt_spp=1, rays=log(500, 1000000), any_hit=rng.random() < 0.4)
    if kind == "preview":
        return _case(kind, rng.choice(("room", "arealight", "mesh")), min(subdiv, 5), log(8, 48), log(8, 48), log(32, 256),
                     rng.randint(1, 4), inc, rng.randint(1, 8))
    if kind == "window":
        win_w, win_h, sqrt_spp = log(4, 96), log(4, 64), rng.randint(1, 6)
        while win_w * win_h * sqrt_spp * sqrt_spp * inc > 65536:
            win_w, win_h = max(4, win_w * 3 // 4), max(4, win_h * 3 // 4)
        return _case(kind, rng.choice(("room", "medium", "mesh")), min(subdiv, 6), win_w + rng.randint(0, 90),
                     win_h + rng.randint(0, 60), bins, sqrt_spp, inc, depth, win_w=win_w, win_h=win_h)
    if kind == "modes":
        return _case(kind, rng.choice(("arealight", "medium", "room")), 0, log(16, 96), log(16, 96), log(32, 256),
                     rng.randint(1, 6), inc, rng.randint(2, 8), bounce_films=rng.randint(1, 4))
    if kind == "guided":
        return _case(kind, "guided", 0, log(48, 400), log(48, 400), log(64, 512), rng.randint(1, 4), 1, rng.randint(3, 9))
    if kind == "batch":
        return _case(kind, "batch", 0, log(16, 96), log(16, 96), log(64, 512), rng.randint(2, 6), inc, rng.randint(3, 10),
                     scenes=rng.randint(2, 16))
    while width * height * sqrt_spp * sqrt_spp * inc > 6_000_000:
        sqrt_spp = max(1, sqrt_spp - 1)
        width, height = width * 7 // 8, height * 7 // 8
    while width * height * bins > 40_000_000:
        bins //= 2
    if kind == "frame":
        return _case(kind, rng.choice(("mesh", "room", "arealight")), subdiv, width, height, bins, sqrt_spp, inc, depth,
                     film=rng.choice(("rgbe", "f32", "f64")))
    scene = rng.choice(("room", "mesh", "mesh", "medium", "arealight"))
    flags = rng.choice((0, 0, 1, 2)) if scene != "mesh" else rng.choice((0, 0, 0, 2, 6))
    if flags == 6:               # connections grow with the square of the depth
        depth, sqrt_spp, inc = min(depth, 8), min(sqrt_spp, 4), 1
    return _case(kind, scene, subdiv, width, height, bins, sqrt_spp, inc, depth, flags=flags)


# ---- scenes ---------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _unit_mesh(subdiv):
    return S.displaced_icosphere(subdiv, (0.0, 0.0, 0.0), 1.0, 0.05, 3, 2.0, seed=1001)


def _add_sphere(sc, subdiv, rng, radius=0.25):
    """The displaced icosphere of ``subdiv``, turned and placed in the room by ``rng``."""
    v, t = _unit_mesh(subdiv)
    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
    q *= np.sign(np.diag(r))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    centre = np.array([rng.uniform(0.4, 0.6), 0.32, rng.uniform(0.4, 0.5)])
    sc.materials.append(S.Material(S.MAT_LAMBERTIAN, (0.6, 0.6, 0.6)))
    sc.meshes.append(S.Mesh("sphere", (v @ q.T.astype(np.float32) * radius + centre).astype(np.float32), t,
                            len(sc.materials) - 1))


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    span = 5.12                                      # path length the film covers, as the workloads' films
    kw = dict(width=case["width"], height=case["height"], time_bins=case["bins"], exposure=span / case["bins"],
              max_bounces=case["depth"], sqrt_spp=case["sqrt_spp"], incoming_samples=case["inc"])
    geometry = 2 + int(rng.integers(0, 1 << 20))     # the boxes' places
    if case["scene"] == "guided":
        sc = S.guided(geometry, **kw)
    else:
        sc = S.cornell(geometry, **kw)
    if case["scene"] == "mesh":
        _add_sphere(sc, case["subdiv"], rng)
    if case["scene"] == "medium":
        sc.medium = S.Medium((0.05,) * 3, (0.5,) * 3, 0.3)
    if case["scene"] == "arealight":
        sc.lights = [S.rect_light((0.4, 0.99, 0.4), (0.4, 0.0, 0.4), (0.2, 0.2), 10.0)]
    sc.seed = 1 + int(rng.integers(0, 1 << 30))
    sc.flags = case.get("flags", 0)
    return sc


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _film_tensors(sc):
    shape = (sc.height, sc.width)
    return {"streak": torch.zeros(shape + (sc.time_bins, 3), dtype=torch.float64, device="cuda"),
            "steady": torch.zeros(shape + (3,), dtype=torch.float64, device="cuda"),
            "weight": torch.zeros(shape, dtype=torch.float64, device="cuda")}


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _film_device(ctx, f):
    _abi.check(_abi.lib().tr_get_film_device(ctx.h, _ptr(f["streak"]), _ptr(f["steady"]), _ptr(f["weight"])))
    return f


# ---- the proposal's inputs -------------------------------------------------------------------

def _network(seed):
    """Parameters of a proposal: hidden layers as the library initialises them, output biases of eight
    lobes of moderate width spread over the directions, as training leaves them."""
    rng = np.random.default_rng(seed)
    w = rng.uniform(-1.0, 1.0, (4, 64, 64)) * np.array([math.sqrt(6 / 64)] * 3 + [0.1]).reshape(4, 1, 1)
    b = np.zeros((4, 64))
    mean = rng.normal(size=(8, 3))
    mean /= np.linalg.norm(mean, axis=1, keepdims=True)
    b[3, 0:40:5] = rng.uniform(-0.5, 0.5, 8)
    for k in range(3):
        b[3, 1 + k:40:5] = mean[:, k]
    b[3, 4:40:5] = rng.uniform(1.0, 3.0, 8)
    return np.concatenate([w.reshape(-1), b.reshape(-1)]).astype(np.float32)


def _train_batch(n, seed):
    """Features, directions and weights of n path vertices on the room's surfaces (device tensors)."""
    g = torch.Generator("cuda").manual_seed(seed)
    u = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    pos = u(n, 3)
    axis = torch.randint(0, 3, (n,), generator=g, device="cuda")
    far = u(n) < 0.5
    pos.scatter_(1, axis[:, None], far.float()[:, None])
    nrm = torch.zeros(n, 3, device="cuda").scatter_(1, axis[:, None], torch.where(far, -1.0, 1.0)[:, None])

    def hemisphere():
        d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
        return torch.nn.functional.normalize(d + 1.001 * nrm, dim=1)

    x = torch.zeros(n, 64, device="cuda")
    for k in range(6):
        for d in range(3):
            x[:, 6 * k + 2 * d] = torch.sin(2.0 ** k * math.pi * pos[:, d])
            x[:, 6 * k + 2 * d + 1] = torch.cos(2.0 ** k * math.pi * pos[:, d])
    x[:, 36:39], x[:, 39:42], x[:, 42:45], x[:, 45] = pos, nrm, hemisphere(), u(n)
    weight = torch.where(u(n) < 0.3, torch.zeros(n, device="cuda"), -torch.log(u(n).clamp_min(1e-6)))
    return x.to(torch.bfloat16).contiguous(), hemisphere().contiguous(), weight.contiguous()


# ---- the calls -------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "next": 0}
    if kind == "train":
        st["guide"] = R.Guide(0, seed=1)
        st["guide"].set_params(_network(seed))
        st["x"], st["dirs"], st["w"] = _train_batch(case["samples"], seed)
        torch.cuda.synchronize()
        return st
    if kind == "batch":
        rng = np.random.default_rng(seed)
        scenes = []
        for i in range(case["scenes"]):
            sc = _scene(dict(case, scene="room"), seed * 131 + i)
            _add_sphere(sc, 3 + i % 4, rng, 0.2)
            if i % 2:
                s = float(rng.uniform(0.1, 1.0))
                sc.medium = S.Medium((s / 10,) * 3, (s,) * 3, float(rng.uniform(-0.3, 0.6)))
            sc.flags = S.FLAG_ORTHONORMAL_FRAME
            scenes.append(sc)
        st["ctxs"] = [R.Context(sc) for sc in scenes]
        st["batch"] = R.Batch(st["ctxs"])
        st["spp"] = scenes[0].spp
        st["films"] = [_film_tensors(sc) for sc in scenes]
        torch.cuda.synchronize()
        return st
    sc = _scene(case, seed)
    st["scene"], st["spp"] = sc, sc.spp
    if kind in ("frame", "rays"):
        v, t, m = (torch.from_numpy(a if a.dtype == np.float32 else a.view(np.int32)).pin_memory() for a in sc.flatten())
        st["arrays"] = (v.numpy(), t.numpy().view(np.uint32), m.numpy().view(np.uint32))
        if kind == "frame":
            dtype, ch = FILM_TYPES[case["film"]]
            H, W, T = sc.height, sc.width, sc.time_bins
            st["out"] = {"streak": _pinned((H, W, T, ch), dtype), "steady": _pinned((H, W, ch), dtype)}
            if case["film"] != "rgbe":
                st["out"]["weight"] = _pinned((H, W), dtype)
        else:
            g = torch.Generator("cuda").manual_seed(seed)
            n = case["rays"]
            st["any_hit"] = case["any_hit"]
            st["rays"] = torch.empty(n, 8, device="cuda")
            st["rays"][:, 0:3] = torch.rand(n, 3, generator=g, device="cuda")
            st["rays"][:, 3] = 1e-5
            st["rays"][:, 4:7] = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1)
            # line-of-sight segments end within the room; closest-hit rays do not end
            st["rays"][:, 7] = 0.5 if case["any_hit"] else math.inf
            st["hits"] = torch.zeros(n, 4, device="cuda")
        torch.cuda.synchronize()
        return st
    if kind == "modes":
        sc.camera_unwarp, sc.bounce_films = 1, case["bounce_films"]
        sc.components = S.COMP_DEPTH | S.COMP_POSITIONS | S.COMP_NORMALS
        H, W, T = sc.height, sc.width, sc.time_bins
        st["films"] = [[_pinned(s, torch.float64) for s in ((H, W, T, 3), (H, W, 3), (H, W))]
                       for _ in range(1 + sc.bounce_films)]
    if kind == "window":
        rng = np.random.default_rng(seed + 1)
        x0 = int(rng.integers(0, sc.width - case["win_w"] + 1))
        y0 = int(rng.integers(0, sc.height - case["win_h"] + 1))
        st["window"] = (x0, y0, x0 + case["win_w"], y0 + case["win_h"])
    if kind == "guided":
        sc.flags |= S.FLAG_ORTHONORMAL_FRAME
    st["ctx"] = R.Context(sc)
    if kind == "guided":
        st["guide"] = R.Guide(0, seed=1)
        st["guide"].set_params(_network(seed))
        st["ctx"].set_guide(st["guide"], mix_prob=0.7, learning_rate=0.0, train_pool=0)
    if kind in ("pass", "window", "guided"):
        st["film"] = _film_tensors(sc)
    torch.cuda.synchronize()
    return st


def run(st):
    kind, begin = st["kind"], st["next"]
    if kind == "train":
        loss = C.c_float()
        _abi.check(_abi.lib().tr_guide_train_step(st["guide"].h, _ptr(st["x"]), _ptr(st["dirs"]), _ptr(st["w"]),
                                                  st["x"].shape[0], 3e-3, C.byref(loss), None))
        grads = np.empty(R.Guide.PARAMS, np.float32)
        _abi.check(_abi.lib().tr_guide_get_grads(st["guide"].h, grads.ctypes.data))
        return {"loss": float(loss.value), "grads": grads, "params": st["guide"].params()}
    if kind == "rays":
        with R.Context(st["scene"], 0, st["arrays"]) as ctx:
            ctx.trace_device(st["rays"].data_ptr(), st["rays"].shape[0], st["hits"].data_ptr(), st["any_hit"])
        hits = st["hits"]
        if st["any_hit"]:              # which occluder a query meets first is up to the traversal
            return {"occluded": hits[:, 1].view(torch.int32) != -1}
        return {"t": hits[:, 0], "triangle": hits[:, 1].view(torch.int32), "uv": hits[:, 2:4]}
    if kind == "frame":
        with R.Context(st["scene"], 0, st["arrays"]) as ctx:
            ctx.render_film(0, st["spp"], **{k: v.numpy() for k, v in st["out"].items()})
        return st["out"]
    st["next"] = begin + st["spp"]
    if kind == "batch":
        st["batch"].render(begin, st["spp"])
        return [_film_device(c, f) for c, f in zip(st["ctxs"], st["films"])]
    ctx = st["ctx"]
    if kind == "window":
        x0, y0, x1, y1 = st["window"]
        _abi.check(_abi.lib().tr_render_region_noalloc(ctx.h, x0, y0, x1, y1, begin, st["spp"], None))
        return _film_device(ctx, st["film"])
    ctx.render(begin, st["spp"])
    if kind == "preview":
        return ctx.film()
    if kind == "modes":
        ctx.film_into(*(t.numpy() for t in st["films"][0]))
        for b, f in enumerate(st["films"][1:]):
            _abi.check(_abi.lib().tr_get_film_bounce(ctx.h, b, *(t.data_ptr() for t in f)))
        return {"films": st["films"], "components": ctx.components()}
    return _film_device(ctx, st["film"])


def _triangles(case):
    return ROOM_TRIANGLES + (20 * 4 ** case["subdiv"] if case["scene"] == "mesh" else 0)


def work(case):
    """Bytes: the scene read and the film (or the other outputs) written, once.  Operations: for a ray,
    four box tests (24 flops each) at each of the log4(triangles) levels it has to descend and two triangle
    tests (60 flops); a path has about as many closest-hit and shadow rays as the workloads' paths."""
    if case["kind"] == "train":
        n = case["samples"]
        return {"bytes": n * (128 + 12 + 4) + 4 * 16640 * 6, "flops": 6.0 * n * 4 * 64 * 64}
    n_scenes = case.get("scenes", 1)
    tris = _triangles(case)
    ray = 24.0 * 4 * max(1.0, math.log(tris, 4)) + 2 * 60
    if case["kind"] == "rays":
        return {"bytes": tris * (12 + 4 + 6) + case["rays"] * 48, "flops": case["rays"] * ray}
    pixels = case["width"] * case["height"]
    paths = (case["win_w"] * case["win_h"] if case["kind"] == "window" else pixels) * case["sqrt_spp"] ** 2 * case["inc"]
    cell = {"rgbe": 4, "f32": 12}.get(case.get("film"), 24)
    film = pixels * ((case["bins"] + 1) * cell + (0 if cell == 4 else cell // 3))
    if case["kind"] == "modes":
        film = film * (1 + case["bounce_films"]) + pixels * 56
    rays = 4.0 if not case.get("flags", 0) & 2 else 8.0
    return {"bytes": n_scenes * (film + tris * 22), "flops": n_scenes * paths * rays * ray}


# ---- what the calls compute, in 64 bits -------------------------------------------------------

def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "rays" and not case["any_hit"] and case["rays"] * _triangles(case) <= 4_000_000_000:
        return {"t": _exact_closest(case, seed), "triangle": None, "uv": None}
    return None                      # a film in 64 bits is another path tracer


def _exact_closest(case, seed):
    """Closest-hit distances by testing every triangle (Moeller & Trumbore 1997)."""
    sc = _scene(case, seed)
    v, t, _ = sc.flatten()
    p = torch.from_numpy(v).cuda().double()[torch.from_numpy(t.astype(np.int64)).cuda()]
    p0, e1, e2 = p[:, 0], p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
    rays = prepare(case, seed)["rays"].double()
    out = []
    step = max(1, 20_000_000 // len(p))
    for r in rays.split(step):
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        h = torch.linalg.cross(d.expand(-1, len(p), -1), e2[None].expand(len(r), -1, -1))
        det = (h * e1).sum(-1)
        s = o - p0
        u = (h * s).sum(-1) / det
        q = torch.linalg.cross(s, e1[None].expand_as(s))
        w = (q * d).sum(-1) / det
        dist = (q * e2).sum(-1) / det
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (dist > 1e-5)
        out.append(torch.where(ok, dist, math.inf).amin(1))
    return torch.cat(out).float().double()


def _exact_train(case, seed):
    """Loss -sum w log q / sum w of the vMF mixture, its gradients, and the parameters after the first
    Adam step, for the unrounded network."""
    p = torch.from_numpy(_network(seed)).cuda().double().requires_grad_(True)
    x, dirs, w = (a.double() for a in _train_batch(case["samples"], seed))
    weights, bias = p[:4 * 4096].view(4, 64, 64), p[4 * 4096:].view(4, 64)
    h = x
    for l in range(3):
        h = torch.relu(h @ weights[l] + bias[l])
    o = (h @ weights[3] + bias[3])[:, :40].reshape(-1, 8, 5)
    kappa = 0.05 + 2000.0 * torch.sigmoid(o[..., 4] - 8.0)
    cosine = (torch.nn.functional.normalize(o[..., 1:4], dim=2) * dirs[:, None]).sum(-1)
    log_vmf = torch.log(kappa) - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa)) + kappa * (cosine - 1)
    log_q = torch.logsumexp(torch.log_softmax(o[..., 0], 1) + log_vmf, 1)
    loss = -(w * log_q).sum() / w.sum()
    (g,) = torch.autograd.grad(loss, p)
    after = p.detach() - 3e-3 * g / (g.abs() + 1e-8)
    return {"loss": float(loss), "grads": g, "params": after}
