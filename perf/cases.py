"""The work that programs have this renderer do, as cases to be timed and compared.

Two kinds of program use it.  Some cast batches of rays against one mesh (``Tree.intersect`` and
``Tree.intersect_p``): visibility and picking, primary rays, occlusion.  The others render scenes
through the ``su_*`` API (``SuLibrary``): previews, batch frames, many views of one scene, in the
plain, guided and spectral modes.  Meshes, scenes and their sizes are those of the benchmark,
``sprout_b200/scenes.py`` and the tests.

A ray cast's tree and a rendered scene are built once and kept, as such programs keep them; rays,
cameras and sample streams come from the seed.
"""

import json
import math

import numpy as np
import torch

from sprout_b200 import _lib, capi, scenes
from sprout_b200.cast import Tree, sphere_mesh

MAX_T = 3.4027715434167032e38  # "no limit" of a ray


def listed():
    return [
        # A few thousand line-of-sight queries against a mid-size mesh, as a game or simulation
        # loop asks for each frame: the smallest call, where its latency counts.
        {"name": "occlusion_small", "kind": "occlusion", "n": 36, "rays": 4099},
        # Primary visibility of one 800 x 450 view with barycentrics (coherent rays, a G-buffer).
        {"name": "primary_rays", "kind": "primary", "n": 128, "width": 800, "height": 450},
        # The cast benchmark: 16,777,216 incoherent closest-hit rays, 1,048,576 triangles.
        {"name": "closest_large", "kind": "closest", "n": 512, "rays": 1 << 24},
        # Ambient occlusion of the same mesh: short any-hit rays from points of its surface.
        {"name": "occlusion_large", "kind": "occlusion", "n": 512, "rays": 4194301},
        # Rays and results in the caller's pinned host memory (copies inside the call).
        {"name": "closest_host", "kind": "host", "n": 256, "rays": 1000003},
        # Interactive preview: the camera has moved, one progressive sample per pixel is shown.
        {"name": "preview", "kind": "preview", "width": 333, "height": 187, "samples": 1},
        # A batch frame of the Cornell box at the benchmark's size (surfaces, one lamp).
        {"name": "cornell", "kind": "cornell", "width": 512, "height": 512, "samples": 64},
        # 400 instances of one mesh lit by 4,096 emitters: two-level tree and light tree.
        {"name": "instances", "kind": "instances", "width": 960, "height": 540, "samples": 32},
        # Several views of a heterogeneous medium in one call (a small part of the benchmark's 64).
        {"name": "volume_views", "kind": "volume", "grid": 256, "side": 384, "views": 3, "samples": 32},
        # The same scene class in the hero-wavelength spectral mode.
        {"name": "spectral_view", "kind": "spectral", "grid": 256, "side": 256, "views": 2, "samples": 24},
        # A guided frame of the doorway interior: online training, inference and tracing.
        {"name": "guided", "kind": "guided", "width": 640, "height": 360, "samples": 24},
        # The guiding network by itself: forward outputs and training gradient of a batch.
        {"name": "guide_network", "kind": "network", "batch": 65536},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["occlusion", "occlusion", "primary", "closest", "closest", "host", "preview", "cornell",
                       "instances", "volume", "spectral", "guided", "network"])
    if kind in ("occlusion", "closest", "host"):
        most = {"occlusion": 1 << 22, "closest": 1 << 24, "host": 1 << 20}[kind]
        return {"kind": kind, "n": _log(rng, 8, 512), "rays": _log(rng, 257, most)}
    if kind == "primary":
        return {"kind": kind, "n": _log(rng, 16, 256), "width": _log(rng, 40, 1280), "height": _log(rng, 30, 720)}
    if kind == "preview":
        return {"kind": kind, "width": _log(rng, 48, 640), "height": _log(rng, 32, 360), "samples": rng.randint(1, 4)}
    if kind == "cornell":
        return {"kind": kind, "width": _log(rng, 64, 512), "height": _log(rng, 64, 512), "samples": _log(rng, 4, 64)}
    if kind == "instances":
        return {"kind": kind, "width": _log(rng, 64, 960), "height": _log(rng, 64, 540), "samples": _log(rng, 2, 32)}
    if kind == "volume":
        return {"kind": kind, "grid": rng.choice([64, 96, 129, 256]), "side": _log(rng, 48, 384),
                "views": rng.randint(1, 3), "samples": _log(rng, 4, 32)}
    if kind == "spectral":
        return {"kind": kind, "grid": rng.choice([64, 96, 129, 256]), "side": _log(rng, 48, 256),
                "views": rng.randint(1, 2), "samples": _log(rng, 4, 24)}
    if kind == "guided":
        return {"kind": kind, "width": _log(rng, 160, 640), "height": _log(rng, 90, 360), "samples": rng.randint(17, 24)}
    return {"kind": kind, "batch": _log(rng, 128, 65536)}


# ---- ray casts -------------------------------------------------------------------------------

_mesh = {}


def _tree(n):
    """The benchmark's displaced sphere of 4 n^2 triangles and its tree; the last one is kept."""
    if n not in _mesh:
        _mesh.clear()
        pos, idx = sphere_mesh(n, 0.1, 1)
        _mesh[n] = (Tree().build(pos, idx), torch.from_numpy(pos).cuda(),
                    torch.from_numpy(idx.astype(np.int64)).cuda())
    return _mesh[n]


def _directions(count, g):
    z = 2.0 * torch.rand(count, device="cuda", generator=g) - 1.0
    phi = 2.0 * math.pi * torch.rand(count, device="cuda", generator=g)
    r = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], 1)


def _rays(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind = case["kind"]
    if kind == "primary":
        # a pinhole camera of 40 degrees at distance 3, looking at the mesh from a seeded side
        w, h = case["width"], case["height"]
        eye = 3.0 * _directions(1, g)[0].double().cpu().numpy()
        m = torch.from_numpy(scenes._look_at(eye)).cuda()
        x = (torch.arange(w, device="cuda") + 0.5) / w * 2.0 - 1.0
        y = (1.0 - (torch.arange(h, device="cuda") + 0.5) / h * 2.0) * (h / w)
        d = torch.stack([x[None, :].expand(h, w), y[:, None].expand(h, w),
                         torch.full((h, w), 1.0 / math.tan(math.radians(20.0)), device="cuda")], -1).reshape(-1, 3)
        d = torch.nn.functional.normalize(d, dim=1) @ m[:3, :3]
        o = m[3, :3].expand_as(d)
        lo, hi = torch.zeros(len(d), 1, device="cuda"), torch.full((len(d), 1), 100.0, device="cuda")
    elif kind == "occlusion":
        # ambient occlusion: from a little above random points of the surface, the hemisphere
        n = case["rays"]
        _, pos, idx = _tree(case["n"])
        t = pos[idx[torch.randint(0, len(idx), (n,), device="cuda", generator=g)]]
        b = torch.rand(n, 2, device="cuda", generator=g)
        b = torch.where(b.sum(1, keepdim=True) > 1.0, 1.0 - b, b)
        o = t[:, 0] + b[:, :1] * (t[:, 1] - t[:, 0]) + b[:, 1:] * (t[:, 2] - t[:, 0])
        nrm = torch.nn.functional.normalize(o, dim=1)
        d = _directions(n, g)
        d = torch.where((d * nrm).sum(1, keepdim=True) < 0.0, -d, d)
        lo = torch.full((n, 1), 1e-4, device="cuda")
        hi = 0.05 + 0.45 * torch.rand(n, 1, device="cuda", generator=g)
    else:
        # the cast benchmark's: origins uniform in [-2, 2]^3, uniform directions
        n = case["rays"]
        o = 4.0 * torch.rand(n, 3, device="cuda", generator=g) - 2.0
        d = _directions(n, g)
        lo, hi = torch.zeros(n, 1, device="cuda"), torch.full((n, 1), MAX_T, device="cuda")
    return torch.cat([o, lo, d, hi], 1).float().contiguous()


# ---- rendered scenes --------------------------------------------------------------------------

_engine = {"key": None, "su": None, "cam": None}
_density = {}


def _fbm(n):
    if n not in _density:
        _density[n] = scenes.fbm_density(n)
    return _density[n]


def _integrator(case, seed):
    kind = case["kind"]
    if kind == "guided":
        ptmis = {"min_bounces": 4, "max_bounces": 8, "guiding": True, "seed": seed % 65536}
    elif kind == "spectral":
        ptmis = {"min_bounces": 4, "max_bounces": 32, "spectral": True}
    else:
        return None
    return json.dumps({"surface": {"PTMIS": ptmis}}).encode()


def _scene(case):
    """The engine with the case's scene, built where the engine holds another one."""
    key = json.dumps({k: v for k, v in case.items() if k not in ("name", "seed")}, sort_keys=True)
    if _engine["key"] == key:
        return _engine["su"], _engine["cam"]
    if _engine["su"] is not None:
        _engine["su"].su_release()
    su = capi.SuLibrary()
    kind = case["kind"]
    assert su.su_init(kind == "preview") == 0
    w, h, spp = case.get("width", 0), case.get("height", 0), case["samples"]
    if kind in ("cornell", "preview"):
        cam = scenes.cornell(su, w, h, sphere_subdivisions=6, tonemap=True, spp=spp)
    elif kind == "instances":
        cam = scenes.wavefront(su, w, h, spp)
    elif kind == "guided":
        cam = scenes.doorway(su, w, h, spp, spheres=24, boxes=60, sphere_subdivisions=3, guiding=True)
    else:
        cam = scenes.volume(su, case["side"], case["side"], spp, _fbm(case["grid"]))
        if kind == "spectral":
            su.su_create_integrators(_integrator(case, 0))
    assert su.su_start_render_frame(0) == 0, su.messages
    _engine.update(key=key, su=su, cam=cam)
    return su, cam


def _camera(case, seed):
    """A seeded camera near the scene's own, as a user who moves about places it."""
    rng = np.random.default_rng(seed)
    j = rng.uniform(-1.0, 1.0, 3)
    if case["kind"] == "instances":
        return scenes._look_at((2.0 * j[0], 6.0 + j[1], -17.0 + j[2]), (0.0, 2.0, 0.0))
    if case["kind"] == "guided":
        return scenes._look_at((-2.4 + 0.2 * j[0], 1.5 + 0.2 * j[1], -2.7 + 0.2 * j[2]), (0.6, 0.9, 2.0))
    return scenes._look_at((0.3 * j[0], 1.0 + 0.2 * j[1], -3.4 + 0.2 * j[2]), (0.0, 1.0, 0.0))


# ---- the guiding network -----------------------------------------------------------------------

LAYERS = [(32, 64), (64, 64), (64, 64), (64, 64), (64, 40)]


def _network(case, seed):
    """Parameters (He-style uniform), vertex encodings, directions and weights of a batch."""
    rng = np.random.default_rng(seed)
    params = np.concatenate([np.concatenate([rng.uniform(-1, 1, i * o) * math.sqrt(6.0 / i), np.zeros(o)])
                             for i, o in LAYERS]).astype(np.float32)
    n = case["batch"]
    x = rng.normal(size=(n, 32)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    return params, x, d, rng.uniform(0.0, 3.0, n).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case, "kind": kind}
    if kind in ("occlusion", "primary", "closest", "host"):
        state["tree"] = _tree(case["n"])[0]
        rays = _rays(case, seed)
        if kind == "host":
            n = len(rays)
            pinned = torch.empty(n, 8, pin_memory=True)
            pinned.copy_(rays)
            out = [torch.empty(n, dtype=torch.int32, pin_memory=True), torch.empty(n, pin_memory=True)]
            state["pinned"] = [pinned] + out  # the arrays below are views of these
            state["rays"] = pinned.numpy()
            state["out"] = (out[0].numpy().view(np.uint32), out[1].numpy(), None)
        else:
            state["rays"] = rays
    elif kind == "network":
        state["inputs"] = _network(case, seed)
        n = case["batch"]
        state["outputs"] = np.zeros((n, 40), np.float32), np.zeros(len(state["inputs"][0]), np.float32)
    else:
        _scene(case)
        if kind in ("volume", "spectral"):
            side = case["side"]
            state["views"] = [(side, side, scenes.VOLUME_FOV, scenes._look_at(p))
                              for p, _ in scenes.volume_views(case["views"], seed)]
        else:
            state["camera"] = _camera(case, seed)
            state["integrator"] = _integrator(case, seed)
    return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "occlusion":
        return state["tree"].intersect_p(state["rays"])
    if kind == "primary":
        return state["tree"].intersect(state["rays"], want_uv=True)
    if kind == "closest":
        return state["tree"].intersect(state["rays"])
    if kind == "host":
        return state["tree"].intersect(state["rays"], out=state["out"])
    if kind == "network":
        lib = _lib.load()
        params, x, d, c = (a.ctypes.data for a in state["inputs"])
        out, grad = state["outputs"]
        _lib.check(lib.spb_guide_forward(params, x, case["batch"], out.ctypes.data))
        _lib.check(lib.spb_guide_gradients(params, x, d, c, case["batch"], grad.ctypes.data))
        return {"outputs": out, "gradient": grad}
    su, cam = _scene(case)
    if kind in ("volume", "spectral"):
        return su.render_views(state["views"], case["samples"])
    if state["integrator"] is not None:
        # a guided frame begins with an untrained network
        assert su.su_create_integrators(state["integrator"]) == 0
    assert su.set_transformation(cam, state["camera"]) == 0
    if kind == "preview":
        assert su.su_start_render_frame(0) == 0
        for _ in range(case["samples"]):
            assert su.su_render_iteration() == 0
    else:
        assert su.su_render_frame(0) == 0
    assert su.su_postprocess() == 0
    return su.framebuffer(case["width"], case["height"])[0]


def exact(case, seed):
    """Closest-hit distances and barycentrics by testing every ray against every triangle, and
    the network, in 64 bits.  An image has no such value: it is one draw of its sample streams."""
    kind = case["kind"]
    if kind == "network":
        return _exact_network(*_network(case, seed))
    if kind not in ("primary", "closest", "host"):
        return None
    rays = case["width"] * case["height"] if kind == "primary" else case["rays"]
    if float(rays) * 4 * case["n"] ** 2 > 4e10:
        return None
    r = _rays(case, seed).double()
    _, pos, idx = _tree(case["n"])
    a, b, c = (pos.double()[idx[:, k]] for k in range(3))
    e1, e2 = b - a, c - a
    # Every quantity of the ray-triangle test is bilinear in (d, o x d, o, 1) and the triangle:
    # det = -d . n, u det = d . (e2 x (o - a)), v det = -d . (e1 x (o - a)), t det = (o - a) . n
    n = torch.cross(e1, e2, dim=1)
    o, d, t0, t1 = r[:, 0:3], r[:, 4:7], r[:, 3:4], r[:, 7:8]
    line = torch.cat([d, torch.cross(o, d, dim=1)], 1)
    of_u = torch.cat([-torch.cross(e2, a, dim=1), e2], 1).T
    of_v = torch.cat([torch.cross(e1, a, dim=1), -e1], 1).T
    at = torch.cat([o, -torch.ones_like(t0)], 1)
    plane = torch.cat([n, (a * n).sum(1, keepdim=True)], 1).T
    best_t, best_u, best_v = [], [], []
    step = max(1, (1 << 28) // len(idx))
    for k in range(0, len(r), step):
        s = slice(k, k + step)
        inv = 1.0 / (-d[s] @ n.T)
        u = line[s] @ of_u * inv
        v = line[s] @ of_v * inv
        t = at[s] @ plane * inv
        hit = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= t0[s]) & (t <= t1[s])
        t, i = torch.where(hit, t, math.inf).min(1, keepdim=True)
        got = torch.isfinite(t)
        best_t.append(torch.where(got, t, t1[s])[:, 0])
        best_u.append(torch.where(got, u.gather(1, i), 0.0)[:, 0])
        best_v.append(torch.where(got, v.gather(1, i), 0.0)[:, 0])
    t = torch.cat(best_t)
    if kind == "primary":
        return None, t, torch.stack([torch.cat(best_u), torch.cat(best_v)], 1)
    return None, t


def _exact_network(params, x, d, c):
    p = torch.from_numpy(params).cuda().double().requires_grad_(True)
    a, k = torch.from_numpy(x).cuda().double(), 0
    for layer, (i, o) in enumerate(LAYERS):
        w, b = p[k:k + i * o].reshape(o, i), p[k + i * o:k + i * o + o]
        k += i * o + o
        a = a @ w.T + b
        if layer < len(LAYERS) - 1:
            a = torch.relu(a)
    # the mixture of eight von Mises-Fisher lobes and the batch's weighted -log density
    lobes = a[:, :32].reshape(-1, 8, 4)
    mu = torch.nn.functional.normalize(lobes[:, :, :3], dim=2)
    kappa = torch.exp(lobes[:, :, 3].clamp(-3.0, 6.0))
    cos = (mu * torch.from_numpy(d).cuda().double()[:, None, :]).sum(2)
    log_q = (torch.log_softmax(a[:, 32:], 1) + torch.log(kappa / (2 * math.pi * -torch.expm1(-2 * kappa)))
             + kappa * (cos - 1.0))
    loss = (-torch.logsumexp(log_q, 1) * torch.from_numpy(c).cuda().double()).mean()
    grad, = torch.autograd.grad(loss, p)
    return {"outputs": a.detach(), "gradient": grad}


def work(case):
    """Bytes: inputs and results once, with the triangles (36 B) or voxels that a pass reads.
    Operations: for each ray one way down an 8-wide tree (8 boxes of 12 FLOP a level) and one
    triangle (60 FLOP); for each sample three such rays and 200 FLOP of shading a vertex; for the
    network the products of its layers."""
    kind = case["kind"]

    def ray(triangles):
        return 96 * max(1, math.ceil(math.log(triangles, 8))) + 60

    if kind in ("occlusion", "primary", "closest", "host"):
        rays = case["width"] * case["height"] if kind == "primary" else case["rays"]
        triangles = 4 * case["n"] ** 2
        out = {"occlusion": 1, "primary": 16}.get(kind, 8)
        return {"bytes": rays * (32 + out) + 36 * triangles, "flops": rays * ray(triangles)}
    if kind == "network":
        n, forward = case["batch"], 2 * sum(i * o for i, o in LAYERS)
        first = 2 * LAYERS[0][0] * LAYERS[0][1]
        parameters = sum(i * o + o for i, o in LAYERS)
        return {"bytes": 4 * n * (2 * 32 + 40 + 4) + 12 * parameters, "flops": n * (4 * forward - first)}
    if kind in ("volume", "spectral"):
        pixels, triangles = case["views"] * case["side"] ** 2, 1000
        scene = 4 * case["grid"] ** 3
    else:
        pixels = case["width"] * case["height"]
        triangles = {"instances": 9098, "guided": 31448}.get(kind, 81932)
        scene = 36 * triangles
    return {"bytes": 16 * pixels + scene, "flops": pixels * case["samples"] * 3 * (ray(triangles) + 200)}
