"""Timing cases: the work a program gives this framework, through its public entry points.

listed() are twelve named cases and draw() makes more of the same ranges. Scenes are the seeded
heightfield + cube scenes of the benchmark configurations; they and the server stay resident between
calls, as in a program that loads its level once. Everything else (rays, cameras, lights, images,
requests) comes from the case and the seed.

Families:

* cast: one ray-cast launch (closest hit, closest hit with one ray per thread, any hit) over a ray buffer.
* primary: camera rays generated into a buffer, then their closest hits.
* frame: a short sequence of wavefront frames with TAA from a fresh history.
* batch: many uneven ray batches over several scenes in one launch.
* serve: a burst of ray queries and renders through the server, host buffers in and out.
* taa: the TAA resolve alone, with camera motion.
* display: tonemap + gamma of a linear image, then the scaling pass to the window's 8-bit image.
"""
import functools
import math
import random

import numpy as np
import torch

import phantasyenginetestbed_gb300 as P
from phantasyenginetestbed_gb300 import batch as B
from phantasyenginetestbed_gb300 import renderer as R
from phantasyenginetestbed_gb300 import serve as S

CAM_DIR = (0.0, 0.8, -0.6)
CAM_UP = (0.0, 0.6, 0.8)
BATCH_SCENES = ("c3_10k", "c3_155k", "c3_1m", "c3_2m")
SERVE_SCENES = ("c3_10k", "c3_155k", "c3_1m")


def listed():
    return [
        # The smallest call of a game or a service: a few thousand visibility probes, closest hit, on a
        # small level. Latency and launches count.
        {"name": "query_4k", "family": "cast", "entry": "closest", "rays": "surface", "scene": "c3_10k", "n": 4096},
        # Picking / depth pre-pass: 512x512 camera rays on the 9,392-triangle scene, the plain configuration.
        {"name": "primary_512", "family": "primary", "entry": "plain", "scene": "c1_64_100", "w": 512, "h": 512},
        # Ambient probes of one frame: diffuse secondary rays of a million camera hits, an odd count.
        {"name": "diffuse_1m", "family": "cast", "entry": "closest", "rays": "diffuse", "scene": "c2_256_2000",
         "n": 1000003},
        # Shadow rays of one frame towards a point light, results scattered to their pixels.
        {"name": "shadow_778k", "family": "cast", "entry": "any_scatter", "rays": "shadow", "scene": "c2_256_2000",
         "n": 777601},
        # The large incoherent workload: diffuse rays on a level of two million triangles.
        {"name": "diffuse_8m_2m", "family": "cast", "entry": "closest", "rays": "diffuse", "scene": "c3_2m",
         "n": 8388608},
        # The headline: eight 1080p frames, one point light, split into two parts, replayed from a graph.
        {"name": "frame_1080p", "family": "frame", "scene": "c2_256_2000", "textured": False, "w": 1920, "h": 1080,
         "lights": 1, "frames": 8, "moving": False, "parts": 2, "in_flight": 1, "graph": True},
        # A walk through a textured level: the camera moves every frame, four lights.
        {"name": "frame_720p_moving", "family": "frame", "scene": "c2_256_2000", "textured": True, "w": 1280, "h": 720,
         "lights": 4, "frames": 4, "moving": True, "parts": 1, "in_flight": 1, "graph": True},
        # A thumbnail: one small frame, launched directly.
        {"name": "frame_256", "family": "frame", "scene": "c3_10k", "textured": False, "w": 256, "h": 256,
         "lights": 1, "frames": 1, "moving": False, "parts": 1, "in_flight": 1, "graph": False},
        # 64 uneven batches, half pinhole and half surface rays, 70/30 closest/any, over four scenes.
        {"name": "batch_64", "family": "batch", "items": 64, "lo": 1024, "hi": 1 << 20},
        # A burst of requests at a server: small and middling queries and renders.
        {"name": "serve_burst", "family": "serve", "queries": 24, "renders": 8, "max_rays": 262144, "max_w": 1280},
        # TAA of a 1080p image under camera motion, for a host with its own shading.
        {"name": "taa_1080p", "family": "taa", "w": 1920, "h": 1080, "moving": True},
        # Display of a 1080p image in a 2560x1440 window.
        {"name": "display_1440p", "family": "display", "w": 1920, "h": 1080, "dw": 2560, "dh": 1440},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["cast", "cast", "cast", "primary", "frame", "frame", "batch", "serve", "taa", "display"])
    if family == "cast":
        return {"family": family, "entry": rng.choice(["closest", "closest", "plain", "any", "any_scatter"]),
                "rays": rng.choice(["surface", "diffuse", "shadow"]),
                "scene": rng.choice(["c1_64_100", "c3_10k", "c2_256_2000", "c3_155k", "c3_1m", "c3_2m"]),
                "n": _log(rng, 4096, 4 << 20)}
    if family == "primary":
        return {"family": family, "entry": rng.choice(["plain", "closest"]),
                "scene": rng.choice(["c1_64_100", "c2_256_2000", "c3_1m"]),
                "w": 8 * rng.randint(16, 240), "h": 8 * rng.randint(16, 135)}
    if family == "frame":
        mode = rng.choice(["whole", "parts", "flight"])
        return {"family": family, "scene": rng.choice(["c3_10k", "c2_256_2000", "c3_1m"]),
                "textured": rng.random() < 0.5, "w": 8 * rng.randint(32, 240), "h": 8 * rng.randint(16, 135),
                "lights": rng.randint(1, 4), "frames": rng.randint(1, 4), "moving": rng.random() < 0.5,
                "parts": 2 if mode == "parts" else 1, "in_flight": 2 if mode == "flight" else 1,
                "graph": rng.random() < 0.7}
    if family == "batch":
        return {"family": family, "items": rng.randint(4, 64), "lo": 1024, "hi": _log(rng, 16384, 1 << 20)}
    if family == "serve":
        return {"family": family, "queries": rng.randint(4, 24), "renders": rng.randint(1, 8),
                "max_rays": _log(rng, 16384, 262144), "max_w": rng.choice([512, 768, 1024, 1280])}
    if family == "taa":
        return {"family": family, "w": rng.randint(200, 1920), "h": rng.randint(100, 1080), "moving": rng.random() < 0.7}
    return {"family": "display", "w": rng.randint(200, 1920), "h": rng.randint(100, 1080),
            "dw": rng.randint(200, 2560), "dh": rng.randint(100, 1440)}


# ------------------------------------------------------------------------------------------------------
# Scenes and rays
# ------------------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _host_scene(name):
    s = P.standard_scene(name)
    return s, P.build_sbvh(s.tri_verts)


@functools.lru_cache(maxsize=None)
def _slot_verts(name):
    """Slot vertices on the device, (slots, 3, 4): a host's own copy for its surface normals."""
    _, b = _host_scene(name)
    return torch.from_numpy(np.stack([b.verts["v0"], b.verts["v1"], b.verts["v2"]], axis=1)).cuda()


@functools.lru_cache(maxsize=None)
def _scene(name, textured=False):
    """A resident scene with its materials; `textured` gives half of them albedo, roughness and metallic textures."""
    s, b = _host_scene(name)
    if not textured:
        return P.Scene.from_bvh(b, s)
    rng = np.random.default_rng(len(s.materials))
    datas, mats = s.datas.copy(), s.materials.copy()
    for c, uv in enumerate(("uv0", "uv1", "uv2")):   # planar texture coordinates, several repeats
        datas[uv][:, 0] = s.tri_verts[:, 3 * c] * (5.0 / s.scale) - 1.3
        datas[uv][:, 1] = s.tri_verts[:, 3 * c + 1] * (5.0 / s.scale) - 0.7
    textures = [rng.integers(128, 256, (256, 320, 4), dtype=np.uint8), rng.integers(64, 256, (128, 128), dtype=np.uint8),
                rng.integers(0, 64, (64, 64, 2), dtype=np.uint8)]
    pick = rng.integers(0, 4, len(mats))
    mats["texIndex"][:] = -1
    mats["texIndex"][pick == 1, 0] = 0
    mats["texIndex"][pick == 2] = [0, 1, 2, -1]
    scene = P.Scene(b.nodes, b.verts, b.slot_datas(datas), s.materials)
    scene.setMaterialsAndTextures(mats, textures)
    return scene


def _triangles(name):
    g, cubes, _, _ = P.STANDARD_SCENES[name]
    return 2 * g * g + 12 * cubes


def _scale(name):
    return P.STANDARD_SCENES[name][0] / 64.0


def _cam_pos(name, seed, f=0):
    """The configurations' view point, moved a little by the seed, and along a path by the frame."""
    k, r = _scale(name), random.Random(seed)
    return (k * (0.5 + r.uniform(-0.03, 0.03) + 0.002 * f), k * (-0.3 + r.uniform(-0.03, 0.03) + 0.003 * f),
            k * (0.6 + r.uniform(-0.03, 0.03)))


def _camera(name, seed, res):
    return P.camera_def(_cam_pos(name, seed), CAM_DIR, CAM_UP, 60.0, res)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _pack(o, d, tmin, tmax):
    rays = torch.empty((len(o), 8), dtype=torch.float32, device="cuda")
    rays[:, 0:3], rays[:, 3], rays[:, 4:7], rays[:, 7] = o, tmin, d, tmax
    return rays


def _unit(v):
    return v / v.square().sum(1, keepdim=True).sqrt()


def _surface_rays(name, n, g):
    """Uniform directions from random points of random triangles."""
    tv = _slot_verts(name)
    tri = tv[torch.randint(0, len(tv), (n,), generator=g, device="cuda")]
    a, b = torch.rand((n, 1), generator=g, device="cuda"), torch.rand((n, 1), generator=g, device="cuda")
    a, b = torch.where(a + b > 1, 1 - a, a), torch.where(a + b > 1, 1 - b, b)
    p = tri[:, 0, :3] + a * (tri[:, 1, :3] - tri[:, 0, :3]) + b * (tri[:, 2, :3] - tri[:, 0, :3])
    return _pack(p, _unit(torch.randn((n, 3), generator=g, device="cuda")), 1e-3, 4.0 * _scale(name))


def _secondary_rays(name, n, kind, seed, g):
    """Secondary rays of a camera pass over about n pixels, in its 8x8-tile order: cosine-weighted about the
    surface normal ("diffuse") or towards a point light ("shadow"), from the hits repeated to n rays."""
    side = max(64, 8 * math.ceil(math.sqrt(n) / 8))
    rays = torch.empty((side * side, 8), dtype=torch.float32, device="cuda")
    P.gen_primary_rays(rays, _camera(name, seed, (side, side)), (side, side), order=1)
    hits = torch.empty((side * side, 4), dtype=torch.float32, device="cuda")
    P.cast_closest_plain(_scene(name), rays, hits)
    slot = hits.view(torch.int32)[:, 0]
    keep = torch.nonzero(slot >= 0)[:, 0]
    keep = keep[torch.arange(n, device="cuda") % len(keep)]
    tv, o, d = _slot_verts(name)[slot[keep].long()], rays[keep, 0:3], rays[keep, 4:7]
    p = o + d * hits[keep, 1:2]
    if kind == "shadow":
        k = _scale(name)
        light = torch.tensor([0.5 * k, 0.5 * k, 2.0 * k], device="cuda")
        to = light + 0.02 * k * torch.randn((n, 3), generator=g, device="cuda") - p
        dist = to.square().sum(1).sqrt()
        return _pack(p, to / dist[:, None], 1e-3, dist)
    nrm = _unit(torch.linalg.cross(tv[:, 1, :3] - tv[:, 0, :3], tv[:, 2, :3] - tv[:, 0, :3]))
    nrm = torch.where((nrm * d).sum(1, keepdim=True) > 0, -nrm, nrm)
    return _pack(p, _unit(nrm + 0.999 * _unit(torch.randn((n, 3), generator=g, device="cuda"))), 1e-3, 4.0 * _scale(name))


def _rays(name, n, kind, seed, g):
    return _surface_rays(name, n, g) if kind == "surface" else _secondary_rays(name, n, kind, seed, g)


def _lights(name, count, seed):
    k, r = _scale(name), random.Random(seed)
    pos = [[0.5 + r.uniform(-0.1, 0.1), 0.5 + r.uniform(-0.1, 0.1), 2.0]]
    pos += [[r.uniform(0.1, 0.9), r.uniform(0.1, 0.9), r.uniform(0.4, 1.0)] for _ in range(count - 1)]
    return R.make_lights(np.array(pos, np.float32) * np.float32(k), range_=1000.0 * k)


def _hit_views(hits):
    return {"slot": hits.view(torch.int32)[:, 0], "tuv": hits[:, 1:4]}


class _Address:
    """A renderer's result buffer as torch sees it: a tensor made of it keeps it, and so the renderer, alive."""

    def __init__(self, renderer, address, shape):
        self.renderer = renderer
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (address, False), "version": 3}


# ------------------------------------------------------------------------------------------------------
# Preparation
# ------------------------------------------------------------------------------------------------------


def prepare(case, seed):
    return {"cast": _prepare_cast, "primary": _prepare_primary, "frame": _prepare_frame, "batch": _prepare_batch,
            "serve": _prepare_serve, "taa": _prepare_taa, "display": _prepare_display}[case["family"]](case, seed)


def _prepare_cast(case, seed):
    name, n, g = case["scene"], case["n"], _gen(seed)
    st = {"run": _run_cast, "entry": case["entry"], "scene": _scene(name), "rays": _rays(name, n, case["rays"], seed, g)}
    if case["entry"] in ("any", "any_scatter"):
        st["vis"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        st["scatter"] = None
        if case["entry"] == "any_scatter":   # each ray's pixel: a permutation within runs, as compaction leaves it
            order = torch.arange(n, device="cuda") // 64 * 64 + torch.rand(n, generator=g, device="cuda") * 63
            st["scatter"] = torch.argsort(order).to(torch.int32)
        st["result"] = {"vis": st["vis"]}
    else:
        st["hits"] = torch.empty((n, 4), dtype=torch.float32, device="cuda")
        st["result"] = _hit_views(st["hits"])
    return st


def _prepare_primary(case, seed):
    name, res = case["scene"], (case["w"], case["h"])
    n, r = res[0] * res[1], random.Random(seed)
    st = {"run": _run_primary, "entry": case["entry"], "scene": _scene(name), "res": res, "cam": _camera(name, seed, res),
          "jitter": (r.uniform(-0.5, 0.5), r.uniform(-0.5, 0.5)),
          "rays": torch.empty((n, 8), dtype=torch.float32, device="cuda"),
          "hits": torch.empty((n, 4), dtype=torch.float32, device="cuda")}
    st["result"] = {"dir": st["rays"][:, 4:7], **_hit_views(st["hits"])}
    return st


def _prepare_frame(case, seed):
    name, res = case["scene"], (case["w"], case["h"])
    r = R.CudaTracerRenderer(use_graph=case["graph"])
    r.setStaticScene(_scene(name, case["textured"]))
    r.setTargetResolution(res)
    if case["parts"] > 1:
        r.set_frame_parts(case["parts"])
    if case["in_flight"] > 1:
        r.set_frames_in_flight(case["in_flight"])
    cams = [(_cam_pos(name, seed, f if case["moving"] else 0), P.halton_jitter(f)) for f in range(case["frames"])]
    return {"run": _run_frame, "renderer": r, "res": res, "seed": seed, "cams": cams,
            "lights": _lights(name, case["lights"], seed), "seen": {}}


def _batch_plan(case):
    """Scene, kind, size and ray pattern of every batch: the same for every seed."""
    r = random.Random(case["items"] * 1000003 + case["hi"])
    return [(r.randrange(len(BATCH_SCENES)), B.CLOSEST if r.random() < 0.7 else B.ANY, _log(r, case["lo"], case["hi"]),
             i % 2 == 0) for i in range(case["items"])]


def _prepare_batch(case, seed):
    plan, g = _batch_plan(case), _gen(seed)
    hits = torch.empty((sum(n for _, k, n, _ in plan if k == B.CLOSEST), 4), dtype=torch.float32, device="cuda")
    vis = torch.empty(sum(n for _, k, n, _ in plan if k == B.ANY), dtype=torch.uint8, device="cuda")
    items, at, held = [], [0, 0], []
    for i, (si, kind, n, pinhole) in enumerate(plan):
        name = BATCH_SCENES[si]
        if pinhole:
            w, h = 1024, (n + 1023) // 1024
            rays = torch.empty((w * h, 8), dtype=torch.float32, device="cuda")
            P.gen_primary_rays(rays, _camera(name, seed + i, (w, h)), (w, h), order=0)
        else:
            rays = _surface_rays(name, n, g)
        out = hits if kind == B.CLOSEST else vis
        items.append((si, kind, n, rays, out[at[kind]:at[kind] + n]))
        at[kind] += n
        held.append(rays)
    return {"run": _run_batch, "batch": B.Batch([_scene(s) for s in BATCH_SCENES], items), "held": held,
            "result": {**_hit_views(hits), "vis": vis}}


@functools.lru_cache(maxsize=None)
def _server():
    s = S.Server(memory_budget=60 << 30, render_slots=4, max_render_pixels=1280 * 720, max_lights=1)
    return s, [s.add_scene(_scene(name)) for name in SERVE_SCENES]


def _pinned(n, dtype):
    t = torch.zeros(max(1, n) * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True)
    return t.numpy().view(dtype)[:n]


def _serve_plan(case):
    """The requests in arrival order: the same for every seed."""
    r = random.Random(case["queries"] * 1009 + case["renders"])
    plan = []
    for _ in range(case["queries"]):
        plan.append(("rays", r.randrange(len(SERVE_SCENES)), _log(r, 4096, case["max_rays"]),
                     S.REQ_CLOSEST if r.random() < 0.7 else S.REQ_ANY))
    for _ in range(case["renders"]):
        w = max(256, _log(r, 256, case["max_w"]) // 8 * 8)
        plan.append(("render", r.randrange(len(SERVE_SCENES)), (w, max(144, w * 9 // 16 // 8 * 8)), r.randint(1, 4)))
    r.shuffle(plan)
    return plan


def _prepare_serve(case, seed):
    plan, g = _serve_plan(case), _gen(seed)
    hits = _pinned(sum(q[2] for q in plan if q[0] == "rays" and q[3] == S.REQ_CLOSEST), P.RAY_HIT_DTYPE)
    vis = _pinned(sum(q[2] for q in plan if q[0] == "rays" and q[3] == S.REQ_ANY), np.uint8)
    images = _pinned(sum(q[2][0] * q[2][1] * 4 for q in plan if q[0] == "render"), np.float32)
    at, reqs = [0, 0, 0], []
    for i, q in enumerate(plan):
        name = SERVE_SCENES[q[1]]
        if q[0] == "rays":
            rays = _pinned(q[2], P.RAY_IN_DTYPE)
            rays.view(np.float32).reshape(-1, 8)[:] = _surface_rays(name, q[2], g).cpu().numpy()
            which = 0 if q[3] == S.REQ_CLOSEST else 1
            out = (hits if which == 0 else vis)[at[which]:at[which] + q[2]]
            at[which] += q[2]
            reqs.append(("rays", (q[1], rays, out, q[3])))
        else:
            out = images[at[2]:at[2] + q[2][0] * q[2][1] * 4]
            at[2] += len(out)
            reqs.append(("render", (q[1], q[2], q[3], _camera(name, seed + i, q[2]), _cam_pos(name, seed + i),
                                    _lights(name, 1, seed + i), seed + i, out)))
    floats = hits.view(np.float32).reshape(-1, 4)
    server, ids = _server()
    return {"run": _run_serve, "server": server, "ids": ids, "requests": reqs,
            "result": {"slot": hits["triangleIndex"], "tuv": floats[:, 1:4], "vis": vis, "images": images}}


def _prepare_taa(case, seed):
    w, h, g = case["w"], case["h"], _gen(seed)
    new = lambda *s: torch.rand(s, generator=g, device="cuda")  # noqa: E731
    cur, hist = new(h, w, 4), new(h, w, 4)
    cur[..., 3] = 1.0
    hist[..., 3] = 1.0 + torch.floor(hist[..., 3] * 16)
    st = {"run": _run_taa, "res": (w, h), "cur": cur, "hist": hist, "rough": new(h, w), "vel": None, "prev": None,
          "color": torch.empty((h, w, 4), device="cuda"), "out": torch.empty((h, w, 4), device="cuda")}
    if case["moving"]:   # a smooth pan with a few pixels off screen
        y, x = torch.meshgrid(torch.linspace(-1, 1, h, device="cuda"), torch.linspace(-1, 1, w, device="cuda"), indexing="ij")
        pan = new(2) * 0.01 - 0.005
        st["vel"] = torch.stack([pan[0] + 0.004 * x * y, pan[1] + 0.003 * (x - y)], dim=-1).contiguous()
        st["prev"] = (0.8 * st["vel"] + 1e-4 * new(h, w, 2)).contiguous()
    return st


def _prepare_display(case, seed):
    w, h, g = case["w"], case["h"], _gen(seed)
    linear = torch.rand((h, w, 4), generator=g, device="cuda").square() * 4.0
    return {"run": _run_display, "res": (w, h), "window": (case["dw"], case["dh"]), "linear": linear,
            "display": torch.empty((h, w, 4), device="cuda"),
            "image": torch.empty((case["dh"], case["dw"], 4), dtype=torch.uint8, device="cuda")}


# ------------------------------------------------------------------------------------------------------
# One pass
# ------------------------------------------------------------------------------------------------------


def run(state):
    return state["run"](state)


def _run_cast(st):
    if st["entry"] == "closest":
        P.cast_closest(st["scene"], st["rays"], st["hits"])
    elif st["entry"] == "plain":
        P.cast_closest_plain(st["scene"], st["rays"], st["hits"])
    else:
        P.cast_any(st["scene"], st["rays"], st["vis"], scatter=st["scatter"])
    return st["result"]


def _run_primary(st):
    P.gen_primary_rays(st["rays"], st["cam"], st["res"], st["jitter"], order=1)
    (P.cast_closest_plain if st["entry"] == "plain" else P.cast_closest)(st["scene"], st["rays"], st["hits"])
    return st["result"]


def _run_frame(st):
    r, seen, (w, h) = st["renderer"], st["seen"], st["res"]
    r.resetTAA()
    r.set_seed(st["seed"], 0)
    for pos, jitter in st["cams"]:
        r.updateCamera(pos, CAM_DIR, CAM_UP, 60.0, jitter)
        res = r.render(st["lights"])
    r.join()
    out = {"color": (res.color, (h, w, 4)), "history": (res.history, (h, w, 4)), "raw": (res.raw_color, (h, w, 4)),
           "roughness": (res.roughness, (h, w))}
    if res.velocity:
        out["velocity"] = (res.velocity, (h, w, 2))
    for address, shape in out.values():
        if address not in seen:
            seen[address] = torch.as_tensor(_Address(r, address, shape), device="cuda")
    return {k: seen[address] for k, (address, _) in out.items()}


def _run_batch(st):
    st["batch"].launch()
    return st["result"]


def _run_serve(st):
    server, ids, rids = st["server"], st["ids"], []
    for what, a in st["requests"]:
        rids.append((server.submit_rays if what == "rays" else server.submit_render)(ids[a[0]], *a[1:]))
    for rid in rids:
        server.wait(rid)
        server.release(rid)
    return st["result"]


def _run_taa(st):
    R.taa_resolve(st["res"], st["cur"], st["hist"], st["color"], st["out"], st["vel"], st["prev"], st["rough"])
    return {"color": st["color"], "history": st["out"]}


def _run_display(st):
    R.postprocess(st["res"], st["linear"], display=st["display"])
    R.scale(st["res"], st["display"], st["window"], rgba8=st["image"])
    return {"display": st["display"], "image": st["image"]}


# ------------------------------------------------------------------------------------------------------
# The work of one pass
# ------------------------------------------------------------------------------------------------------


def _scene_bytes(name, n):
    """Nodes and triangles, each once, or what n rays can touch of them: a 64-byte node a level, a leaf."""
    t = _triangles(name)
    return min(64.0 * 0.5 * t + 48.0 * t, n * (64.0 * math.log2(t) + 96.0))


def _ray_flops(name, n):
    """A ray's way down the tree to one leaf: two boxes a level (6 subtractions and products each), two triangles."""
    return n * (24.0 * math.log2(_triangles(name)) + 2 * 50.0)


def work(case):
    f = case["family"]
    if f == "cast":
        n, name = case["n"], case["scene"]
        out = 16 if case["entry"] in ("closest", "plain") else 5 if case["entry"] == "any_scatter" else 1
        return {"bytes": n * (32.0 + out) + _scene_bytes(name, n), "flops": _ray_flops(name, n)}
    if f == "primary":
        n, name = case["w"] * case["h"], case["scene"]
        return {"bytes": n * (32.0 + 32.0 + 16.0) + _scene_bytes(name, n), "flops": 30.0 * n + _ray_flops(name, n)}
    if f == "frame":   # per frame: camera, bounce and shadow rays; history in, three images and the roughness out
        n, name, frames = case["w"] * case["h"], case["scene"], case["frames"]
        rays = n * (1.0 + 0.5 + 0.5 * case["lights"])
        return {"bytes": frames * (n * 68.0 + _scene_bytes(name, rays)), "flops": frames * _ray_flops(name, rays)}
    if f == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for si, kind, n, _ in _batch_plan(case):
            total["bytes"] += n * (32.0 + (16 if kind == B.CLOSEST else 1))
            total["flops"] += _ray_flops(BATCH_SCENES[si], n)
        total["bytes"] += sum(_scene_bytes(s, 1e9) for s in BATCH_SCENES)
        return total
    if f == "serve":
        total = {"bytes": 0.0, "flops": 0.0}
        for q in _serve_plan(case):
            if q[0] == "rays":
                total["bytes"] += q[2] * (32.0 + (16 if q[3] == S.REQ_CLOSEST else 1))
                total["flops"] += _ray_flops(SERVE_SCENES[q[1]], q[2])
            else:
                n = q[2][0] * q[2][1]
                total["bytes"] += 16.0 * n * q[3]
                total["flops"] += q[3] * _ray_flops(SERVE_SCENES[q[1]], 2.0 * n)
        return total
    n = case["w"] * case["h"]
    if f == "taa":
        return {"bytes": n * (16.0 + 16 + 4 + 32 + (16 if case["moving"] else 0)), "flops": 60.0 * n}
    return {"bytes": 32.0 * n + 4.0 * case["dw"] * case["dh"], "flops": 100.0 * n + 100.0 * case["dw"] * case["dh"]}


# ------------------------------------------------------------------------------------------------------
# 64-bit results
# ------------------------------------------------------------------------------------------------------


def exact(case, seed):
    if case["family"] == "cast" and case["entry"] in ("closest", "plain") and case["n"] * _triangles(case["scene"]) <= 2e8:
        return _exact_closest(case, seed)
    if case["family"] == "primary":
        return _exact_primary(case, seed)
    if case["family"] == "taa":
        return _exact_taa(case, seed)
    if case["family"] == "display":
        return _exact_display(case, seed)
    return None


def _exact_closest(case, seed):
    """Every ray against every triangle; the slot is the tree's, so it has no value here."""
    st = _prepare_cast(case, seed)
    rays = st["rays"].double()
    tv = torch.from_numpy(np.array(_host_scene(case["scene"])[0].tri_verts)).cuda().double().reshape(-1, 3, 3)
    p0, e1, e2 = tv[None, :, 0], tv[None, :, 1] - tv[None, :, 0], tv[None, :, 2] - tv[None, :, 0]
    found = []
    for r in rays.split(256):
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        q = torch.linalg.cross(d.expand(-1, p0.shape[1], -1), e2.expand(len(r), -1, -1))
        det, s = (e1 * q).sum(-1), o - p0
        rr = torch.linalg.cross(s, e1.expand(len(r), -1, -1))
        u, v, t = (s * q).sum(-1) / det, (d * rr).sum(-1) / det, (e2 * rr).sum(-1) / det
        ok = (det.abs() >= 1e-5) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= r[:, 3:4]) & (t < r[:, 7:8])
        best, at = torch.where(ok, t, math.inf).min(1)
        hit, i = torch.isfinite(best), torch.arange(len(r), device="cuda")
        found.append(torch.stack([torch.where(hit, best, r[:, 7]), torch.where(hit, u[i, at], 0.0),
                                  torch.where(hit, v[i, at], 0.0)], dim=1))
    return {"slot": None, "tuv": torch.cat(found)}


def _exact_primary(case, seed):
    w, h = case["w"], case["h"]
    st = _prepare_primary(case, seed)
    c = torch.from_numpy(P.camera_def_array(st["cam"])).double().reshape(4, 3)
    jx, jy = (float(np.float32(j)) for j in st["jitter"])
    i = torch.arange(w * h)
    tile, k = i // 64, i % 64
    x, y = tile % (w // 8) * 8 + k % 8, tile // (w // 8) * 8 + k // 8
    cx, cy = (x + jx) / w * 2 - 1, (y + jy) / h * 2 - 1
    d = c[1] + c[2] * cx[:, None] + c[3] * cy[:, None]
    return {"dir": d / d.norm(dim=1, keepdim=True), "slot": None, "tuv": None}


def _bilinear(img, px, py):
    """Linear filtering with clamped edges at pixel position (px, py) of an (h, w, c) image."""
    h, w = img.shape[:2]
    x0, y0 = torch.floor(px - 0.5), torch.floor(py - 0.5)
    ax, ay = (px - 0.5 - x0)[..., None], (py - 0.5 - y0)[..., None]
    x, y = x0.long(), y0.long()
    at = lambda i, j: img[j.clamp(0, h - 1), i.clamp(0, w - 1)]  # noqa: E731
    top = at(x, y) * (1 - ax) + at(x + 1, y) * ax
    return top * (1 - ay) + (at(x, y + 1) * (1 - ax) + at(x + 1, y + 1) * ax) * ay


def _exact_taa(case, seed):
    w, h = case["w"], case["h"]
    st = _prepare_taa(case, seed)
    cur, hist, rough = st["cur"].double(), st["hist"].double(), st["rough"].double()
    vel = torch.zeros((h, w, 2), device="cuda").double() if st["vel"] is None else st["vel"].double()
    prev = torch.zeros_like(vel) if st["prev"] is None else st["prev"].double()
    y, x = torch.meshgrid(torch.arange(h, device="cuda") + 0.5, torch.arange(w, device="cuda") + 0.5, indexing="ij")
    hx, hy = x - vel[..., 0] * w, y - vel[..., 1] * h
    off = (hx < 0) | (hx > w) | (hy < 0) | (hy > h)
    size = torch.tensor([w, h], device="cuda").double()
    pv = (_bilinear(prev, hx, hy) * size).norm(dim=-1)
    distrust = (1.2 * ((vel * size).norm(dim=-1) - pv).abs().sqrt()).clamp(max=1.0)
    trust = (1 - (3.0 * (1 - rough) + rough) * distrust).clamp(0.0, 1.0)
    b = _bilinear(hist, hx, hy)
    n = b[..., 3] * trust + 1
    blend = (1 - 1 / n)[..., None]
    rgb = torch.where(off[..., None], cur[..., :3], cur[..., :3] * (1 - blend) + b[..., :3] * blend)
    one = torch.ones_like(n)
    return {"color": torch.cat([rgb, one[..., None]], -1),
            "history": torch.cat([rgb, torch.where(off, one, n)[..., None]], -1)}


def _exact_display(case, seed):
    lin = _prepare_display(case, seed)["linear"].double()

    def filmic(x):
        return (x * (0.25 * x + 0.105 * 0.25) + 0.20 * 0.025) / (x * (0.25 * x + 0.25) + 0.20 * 0.25) - 0.025 / 0.25

    x = 2.0 * (lin[..., :3] - 0.0015).clamp(min=0.0)
    rgb = (filmic(x) / filmic(11.2)).clamp(min=0.0) ** (1 / 2.2)
    return {"display": torch.cat([rgb, lin[..., 3:]], -1), "image": None}
