"""The work that programs built on this framework have it do, as measurable cases.

Every case goes through the C ABI's public entry points (by the package's Python binding): whole frames in the
batched and in the plain form, single ray batches, many batches over resident scenes in one graph, the
per-stage calls of the drop-in path, the sort, frames of moving objects, and a burst of served requests. Scene
shapes and sizes are those of the repository's benchmark configurations and tests (rsh/scenes.py); what a
program changes from call to call (cameras, lights, materials, rays, object poses, keys) comes from the seed.
"""
from __future__ import annotations

import ctypes as C
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "ray-tracer_gb300"))

import rsh  # noqa: E402
from rsh import scenes  # noqa: E402

FRAME_SCENES = ("cornell", "soup", "architecture")


def listed():
    return [
        # the small scene at its configured size, batched form: an interactive viewer's frame; launch latency counts
        {"name": "frame_cornell_512", "kind": "frame", "form": "batched", "scene": "cornell", "size": 1,
         "width": 512, "height": 512, "depth": 1, "lights": 1, "soft": False},
        # object soup at full HD, three mirror bounces: many small objects, large empty regions
        {"name": "frame_soup_1080p", "kind": "frame", "form": "batched", "scene": "soup", "size": 2000,
         "width": 1920, "height": 1080, "depth": 3, "lights": 2, "soft": False},
        # the headline workload: a million triangles, four lights, incoherent second bounces
        {"name": "frame_architecture_1080p", "kind": "frame", "form": "batched", "scene": "architecture", "size": 40,
         "width": 1920, "height": 1080, "depth": 2, "lights": 4, "soft": False},
        # the default configuration (plain per-frame path) on the small scene
        {"name": "plain_cornell_512", "kind": "frame", "form": "plain", "scene": "cornell", "size": 1,
         "width": 512, "height": 512, "depth": 1, "lights": 1, "soft": False},
        # the default configuration on the large scene: the drop-in replacement of a whole engine frame
        {"name": "plain_architecture_1080p", "kind": "frame", "form": "plain", "scene": "architecture", "size": 40,
         "width": 1920, "height": 1080, "depth": 2, "lights": 4, "soft": False},
        # a program's own incoherent rays against a resident scene: ambient or global illumination queries
        {"name": "trace_closest_1m", "kind": "trace", "form": "batched", "any_hit": False, "tris": 300_000,
         "rays": 1_000_003},
        # a small visibility query through the default path: the smallest call a program makes
        {"name": "trace_any_small", "kind": "trace", "form": "plain", "any_hit": True, "tris": 20_000, "rays": 20_001},
        # many batches of uneven size over several resident scenes, one captured graph per step
        {"name": "batch_64_segments", "kind": "batch", "segments": 64, "scenes": 8, "min_tris": 10_000,
         "max_tris": 300_000, "min_rays": 4096, "max_rays": 1_000_000, "mix": 3, "compress": True},
        # the stage-by-stage calls of a host that keeps its own buffers: one shadow pass at an odd size
        {"name": "stages_shadow", "kind": "stages", "width": 1279, "height": 719, "lights": 3, "grid_bits": 4,
         "dir_log2": 6, "packet": 8},
        # the pair sort alone, on keys that fill their width
        {"name": "sort_16m", "kind": "sort", "n": 16_000_057, "key_bits": 31},
        # a frame of moving objects: per-object transforms, the hierarchies rebuilt, then a frame
        {"name": "moving_soup", "kind": "moving", "size": 1000, "width": 1279, "height": 721, "depth": 1, "lights": 2},
        # a burst of requests of mixed sizes, depths and lights against a running server
        {"name": "serve_16", "kind": "serve", "requests": 16, "scenes": 4, "min_tris": 50_000, "max_tris": 300_000,
         "max_res": 3, "mix": 5},
    ]


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame_size(rng: random.Random, max_width: int) -> tuple[int, int]:
    w = _log_int(rng, 64, max_width)
    return w, max(16, min(1080, int(w * rng.uniform(0.45, 1.1))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["frame", "frame", "frame", "plain", "plain", "trace", "trace", "batch", "stages", "sort",
                       "moving", "serve"])
    if kind in ("frame", "plain"):
        plain = kind == "plain"
        scene = rng.choice(FRAME_SCENES)
        size = {"cornell": 1, "soup": _log_int(rng, 100, 2000), "architecture": rng.randint(8, 40)}[scene]
        soft = rng.random() < 0.2
        w, h = _frame_size(rng, 480 if soft else (1280 if plain else 1920))
        return {"kind": "frame", "form": "plain" if plain else "batched", "scene": scene, "size": size, "width": w,
                "height": h, "depth": rng.randint(1, 2 if plain else 3), "lights": rng.randint(1, 2 if soft else 4),
                "soft": soft}
    if kind == "trace":
        plain = rng.random() < 0.5
        return {"kind": "trace", "form": "plain" if plain else "batched", "any_hit": rng.random() < 0.5,
                "tris": _log_int(rng, 1000, 700_000), "rays": _log_int(rng, 1000, 1_000_000 if plain else 4_000_000)}
    if kind == "batch":
        return {"kind": "batch", "segments": _log_int(rng, 2, 128), "scenes": rng.randint(1, 8),
                "min_tris": 10_000, "max_tris": _log_int(rng, 20_000, 300_000), "min_rays": _log_int(rng, 100, 4096),
                "max_rays": _log_int(rng, 20_000, 1_000_000), "mix": rng.randrange(1 << 20),
                "compress": rng.random() < 0.5}
    if kind == "stages":
        w, h = _frame_size(rng, 1920)
        return {"kind": "stages", "width": w, "height": h, "lights": rng.randint(1, 4), "grid_bits": rng.randint(3, 6),
                "dir_log2": rng.randint(3, 5), "packet": rng.choice([8, 16, 32])}
    if kind == "sort":
        return {"kind": "sort", "n": _log_int(rng, 10_000, 32_000_000), "key_bits": rng.randint(12, 32)}
    if kind == "moving":
        w, h = _frame_size(rng, 1920)
        return {"kind": "moving", "size": _log_int(rng, 50, 2000), "width": w, "height": h, "depth": rng.randint(1, 2),
                "lights": rng.randint(1, 2)}
    return {"kind": "serve", "requests": rng.randint(2, 20), "scenes": rng.randint(1, 4), "min_tris": 20_000,
            "max_tris": 300_000, "max_res": rng.randint(1, 3), "mix": rng.randrange(1 << 20)}


# ------------------------------------------------------------------------------------------- inputs
_geometry: dict = {}


def _scene_data(kind: str, size: int) -> scenes.SceneData:
    """A scene's geometry, as a program loads it from its model files: the same for every seed."""
    key = (kind, size)
    if key not in _geometry:
        if len(_geometry) > 40:
            _geometry.clear()
        if kind == "cornell":
            _geometry[key] = scenes.cornell()
        elif kind == "soup":
            _geometry[key] = scenes.soup(n_spheres=size, extent=50.0 * (size / 2000.0) ** (1.0 / 3.0))
        elif kind == "architecture":
            _geometry[key] = scenes.architecture(grid=size)
        else:
            _geometry[key] = scenes.random_soup(size, np.random.default_rng([7, size]))
    return _geometry[key]


def _materials(s: scenes.SceneData, rng: np.random.Generator) -> np.ndarray:
    m = s.materials.copy()
    m[:, :3] = rng.uniform(0.2, 0.9, (len(m), 3))
    m[:, 3] = rng.uniform(0.0, 1.0, len(m))
    return m


def _view(s: scenes.SceneData, rng: np.random.Generator, w: int, h: int):
    """A camera near the scene's own, and a light set near its lights (more of them between the first two)."""
    reach = float(np.linalg.norm(np.array(s.eye) - np.array(s.target)))
    eye = np.array(s.eye) + rng.normal(0.0, 0.01 * reach, 3)
    target = np.array(s.target) + rng.normal(0.0, 0.01 * reach, 3)
    return rsh.camera_look_at(eye, target, s.up, s.fov, w, h)


def _lights(s: scenes.SceneData, rng: np.random.Generator, count: int) -> list:
    base = s.lights or [{"position": (0.0, 25.0, 0.0)}, {"position": (25.0, 5.0, 25.0)}]
    reach = float(np.linalg.norm(np.array(s.eye) - np.array(s.target)))
    out = []
    for i in range(count):
        l = dict(base[i % len(base)])
        spread = 0.002 if i < len(base) else 0.05
        p = np.array(l["position"], float) + rng.normal(0.0, spread * reach, 3) * np.array([1.0, 0.2, 1.0])
        l["position"] = tuple(p)
        out.append(l)
    return out


def _surface_rays(s: scenes.SceneData, n: int, seed: int, any_hit: bool) -> torch.Tensor:
    """Rays leaving triangle surfaces, uniform on the sphere or mirrored from the eye, half each; [n, 8] float32
    (origin, tmin, direction, tmax). Any-hit rays are bounded, as visibility queries are."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    tri = torch.from_numpy(s.positions).cuda()
    t = torch.randint(0, s.tri_count, (n,), generator=g, device="cuda")
    uv = torch.rand((n, 2), generator=g, device="cuda")
    uv = torch.where(uv.sum(1, keepdim=True) > 1.0, 1.0 - uv, uv)
    v = tri[t][:, :, :3]
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    p = v[:, 0] + e1 * uv[:, :1] + e2 * uv[:, 1:]
    nrm = torch.nn.functional.normalize(torch.linalg.cross(e1, e2), dim=1)
    uni = torch.nn.functional.normalize(torch.randn((n, 3), generator=g, device="cuda"), dim=1)
    view = torch.nn.functional.normalize(p - torch.tensor(s.eye, device="cuda", dtype=torch.float32), dim=1)
    refl = torch.nn.functional.normalize(view - 2.0 * (view * nrm).sum(1, keepdim=True) * nrm, dim=1)
    d = torch.where(torch.rand((n, 1), generator=g, device="cuda") < 0.5, uni, refl)
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 0:3] = p + 0.01 * d
    rays[:, 3] = 0.01
    rays[:, 4:7] = d
    rays[:, 7] = 0.1 + 10.0 * torch.rand(n, generator=g, device="cuda") if any_hit else math.inf
    return rays


def _mixed_sizes(case: dict) -> list:
    """The batch case's segments: (scene index, rays, any hit), sizes spread over their logarithm."""
    r = random.Random(case["mix"])
    return [(r.randrange(case["scenes"]), _log_int(r, case["min_rays"], case["max_rays"]), r.random() < 0.5)
            for _ in range(case["segments"])]


def _mixed_tris(case: dict) -> list:
    r = random.Random(case["mix"] + 1)
    return [_log_int(r, case["min_tris"], case["max_tris"]) for _ in range(case["scenes"])]


def _requests(case: dict) -> list:
    """The serve case's requests: (scene index, width, height, depth, lights)."""
    r = random.Random(case["mix"] + 2)
    sizes = [(256, 256), (512, 512), (1920, 1080)][: case["max_res"]]
    return [(r.randrange(case["scenes"]), *r.choice(sizes), r.randint(1, 3), r.randint(1, 4))
            for _ in range(case["requests"])]


class State:
    """What a program keeps between calls: its context, scenes, buffers, and a graph or a server."""

    def __init__(self, case: dict, **config):
        self.case = case
        self.ctx = rsh.Context(rsh.default_config(**config))
        self.scenes = []
        self.graph = None
        self.graph_stream = None
        self.server = None

    def scene(self, s: scenes.SceneData, materials: np.ndarray, object_ids=None):
        self.scenes.append(self.ctx.scene(s.positions, s.normals, s.material_ids, materials, object_ids))
        return self.scenes[-1]

    def __del__(self):
        lib = rsh.lib()
        if self.server:
            lib.rsh_server_destroy(self.server)
        if self.graph:
            lib.rsh_batch_graph_destroy(self.graph)
        if self.graph_stream:
            lib.rsh_stream_destroy(self.graph_stream)
        for sc in self.scenes:
            sc.destroy()
        self.ctx.destroy()


def _prepare_frame(case: dict, seed: int, moving: bool = False) -> State:
    rng = np.random.default_rng([seed, 1])
    s = _scene_data("soup" if moving else case["scene"], case["size"])
    flags = rsh.FLAG_FUSED if moving or case["form"] == "batched" else 0
    if not moving and case["soft"]:
        flags |= rsh.FLAG_SOFT_SHADOWS
    st = State(case, flags=flags, reflect_jitter=float(s.jitter), seed=seed & 0xFFFFFFFF)
    ids = None
    if moving:
        # one object per sphere; the ground is one more
        per = scenes.icosphere(2)[1].shape[0]
        ids = np.minimum(np.arange(s.tri_count) // per, case["size"]).astype(np.uint32)
        k = case["size"] + 1
        # a rotation about the vertical, a uniform scale and a displacement per object (small against the
        # scene: objects move about their places)
        a, c = rng.uniform(0.0, 0.1, k), rng.uniform(0.98, 1.02, k)
        m = np.zeros((k, 4, 4), np.float32)
        m[:, 0, 0] = m[:, 2, 2] = c * np.cos(a)
        m[:, 0, 2] = c * np.sin(a)
        m[:, 2, 0] = -c * np.sin(a)
        m[:, 1, 1] = c
        m[:, :3, 3] = rng.normal(0.0, 0.5, (k, 3))
        m[:, 3, 3] = 1.0
        m[-1] = np.eye(4, dtype=np.float32)
        st.model = m
    st.scene(s, _materials(s, rng), ids)
    st.ctx.set_camera(_view(s, rng, case["width"], case["height"]))
    st.ctx.set_lights(_lights(s, rng, case["lights"]))
    st.rgba = torch.zeros((case["height"], case["width"], 4), dtype=torch.uint8, device="cuda")
    return st


def _prepare_trace(case: dict, seed: int) -> State:
    rng = np.random.default_rng([seed, 2])
    st = State(case)
    s = _scene_data("random_soup", case["tris"])
    st.scene(s, _materials(s, rng))
    st.rays = _surface_rays(s, case["rays"], seed, case["any_hit"])
    st.out = torch.zeros(case["rays"], dtype=torch.int32 if case["any_hit"] else torch.int64, device="cuda")
    return st


def _prepare_batch(case: dict, seed: int) -> State:
    rng = np.random.default_rng([seed, 3])
    st = State(case, flags=0 if case["compress"] else rsh.FLAG_NO_COMPRESS)
    data = [_scene_data("random_soup", t) for t in _mixed_tris(case)]
    for s in data:
        st.scene(s, _materials(s, rng))
    segs = _mixed_sizes(case)
    st.hits = torch.zeros(sum(n for _, n, a in segs if not a), dtype=torch.int64, device="cuda")
    st.flags = torch.zeros(sum(n for _, n, a in segs if a), dtype=torch.int32, device="cuda")
    st.rays = [_surface_rays(data[w], n, seed + 977 * i, a) for i, (w, n, a) in enumerate(segs)]
    st.segments = (rsh.BatchSegment * len(segs))()
    at = [0, 0]
    for i, (w, n, a) in enumerate(segs):
        b = st.segments[i]
        b.scene, b.rays, b.n, b.any_hit = st.scenes[w].handle, st.rays[i].data_ptr(), n, int(a)
        b.hits = None if a else st.hits.data_ptr() + 8 * at[0]
        b.flags = st.flags.data_ptr() + 4 * at[1] if a else None
        at[int(a)] += n
    torch.cuda.synchronize()
    stream, graph = C.c_void_p(), C.c_void_p()
    rsh.check(rsh.lib().rsh_stream_create(C.byref(stream)), "rsh_stream_create")
    st.graph_stream = stream
    rsh.check(rsh.lib().rsh_batch_graph_create(st.ctx.handle, st.segments, len(segs), stream, C.byref(graph)),
              "rsh_batch_graph_create")
    st.graph = graph
    return st


def _surface(case: dict, seed: int):
    """A pass's surface buffer: bumpy ground seen by a camera, one pixel in sixteen empty; [h, w, 4] each."""
    w, h = case["width"], case["height"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    ph = torch.rand(4, generator=g, device="cuda") * 6.28
    x = torch.linspace(-50.0, 50.0, w, device="cuda")[None, :].expand(h, w)
    z = torch.linspace(-50.0, 50.0, h, device="cuda")[:, None].expand(h, w)
    y = 2.0 * torch.sin(0.21 * x + ph[0]) * torch.cos(0.17 * z + ph[1]) + 0.3 * torch.sin(1.3 * x + ph[2])
    dx = 0.42 * torch.cos(0.21 * x + ph[0]) * torch.cos(0.17 * z + ph[1]) + 0.39 * torch.cos(1.3 * x + ph[2])
    dz = -0.34 * torch.sin(0.21 * x + ph[0]) * torch.sin(0.17 * z + ph[1])
    some = (torch.rand((h, w), generator=g, device="cuda") < 15.0 / 16.0).float()
    pos = torch.stack([x, y, z, torch.ones_like(x)], 2) * some[:, :, None]
    nrm = torch.stack([-dx, torch.ones_like(x), -dz, torch.zeros_like(x)], 2) * some[:, :, None]
    r = random.Random(seed)
    lights = [{"position": (r.uniform(-40, 40), r.uniform(8, 30), r.uniform(-40, 40))} for _ in range(case["lights"])]
    return pos.contiguous(), nrm.contiguous(), lights


_EPS = 0.01


def _prepare_stages(case: dict, seed: int) -> State:
    st = State(case)
    st.pos, st.nrm, lights = _surface(case, seed)
    st.lights = rsh.make_lights(lights)
    st.n = n = case["width"] * case["height"] * case["lights"]
    tag_bits = max(0, (case["lights"] - 1).bit_length())
    st.hp = rsh.hash_params((-50.0, -3.0, -50.0), (50.0, 30.0, 50.0), case["grid_bits"], case["dir_log2"], tag_bits)
    off = (C.c_uint32 * 4)()
    nodes = rsh.lib().rsh_hierarchy_capacity(n, case["packet"], off)
    ints = lambda k: torch.zeros(k, dtype=torch.int32, device="cuda")  # noqa: E731
    st.rays = torch.zeros((n, 8), device="cuda")
    st.keys, st.trimmed, st.ckeys, st.cbases = ints(n), ints(n), ints(n + 1), ints(n + 1)
    st.counts, st.skeys, st.svals, st.sorted_keys, st.sorted_ids = ints(2), ints(n), ints(n), ints(n), ints(n)
    st.nodes = torch.zeros((nodes, 12), device="cuda")
    return st


def _prepare_sort(case: dict, seed: int) -> State:
    st = State(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, bits = case["n"], case["key_bits"]
    k = torch.randint(0, 1 << bits, (n,), generator=g, device="cuda", dtype=torch.int64)
    st.keys = torch.where(k >= 1 << 31, k - (1 << 32), k).to(torch.int32)  # the same 32 bits
    st.keys_out = torch.zeros(n, dtype=torch.int32, device="cuda")
    st.vals_out = torch.zeros(n, dtype=torch.int32, device="cuda")
    return st


def _prepare_serve(case: dict, seed: int) -> State:
    rng = np.random.default_rng([seed, 5])
    st = State(case)
    data = [_scene_data("random_soup", t) for t in _mixed_tris(case)]
    for s in data:
        st.scene(s, _materials(s, rng))
    handles = (C.c_void_p * len(st.scenes))(*[s.handle for s in st.scenes])
    srv = C.c_void_p()
    rsh.check(rsh.lib().rsh_server_create(st.ctx.handle, handles, len(st.scenes), 16 << 30, 64, C.byref(srv)),
              "rsh_server_create")
    st.server = srv
    st.requests, st.hits, st.flags = [], [], []
    for w, width, height, depth, lights in _requests(case):
        s = data[w]
        q = rsh.Request()
        q.scene_index, q.width, q.height, q.depth, q.light_count = w, width, height, depth, lights
        q.camera = _view(s, rng, width, height)
        for i, l in enumerate(rsh.make_lights(_lights(s, rng, lights))):
            q.lights[i] = l
        st.requests.append(q)
        n = width * height * depth
        st.hits.append(torch.zeros(n, dtype=torch.int64, pin_memory=True))
        st.flags.append(torch.zeros(n * lights, dtype=torch.int32, pin_memory=True))
    return st


def prepare(case: dict, seed: int) -> State:
    kind = case["kind"]
    if kind in ("frame", "moving"):
        return _prepare_frame(case, seed, kind == "moving")
    return {"trace": _prepare_trace, "batch": _prepare_batch, "stages": _prepare_stages, "sort": _prepare_sort,
            "serve": _prepare_serve}[kind](case, seed)


# ------------------------------------------------------------------------------------------- one pass
def run(st: State):
    lib, case, ctx = rsh.lib(), st.case, st.ctx
    kind = case["kind"]
    stream = torch.cuda.current_stream().cuda_stream or None
    if kind == "frame":
        ctx.render(st.scenes[0], case["width"], case["height"], case["depth"], st.rgba.data_ptr(), stream)
        return st.rgba
    if kind == "moving":
        st.scenes[0].set_transforms(st.model, None, stream)
        ctx.render(st.scenes[0], case["width"], case["height"], case["depth"], st.rgba.data_ptr(), stream)
        return st.rgba
    if kind == "trace":
        call = lib.rsh_trace_rays_fused if case["form"] == "batched" else lib.rsh_trace_rays
        out = st.out.data_ptr()
        any_hit = int(case["any_hit"])
        rsh.check(call(ctx.handle, st.scenes[0].handle, st.rays.data_ptr(), case["rays"], any_hit,
                       None if any_hit else out, out if any_hit else None, stream), "trace")
        return st.out
    if kind == "batch":
        rsh.check(lib.rsh_batch_graph_launch(st.graph, stream), "rsh_batch_graph_launch")
        return {"hits": st.hits, "flags": st.flags}
    if kind == "stages":
        p = lambda t: t.data_ptr()  # noqa: E731
        n, hp = st.n, C.byref(st.hp)
        rsh.check(lib.rsh_raygen_shadow(p(st.pos), p(st.nrm), case["width"], case["height"], st.lights, case["lights"],
                                        _EPS, hp, p(st.rays), p(st.keys), stream), "rsh_raygen_shadow")
        rsh.check(lib.rsh_compress(ctx.handle, p(st.keys), n, p(st.trimmed), p(st.ckeys), p(st.cbases), None,
                                   p(st.counts), stream), "rsh_compress")
        rsh.check(lib.rsh_sort_pairs(ctx.handle, p(st.ckeys), None, p(st.skeys), p(st.svals), n, p(st.counts) + 4,
                                     st.hp.key_bits, stream), "rsh_sort_pairs")
        rsh.check(lib.rsh_decompress(ctx.handle, p(st.skeys), p(st.svals), p(st.cbases), p(st.trimmed), p(st.counts),
                                     n, p(st.sorted_keys), p(st.sorted_ids), stream), "rsh_decompress")
        rsh.check(lib.rsh_build_rsh(p(st.rays), p(st.sorted_ids), n, p(st.counts), case["packet"], p(st.nodes),
                                    stream), "rsh_build_rsh")
        return {"rays": st.rays, "keys": st.keys, "counts": st.counts, "sorted_keys": st.sorted_keys,
                "sorted_ids": st.sorted_ids, "node_bounds": st.nodes[:, :10],
                "node_ranges": st.nodes[:, 10:].view(torch.int32)}
    if kind == "sort":
        rsh.check(lib.rsh_sort_pairs(ctx.handle, st.keys.data_ptr(), None, st.keys_out.data_ptr(),
                                     st.vals_out.data_ptr(), case["n"], None, case["key_bits"], stream),
                  "rsh_sort_pairs")
        return {"keys": st.keys_out, "values": st.vals_out}
    ids = []
    for q in st.requests:
        i = C.c_uint64()
        rsh.check(lib.rsh_server_submit(st.server, C.byref(q), C.byref(i)), "rsh_server_submit")
        ids.append(i.value)
    rays = []
    for i, hits, flags in zip(ids, st.hits, st.flags):
        res = rsh.RequestResult()
        rsh.check(lib.rsh_server_wait(st.server, i, 60_000, C.byref(res), hits.data_ptr(), flags.data_ptr()),
                  "rsh_server_wait")
        rays.append(int(res.rays))
    return {"hits": st.hits, "flags": st.flags, "rays": np.array(rays, np.int64)}


# ------------------------------------------------------------------------------------------- what it takes
def _ray_flops(rays: float, tris: float) -> float:
    """One path down an 8-wide tree with clusters of six (24 flops per box, 46 per triangle)."""
    return rays * (24.0 * 8.0 * max(1.0, math.ceil(math.log(max(tris / 6.0, 1.0)) / math.log(8.0))) + 6.0 * 46.0)


def _scene_tris(kind: str, size: int) -> float:
    if kind == "cornell":
        return 2580.0
    if kind == "soup":
        return 320.0 * size + 32.0
    if kind == "architecture":
        return 544.0 * size * size + 40_000.0 + 64.0 * size * (size - 1)
    return float(size)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("frame", "moving"):
        tris = _scene_tris(case.get("scene", "soup"), case["size"])
        npix = case["width"] * case["height"]
        # every pixel's ray, and half of the shadow and reflection slots of each bounce holding a ray
        rays = npix * (1.0 + 0.5 * case["depth"] * (1.0 + case["lights"] * (16 if case.get("soft") else 1)))
        move = 192.0 * tris if kind == "moving" else 0.0  # rest pose in, pose out, positions and normals
        return {"bytes": 100.0 * tris + move + 4.0 * npix, "flops": _ray_flops(rays, tris)}
    if kind == "trace":
        n = case["rays"]
        return {"bytes": 48.0 * case["tris"] + n * (32.0 + (4.0 if case["any_hit"] else 8.0)),
                "flops": _ray_flops(n, case["tris"])}
    if kind == "batch":
        tris = _mixed_tris(case)
        segs = _mixed_sizes(case)
        return {"bytes": 48.0 * sum(tris) + sum(n * (36.0 if a else 40.0) for _, n, a in segs),
                "flops": sum(_ray_flops(n, tris[w]) for w, n, _ in segs)}
    if kind == "stages":
        npix = case["width"] * case["height"]
        n = npix * case["lights"]
        # surfaces in; rays, keys, sorted keys and ids out; a 48-byte node per packet and its parents
        return {"bytes": 32.0 * npix + n * (32.0 + 12.0) + 48.0 * 1.15 * n / case["packet"], "flops": 60.0 * n}
    if kind == "sort":
        return {"bytes": 12.0 * case["n"], "flops": 0.0}
    tris = _mixed_tris(case)
    b = f = 0.0
    for w, width, height, depth, lights in _requests(case):
        npix = width * height
        b += depth * npix * (8.0 + 4.0 * lights)
        f += _ray_flops(npix * (1.0 + 0.5 * depth * (1.0 + lights)), tris[w])
    return {"bytes": b + 48.0 * sum(tris), "flops": f}


def exact(case: dict, seed: int):
    """The stage case's rays in 64 bits. Everything else that a pass returns is whole: hit records, flags, keys,
    orders and 8-bit images; the hierarchy's nodes follow the 32-bit keys' order."""
    if case["kind"] != "stages":
        return None
    pos, nrm, lights = _surface(case, seed)
    pos, nrm = pos.double(), nrm.double()
    h, w, L = case["height"], case["width"], case["lights"]
    eps = float(np.float32(_EPS))
    rays = torch.zeros((h, L, w, 8), dtype=torch.float64, device="cuda")
    rays[..., 7] = -1.0
    some = pos[:, :, 3] != 0.0
    for i, l in enumerate(lights):
        lp = torch.tensor(np.array(l["position"], np.float32).astype(np.float64), device="cuda")
        v = pos[:, :, :3] - lp
        dist = v.norm(dim=2)
        d = v / dist[:, :, None]
        ok = some & (-(d * nrm[:, :, :3]).sum(2) > 0.0) & (dist - 2.0 * eps > eps)
        r = torch.cat([lp + d * eps, torch.full_like(dist, eps)[:, :, None], d, (dist - 2.0 * eps)[:, :, None]], 2)
        rays[:, i] = torch.where(ok[:, :, None], r, rays[:, i])
    return {"rays": rays.reshape(-1, 8), "keys": None, "counts": None, "sorted_keys": None, "sorted_ids": None,
            "node_bounds": None, "node_ranges": None}
