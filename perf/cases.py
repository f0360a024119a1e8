"""The workloads this library is timed on, through its public entry points.

A case is a dict of plain values; `kind` says which path it takes:

  pick     a click: st_pick of one pixel
  frame    one view: (optionally st_upload_primitives, then) st_render_ex, outputs in page-locked
           host memory or in device memory
  moving   one frame of an animated scene: st_update_primitives of the moved primitives, the TLAS
           rebuilt or refit by st_update_scene_bvh, then (optionally) the view rendered
  blas     a mesh made ready for rendering: updateMeshBVH of host arrays
  batch    several views of several resident scenes in one st_render_batch call
  serve    a burst of requests, each with a transform update, through the serving loop
  texture  an image baked into the mip-chained texel-quad layout

Scenes have the shapes and distributions of slimtracin_b200/scenes.py (every draw comes from the
seed); the meshes are icospheres displaced by seeded waves, cheap enough to make many times.
Calls go to the C ABI with arguments built beforehand, as a C host's own loop would make them.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from slimtracin_b200 import api, mixed, scenes, structs as S

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"      # where exact() works
MODES = {"beauty": S.RM_BEAUTY, "depth": S.RM_DEPTH, "normals": S.RM_NORMALS}
BUILDS = {"lbvh": api.ST_BVH_LBVH30, "sah": api.ST_BVH_BINNED_SAH, "refit": api.ST_BVH_REFIT}


def listed():
    return [
        # a click in an editor on the 16-primitive scene: the smallest call there is
        {"name": "pick_16", "kind": "pick", "prims": 16, "width": 640, "height": 480},
        # the drop-in renderScene of a small scene at the window size of the reference's examples,
        # float grid and pixels into the host's frame buffers
        {"name": "frame_implicit_host", "kind": "frame", "scene": "implicit", "size": 16, "width": 640, "height": 480,
         "depth": 2, "mode": "beauty", "cone": False, "out": "host", "upload": False},
        # the full-size frame end to end: primitives uploaded, 1080p PBR mesh scene (1.31 M triangles in
        # 8 instances, glass and mirrors, depth 4), grid and pixels into page-locked host memory
        {"name": "frame_mesh_host", "kind": "frame", "scene": "mesh", "size": 8, "width": 1920, "height": 1080,
         "depth": 4, "mode": "beauty", "cone": False, "out": "host", "upload": True},
        # the same frame kept on the device (an encoder or a denoiser reads it there)
        {"name": "frame_mesh_device", "kind": "frame", "scene": "mesh", "size": 8, "width": 1920, "height": 1080,
         "depth": 4, "mode": "beauty", "cone": False, "out": "device", "upload": False},
        # an odd-sized preview of a small mesh with ray-cone mip selection and deep glass
        {"name": "frame_mesh_odd", "kind": "frame", "scene": "mesh", "size": 5, "width": 1001, "height": 563,
         "depth": 6, "mode": "beauty", "cone": True, "out": "device", "upload": False},
        # every frame of an animation of 4096 primitives: all records, LBVH rebuild, 720p view
        {"name": "moving_lbvh", "kind": "moving", "prims": 4096, "moved": 4096, "build": "lbvh", "width": 1280,
         "height": 720, "depth": 2, "render": True},
        # the better tree for the same scene, built once per edit and read back by the host
        {"name": "tlas_sah", "kind": "moving", "prims": 4096, "moved": 4096, "build": "sah", "width": 0, "height": 0,
         "depth": 0, "render": False},
        # a few objects dragged in a scene of ordinary size: refit only
        {"name": "tlas_refit", "kind": "moving", "prims": 1000, "moved": 37, "build": "refit", "width": 0, "height": 0,
         "depth": 0, "render": False},
        # a mesh of the middle size ingested with the better tree
        {"name": "blas_sah", "kind": "blas", "triangles": 327680, "build": "sah"},
        # many views of several scenes at once (thumbnails, a dataset): sizes and depths mixed
        {"name": "batch_views", "kind": "batch", "views": 16, "mesh_size": 6, "prims": 512, "launch": "per_view"},
        # a burst of interactive clients over two scenes, frames to the host
        {"name": "serve_burst", "kind": "serve", "requests": 24, "prims": 1024, "max_moved": 64},
        # a photograph baked for the renderer
        {"name": "texture_1024", "kind": "texture", "width": 1024, "height": 1024, "bits": 24, "wrap": True, "mipmap": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pick", "frame", "frame", "frame", "moving", "moving", "blas", "batch", "serve", "texture"])
    if kind == "pick":
        return {"kind": kind, "prims": _log_int(rng, 16, 4096), "width": rng.randrange(160, 1921),
                "height": rng.randrange(120, 1081)}
    if kind == "frame":
        scene = rng.choice(["implicit", "mesh", "mesh"])
        return {"kind": kind, "scene": scene, "size": rng.randrange(4, 9) if scene == "mesh" else _log_int(rng, 16, 512),
                "width": _log_int(rng, 160, 1920), "height": _log_int(rng, 120, 1080), "depth": rng.randrange(1, 5),
                "mode": rng.choice(["beauty", "beauty", "beauty", "depth", "normals"]), "cone": rng.random() < 0.3,
                "out": rng.choice(["host", "device"]), "upload": rng.random() < 0.5}
    if kind == "moving":
        n, render = _log_int(rng, 65, 4096), rng.random() < 0.5
        return {"kind": kind, "prims": n, "moved": _log_int(rng, 1, n), "build": rng.choice(["lbvh", "sah", "refit"]),
                "width": rng.randrange(160, 1281) if render else 0, "height": rng.randrange(120, 721) if render else 0,
                "depth": 2 if render else 0, "render": render}
    if kind == "blas":
        return {"kind": kind, "triangles": _log_int(rng, 500, 327680), "build": rng.choice(["lbvh", "sah"])}
    if kind == "batch":
        return {"kind": kind, "views": rng.randrange(2, 17), "mesh_size": rng.randrange(4, 7), "prims": _log_int(rng, 16, 512),
                "launch": rng.choice(["per_view", "persistent"])}
    if kind == "serve":
        return {"kind": kind, "requests": rng.randrange(2, 25), "prims": _log_int(rng, 16, 1024),
                "max_moved": rng.randrange(0, 65)}
    return {"kind": kind, "width": _log_int(rng, 16, 1024), "height": _log_int(rng, 16, 1024), "bits": rng.choice([24, 32]),
            "wrap": rng.random() < 0.5, "mipmap": rng.random() < 0.8}


# ---- scenes from a seed --------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sphere(size):
    v, f = scenes.icosphere(size)
    return v, f.astype(np.uint32)


def _mesh(seed, size, triangles=None, radius=2.5):
    """A displaced icosphere of subdivision `size` (its first `triangles` faces): area-weighted
    normals, spherical uvs, centred on its box."""
    unit, f = _sphere(size)
    if triangles is not None:
        f = np.ascontiguousarray(f[:triangles])
    rng = np.random.default_rng(seed)
    r = np.ones(len(unit))
    for octave in (3.0, 6.0, 12.0, 24.0):
        r += 0.15 / octave * np.sin(octave * (unit @ rng.normal(size=3)) + rng.uniform(0, 2 * math.pi))
    v = radius * unit * r[:, None]
    fn = np.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])
    corner = f.ravel()
    vn = np.stack([np.bincount(corner, np.repeat(fn[:, k], 3), len(v)) for k in range(3)], 1)
    length = np.linalg.norm(vn, axis=1, keepdims=True)
    vn = np.where(length > 0, vn / np.maximum(length, 1e-30), unit)
    uv = np.stack([0.5 + np.arctan2(unit[:, 2], unit[:, 0]) / (2 * math.pi),
                   0.5 - np.arcsin(np.clip(unit[:, 1], -1, 1)) / math.pi], 1)
    p = (v - (v.min(0) + v.max(0)) / 2).astype(np.float32)
    box = np.concatenate([p.min(0), p.max(0)])
    return scenes.MeshData(p, vn.astype(np.float32), uv.astype(np.float32), f, box)


def _images(seed, width, height):
    """A smooth colour image and a normal map of its relief, 8 bits."""
    g = torch.Generator().manual_seed(seed)
    grid = torch.rand((1, 3, 17, 17), generator=g)
    img = torch.nn.functional.interpolate(grid, size=(height, width), mode="bilinear", align_corners=True)[0].numpy()
    relief = img[0] * 8.0
    gy, gx = np.gradient(relief) if min(relief.shape) > 1 else (relief * 0, relief * 0)
    n = np.stack([-gx, -gy, np.ones_like(relief)], -1)
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    colour = (np.moveaxis(img, 0, -1) * 255).astype(np.uint8)
    return np.ascontiguousarray(colour), np.ascontiguousarray(((n * 0.5 + 0.5) * 255).astype(np.uint8))


def _bake(renderer, image, wrap, mipmap, memory=None):
    h, w, channels = image.shape
    need = renderer.L.st_texture_bytes(w, h, int(mipmap))
    memory = np.zeros(need, np.uint8) if memory is None else memory
    tex = S.Texture()
    renderer._check(renderer.L.st_bake_texture(renderer.ctx, image.ctypes.data, w, h, 8 * channels, int(wrap), int(mipmap),
                                               C.byref(tex), memory.ctypes.data, need), "st_bake_texture")
    return tex, memory


def _texture(renderer, image):
    tex, memory = _bake(renderer, image, True, True)
    mips, base = [], memory.ctypes.data
    for k in range(tex.mip_count):
        m = tex.mips[k]
        count = (m.width + 1) * (m.height + 1)
        at = (m.texel_quads if isinstance(m.texel_quads, int) else C.cast(m.texel_quads, C.c_void_p).value) - base
        mips.append((m.width, m.height, memory[at:at + 12 * count].view(S.TEXELQUAD_DT)))
    return scenes.TextureData(tex.width, tex.height, True, True, mips)


def _implicit(seed, count):
    """`count` implicit primitives; up to 64 as the 16-primitive scene spreads them."""
    if count == 16:
        return scenes.implicit16_scene(seed_offset=seed)
    return scenes.moving_scene(seed_offset=seed, count=count)


def _mesh_scene(renderer, seed, size):
    sd, cam = scenes.mesh_scene(seed_offset=seed, subdivisions=0, texture_size=16)
    sd.meshes = [_mesh(seed, size)]
    sd.textures = [_texture(renderer, image) for image in _images(seed, 1024, 1024)]
    return sd, cam


def _resident(renderer, slot, sd):
    """Upload the scene with the trees a host builds once: binned SAH."""
    for md in sd.meshes:
        renderer.build_blas(md, api.ST_BVH_BINNED_SAH)
    renderer.upload(slot, sd, tlas=None)
    renderer.build_tlas(slot, sd, api.ST_BVH_BINNED_SAH)


def _outputs(width, height, on_device):
    """A frame's float grid and pixels, page-locked or on the device, and the parts of the grid."""
    where = {"device": "cuda"} if on_device else {"pin_memory": True}
    grid = torch.empty((height + 1, width + 1, 6), dtype=torch.float32, **where)
    pixels = torch.empty((height, width, 4), dtype=torch.uint8, **where)
    return grid, pixels


def _grid_parts(grid):
    return {"color": grid[..., :4], "depth": grid.view(torch.float64)[..., 2]}


def _frame(width, height, cam, depth, mode="beauty", cone=False):
    angle = math.atan(2.0 / (height * cam.focal_length)) if cone else 0.0
    return scenes.Frame(width, height, cam, depth=depth, mode=MODES[mode], cone_angle=angle, with_pixels=False,
                        with_float=False)


class State:
    def __init__(self, case, max_scenes=1):
        self.case = case
        self.renderer = api.Renderer(0, max_scenes=max_scenes)
        self.L, self.ctx = self.renderer.L, self.renderer.ctx

    def check(self, status, what):
        if status:
            self.renderer._check(status, what)


def _render_options(st, grid, pixels, on_device):
    o = api.st_render_options()
    o.device_outputs = int(on_device)
    o.out_float, o.out_u8 = grid.data_ptr(), pixels.data_ptr()
    return o


def _clicked(case, seed):
    """The pixel clicked on: somewhere in the middle of the frame."""
    rng = np.random.default_rng(seed)
    return [int(side * rng.uniform(0.35, 0.65)) for side in (case["width"], case["height"])]


def _prepare_pick(case, seed):
    st = State(case)
    st.sd, cam = _implicit(seed, case["prims"])
    _resident(st.renderer, 0, st.sd)
    st.sc, st.keep = st.sd.to_ctypes()
    st.frame = _frame(case["width"], case["height"], cam, 1)
    st.x, st.y = _clicked(case, seed)
    st.result = api.st_pick_result()
    return st


def _run_pick(st):
    st.check(st.L.st_pick(st.ctx, 0, C.byref(st.sc), C.byref(st.frame.viewport), st.x, st.y, C.byref(st.result)), "st_pick")
    r = st.result
    return {"found": r.found, "type": r.object_type, "id": r.object_id,
            "position": np.array(r.position[:], np.float32), "distance": np.float32(r.distance),
            "object_distance": np.float32(r.object_distance)}


def _scene_of(case, seed, renderer=None):
    if case["scene"] == "mesh":
        return _mesh_scene(renderer, seed, case["size"])
    return _implicit(seed, case["size"])


def _prepare_frame(case, seed):
    st = State(case)
    st.sd, cam = _scene_of(case, seed, st.renderer)
    _resident(st.renderer, 0, st.sd)
    st.sc, st.keep = st.sd.to_ctypes()
    st.frame = _frame(case["width"], case["height"], cam, case["depth"], case["mode"], case["cone"])
    device = case["out"] == "device"
    st.grid, st.pixels = _outputs(case["width"], case["height"], device)
    st.options = _render_options(st, st.grid, st.pixels, device)
    return st


def _run_frame(st):
    if st.case["upload"]:
        st.check(st.L.st_upload_primitives(st.ctx, 0, C.byref(st.sc)), "st_upload_primitives")
    st.check(st.L.st_render_ex(st.ctx, 0, C.byref(st.sc), C.byref(st.frame.viewport), C.byref(st.options)), "st_render_ex")
    return dict(_grid_parts(st.grid), pixels=st.pixels)


def _prepare_moving(case, seed):
    st = State(case)
    st.sd, cam = _implicit(seed, case["prims"])
    _resident(st.renderer, 0, st.sd)
    rng = np.random.default_rng(seed)
    st.ids = np.sort(rng.choice(case["prims"], case["moved"], replace=False)).astype(np.uint32)
    moved = st.sd.primitives.copy()
    moved["position"] += rng.uniform(-0.05, 0.05, (case["prims"], 3)).astype(np.float32)
    st.records = np.ascontiguousarray(moved[st.ids])
    st.sc, st.keep = st.sd.to_ctypes()
    if case["render"]:
        st.frame = _frame(case["width"], case["height"], cam, case["depth"])
        st.grid, st.pixels = _outputs(case["width"], case["height"], True)
        st.options = _render_options(st, st.grid, st.pixels, True)
    return st


def _run_moving(st):
    st.check(st.L.st_update_primitives(st.ctx, 0, st.records.ctypes.data, st.ids.ctypes.data, len(st.ids)),
             "st_update_primitives")
    # a host that renders leaves the tree on the device; one that only rebuilds reads it back
    scene = None if st.case["render"] else C.byref(st.sc)
    st.check(st.L.st_update_scene_bvh(st.ctx, 0, scene, BUILDS[st.case["build"]]), "st_update_scene_bvh")
    if not st.case["render"]:
        return {"nodes": st.sd.tlas_nodes.view(np.uint8), "count": int(st.sc.bvh.node_count),
                "leaf_ids": st.sd.tlas_leaf_ids.view(np.int32), "height": int(st.sc.bvh.height)}
    st.check(st.L.st_render_ex(st.ctx, 0, C.byref(st.sc), C.byref(st.frame.viewport), C.byref(st.options)), "st_render_ex")
    return dict(_grid_parts(st.grid), pixels=st.pixels)


def _prepare_blas(case, seed):
    st = State(case)
    size = next(s for s in range(16) if 20 * 4 ** s >= case["triangles"])
    st.mesh = _mesh(seed, size, case["triangles"])
    st.mesh.allocate_bvh()
    st.keep = []
    st.struct = st.mesh.to_ctypes(st.keep)
    return st


def _run_blas(st):
    st.check(st.L.st_update_mesh_bvh(st.ctx, C.byref(st.struct), BUILDS[st.case["build"]]), "st_update_mesh_bvh")
    m = st.mesh
    return {"nodes": m.nodes.view(np.uint8), "count": int(st.struct.bvh.node_count), "leaf_ids": m.leaf_ids.view(np.int32),
            "triangles": m.triangles.view(np.uint8), "height": int(st.struct.bvh.height)}


def _view_size(k):
    """The size of the k-th view of a batch or burst: 256x256 to 1280x720, every other one odd."""
    width, height = mixed.RESOLUTIONS[(k * 2 + k // 3) % 3]
    return width - (k % 2) * (k % 8), height - (k % 2) * (k % 5)


def _prepare_batch(case, seed):
    st = State(case, max_scenes=3)
    data = [_implicit(seed, 16)[0], _mesh_scene(st.renderer, seed, case["mesh_size"])[0],
            _implicit(seed + 1, case["prims"])[0]]
    orbits = [((0.0, 0.0, 0.0), 15.0, 2.0), ((0.0, 1.5, 0.0), 15.0, 8.0), ((0.0, 0.0, 0.0), 20.0, 3.0)]
    st.residents = [mixed.Resident(sd.name, sd, *orbit, "sah") for sd, orbit in zip(data, orbits)]
    slots = mixed.upload(st.renderer, st.residents)
    rng = np.random.default_rng(seed)
    items, st.grids, st.frames = [], [], []
    for k in range(case["views"]):
        i = k % 3
        width, height = _view_size(k)
        frame = _frame(width, height, mixed.random_camera(rng, st.residents[i]), 1 + k % 5)
        items.append((slots[i], st.residents[i], frame))
        st.grids.append(_outputs(frame.width, frame.height, True))
    fixed = {"launch_mode": api.LAUNCH_PER_VIEW} if case["launch"] == "per_view" else \
        {"launch_mode": api.LAUNCH_PERSISTENT, "tile_shape": 0, "chunk": 1, "stack_placement": 0, "compaction_threshold": 0}
    st.batch = mixed.Batch(st.renderer, items, [g.data_ptr() for g, _ in st.grids], [p.data_ptr() for _, p in st.grids],
                           **fixed)
    return st


def _run_batch(st):
    st.batch.run()
    return [dict(_grid_parts(grid), pixels=pixels) for grid, pixels in st.grids]


def _prepare_serve(case, seed):
    st = State(case, max_scenes=2)
    data = [_mesh_scene(st.renderer, seed, 5)[0], _implicit(seed, case["prims"])[0]]
    orbits = [((0.0, 1.5, 0.0), 15.0, 8.0), ((0.0, 0.0, 0.0), 20.0, 3.0)]
    st.residents = [mixed.Resident(sd.name, sd, *orbit, "sah") for sd, orbit in zip(data, orbits)]
    slots = mixed.upload(st.renderer, st.residents)
    rng = np.random.default_rng(seed)
    st.requests, st.pixels, st.keep = [], [], []
    for k in range(case["requests"]):
        i = k % 2
        width, height = _view_size(k)
        frame = _frame(width, height, mixed.random_camera(rng, st.residents[i]), 1 + k % 4)
        records, ids = mixed.random_update(rng, st.residents[i], max_count=case["max_moved"])
        pixels = torch.empty((height, width, 4), dtype=torch.uint8, pin_memory=True)
        req = api.st_request()
        req.view.slot = slots[i]
        req.view.scene, req.view.viewport = C.addressof(st.residents[i].sc), C.addressof(frame.viewport)
        req.view.out_u8 = pixels.data_ptr()
        if records is not None:
            req.moved, req.moved_ids, req.moved_count = records.ctypes.data, ids.ctypes.data, len(ids)
        st.requests.append(req)
        st.pixels.append(pixels)
        st.keep.append((frame, records, ids))
    st.tickets = (C.c_uint64 * case["requests"])()
    st.server = api.Server(st.renderer)
    return st


def _run_serve(st):
    size, result = C.sizeof(C.c_uint64), api.st_result()
    for k, req in enumerate(st.requests):
        st.check(st.L.st_submit(st.ctx, C.byref(req), C.cast(C.byref(st.tickets, k * size), C.POINTER(C.c_uint64))), "st_submit")
    for ticket in st.tickets:
        st.check(st.L.st_wait(st.ctx, ticket, C.byref(result), 60.0), "st_wait")
        st.check(result.status, "request")
    return st.pixels


def _prepare_texture(case, seed):
    st = State(case)
    colour, _ = _images(seed, case["width"], case["height"])
    if case["bits"] == 32:
        colour = np.concatenate([colour, np.full(colour.shape[:2] + (1,), 255, np.uint8)], -1)
    st.image = np.ascontiguousarray(colour)
    st.memory = np.zeros(st.L.st_texture_bytes(case["width"], case["height"], int(case["mipmap"])), np.uint8)
    return st


def _run_texture(st):
    tex, memory = _bake(st.renderer, st.image, st.case["wrap"], st.case["mipmap"], st.memory)
    table = (C.sizeof(S.TextureMip) * tex.mip_count + 15) & ~15      # holds addresses; the quads follow
    return {"quads": memory[table:], "mips": int(tex.mip_count)}


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return globals()["_run_" + state.case["kind"]](state)


# ---- what a pass cannot do without -----------------------------------------------------------------
def _view_work(rays, pixels, items):
    """A ray tests at least the two boxes of each level of a balanced tree over `items` (24
    operations a box) and reads one 128-byte triangle or primitive record."""
    levels = max(1, math.ceil(math.log2(max(items, 2))))
    return rays * (24 + 128) + 4 * pixels, rays * 48 * levels


def work(case):
    kind = case["kind"]
    if kind == "pick":
        return {"bytes": 72 * case["prims"] + 48, "flops": 60 * case["prims"]}
    if kind == "frame":
        items = 16 + 20 * 4 ** case["size"] if case["scene"] == "mesh" else case["size"]
        b, f = _view_work((case["width"] + 1) * (case["height"] + 1), case["width"] * case["height"], items)
        return {"bytes": b, "flops": f}
    if kind == "moving":
        n = case["prims"]
        b, f = 76 * case["moved"] + 72 * n + 64 * n + 4 * n, 100 * n
        if case["render"]:
            vb, vf = _view_work((case["width"] + 1) * (case["height"] + 1), case["width"] * case["height"], n)
            b, f = b + vb, f + vf
        return {"bytes": b, "flops": f}
    if kind == "blas":
        t = case["triangles"]
        return {"bytes": t * (36 + 16) + t * (128 + 4 + 32), "flops": 300 * t}
    if kind == "batch":
        sizes = [_view_size(k) for k in range(case["views"])]
        each = [_view_work(w * h, w * h, (16, 20 * 4 ** case["mesh_size"], case["prims"])[k % 3]) for k, (w, h) in enumerate(sizes)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    if kind == "serve":
        sizes = [_view_size(k) for k in range(case["requests"])]
        each = [_view_work(w * h, w * h, (20480, case["prims"])[k % 2]) for k, (w, h) in enumerate(sizes)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    quads = (case["width"] + 1) * (case["height"] + 1) * (4 / 3 if case["mipmap"] else 1)
    return {"bytes": int(case["width"] * case["height"] * case["bits"] / 8 + 12 * quads), "flops": int(12 * quads)}


# ---- the same results in 64 bits --------------------------------------------------------------------
# Primary rays of implicit scenes of up to 64 primitives: every primitive against every ray.
def _v(x):
    return torch.tensor(np.asarray(x, np.float64), device=DEVICE)


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _rotate(v, q):
    axis, w = q[:3].expand_as(v), q[3]
    t = torch.linalg.cross(axis, v)
    return v + 2 * (w * t + torch.linalg.cross(axis, t))


def _select(mask, a, b):
    return torch.where(mask[..., None], a, b)


def _hit_local(kind, o, d):
    """Hits of a unit shape: (hit, distance, normal as the shape reports it)."""
    if kind == S.PT_QUAD:
        t = (o[..., 1] / d[..., 1]).abs()
        p = o + d * t[..., None]
        hit = (d[..., 1] != 0) & (o[..., 1] != 0) & ((o[..., 1] < 0) != (d[..., 1] < 0))
        return hit & (p[..., 0].abs() <= 1) & (p[..., 2].abs() <= 1), t, _v([0, 1, 0]).expand_as(d)
    if kind == S.PT_BOX:
        side = torch.where(torch.signbit(d), 1.0, -1.0).double()
        near, near_axis = ((side - o) / d).max(-1)
        far, far_axis = ((-side - o) / d).min(-1)
        normal = torch.nn.functional.one_hot(torch.where(near < 0, far_axis, near_axis), 3) * side
        return (far >= 0) & (far >= near.clamp(min=0)), torch.where(near < 0, far, near), normal
    if kind == S.PT_SPHERE:
        tc = -_dot(o, d)
        ds = 1 - (_dot(o, o) - tc * tc)
        root = ds.clamp(min=0).sqrt()
        t = torch.where(tc - root <= 0, tc + root, tc - root)
        return (tc > 0) & (ds > 0), t, o + d * t[..., None]
    k = 3 ** -0.5
    corners = [_v(c) for c in ([-k, -k, -k], [k, -k, k], [k, k, -k], [-k, k, k])]
    best = torch.full(o.shape[:-1], math.inf, device=DEVICE, dtype=torch.float64)
    normal = torch.zeros_like(o)
    for opposite in range(4):
        face = [c for i, c in enumerate(corners) if i != opposite]
        n = -_unit(corners[opposite])
        nd, rp = -_dot(d, n.expand_as(d)), _dot(face[0] - o, n.expand_as(d))
        t = (rp / nd).abs()
        p = o + d * t[..., None]
        hit = (nd != 0) & ((rp > 0) != (nd > 0)) & (t < best)
        for a, b, c in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
            inward = torch.linalg.cross(face[b] - face[a], n)
            inward = inward * torch.sign((face[c] - face[a]) @ inward)
            hit &= _dot(p - face[a], inward.expand_as(p)) >= 0
        best, normal = torch.where(hit, t, best), _select(hit, n.expand_as(d), normal)
    return best < math.inf, best, normal


def _screen_bounds(p, cam, width, height):
    """The rectangle of grid points a primary ray may hit primitive `p` from (render/SSB.h:5), as
    (x0, y0, x1, y1), or None; float64, truncated as the reference truncates it."""
    x, y, z = (np.asarray(p["position"], np.float64) - np.asarray(cam.position, np.float64)) @ cam.matrix_cols()
    scale, fl = np.asarray(p["scale"], np.float64), cam.focal_length
    r = {S.PT_SPHERE: scale.max(), S.PT_TETRAHEDRON: scale.max() * math.sqrt(2)}.get(int(p["type"]), np.linalg.norm(scale))
    if z <= r:
        if z <= -r:
            return None
        h = abs(z) / fl
        w = h * width / height
        left, right, top, bottom = x - r, x + r, y + r, y - r
        if h < bottom or top < -h or w < left or right < -w:
            return None
        return (int(width * (left + w) / (2 * w)) if -w < left else 0, int(height * (h - top) / (2 * h)) if top < h else 0,
                int(width * (right + w) / (2 * w)) if right < w else width,
                int(height * (h - bottom) / (2 * h)) if -h < bottom else height)
    den = z * z - r * r
    across, up = r * math.sqrt(x * x + den), r * math.sqrt(y * y + den)
    left, right = ((x * z + k * across) * fl / den * height / width for k in (-1, 1))
    bottom, top = ((y * z + k * up) * fl / den for k in (-1, 1))
    if not (bottom < 1 and top > -1 and left < 1 and right > -1):
        return None
    left, bottom, right, top = max(left, -1), max(bottom, -1), min(right, 1), min(top, 1)
    return int(width / 2 * (left + 1)), int(height / 2 * (1 - top)), int(width / 2 * (right + 1)), int(height / 2 * (1 - bottom))


def _closest(prims, origin, direction, cam, width, height, xs, ys):
    """The closest primitive of each primary ray through the grid points (xs, ys)."""
    best = torch.full(direction.shape[:-1], math.inf, device=DEVICE, dtype=torch.float64)
    which = torch.full(best.shape, -1, device=DEVICE, dtype=torch.long)
    position, normal = torch.zeros_like(direction), torch.zeros_like(direction)
    for i in range(len(prims)):
        p = prims[i]
        rect = _screen_bounds(p, cam, width, height)
        if rect is None:
            continue
        q, scale, at = _v(p["rotation"]), _v(p["scale"]), _v(p["position"])
        inverse = torch.cat([-q[:3], q[3:]])
        o = _rotate((origin - at).expand_as(direction), inverse) / scale
        d = _unit(_rotate(direction, inverse) / scale)
        o = o + d * 1e-4
        hit, t, n = _hit_local(int(p["type"]), o, d)
        where = _rotate((o + d * t[..., None]) * scale, q) + at
        dsq = ((where - origin) ** 2).sum(-1)
        hit &= (dsq < best) & (xs >= rect[0]) & (ys >= rect[1]) & (xs < rect[2]) & (ys < rect[3])
        best, which = torch.where(hit, dsq, best), torch.where(hit, i, which)
        position, normal = _select(hit, where, position), _select(hit, _unit(_rotate(n / scale, q)), normal)
    return which, best, position, normal


def _glow(lights, origin, direction, limit):
    """Which rays cross a light's glow sphere before `limit`, and the nearest one's far end."""
    nearest = torch.full(limit.shape, math.inf, device=DEVICE, dtype=torch.float64)
    seen = torch.zeros_like(limit, dtype=torch.bool)
    for light in lights:
        size = float(light["intensity"]) / 16
        rc = (_v(light["position_or_direction"]) - origin) * (8 / size)
        b, c = _dot(direction, rc.expand_as(direction)), (rc * rc).sum(-1) - 1
        disc = b * b - c
        near, far = b - disc.clamp(min=0).sqrt(), b + disc.clamp(min=0).sqrt()
        hit = (disc >= 0) & (far > 0) & (near < limit * (8 / size))
        nearest = torch.where(hit & (far - size * 8 < nearest), far - size * 8, nearest)
        seen |= hit
    return nearest, seen


def _rays(frame, xs, ys):
    pp = frame.viewport.projection_plane
    start, right, down = (_v([p.x, p.y, p.z]) for p in (pp.start, pp.right, pp.down))
    return _unit(start + right * xs[..., None] + down * ys[..., None])


def _exact_frame(case, seed):
    sd, cam = _scene_of(case, seed)
    frame = _frame(case["width"], case["height"], cam, case["depth"], case["mode"], case["cone"])
    size = case["width"] + 1, case["height"] + 1
    ys, xs = torch.meshgrid(*(torch.arange(s, device=DEVICE, dtype=torch.float64) for s in size[::-1]), indexing="ij")
    origin, direction = _v(cam.position), _rays(frame, xs, ys)
    which, dsq, position, normal = _closest(sd.primitives, origin, direction, cam, *size, xs, ys)
    hit, z = which >= 0, (position - origin) @ _v(cam.matrix_cols()[:, 2])
    color = None
    if case["mode"] == "beauty":
        # no value of the colour: the glow's cubic cancels in the reference's 32 bits to noise whose
        # eighth power is what single pixels show, so a frame in 64 bits is another frame
        nearest, seen = _glow(sd.lights, origin, direction, torch.where(hit, dsq.sqrt(), math.inf))
        z, hit = torch.where(seen & ~hit, nearest, z), hit | seen
    else:
        color = 0.5 * (normal + 1) if case["mode"] == "normals" else (4 / dsq.sqrt())[..., None].expand_as(direction)
        x = _select(hit, (color * 255) ** 2, torch.zeros_like(color))
        color = torch.cat([x, hit.double()[..., None]], -1)
    return {"color": color, "depth": torch.where(hit, z, math.inf), "pixels": None}


def _exact_pick(case, seed):
    sd, cam = _implicit(seed, case["prims"])
    frame = _frame(case["width"], case["height"], cam, 1)
    x, y = (_v([k]) for k in _clicked(case, seed))
    origin, direction = _v(cam.position), _rays(frame, x, y)
    which, dsq, position, _ = _closest(sd.primitives, origin, direction, cam, case["width"] + 1, case["height"] + 1, x, y)
    distance, found = dsq.sqrt(), which >= 0
    for light in sd.lights:
        radius = float(light["intensity"]) / 128
        rc = (_v(light["position_or_direction"]) - origin) / radius
        b, c = _dot(direction, rc.expand_as(direction)), (rc * rc).sum() - 1
        disc = b * b - c
        near, far = b - disc.clamp(min=0).sqrt(), b + disc.clamp(min=0).sqrt()
        hit = (disc >= 0) & (far > 0) & (near < distance / radius)
        distance, found = torch.where(hit, near * radius, distance), found | hit
        position = _select(hit, origin + direction * distance[..., None], position)
    z = (position - origin) @ _v(cam.matrix_cols()[:, 2])
    return {"found": None, "type": None, "id": None, "position": _select(found, position, torch.zeros_like(position))[0],
            "distance": torch.where(found, distance, 0.0)[0], "object_distance": torch.where(found, z, 0.0)[0]}


def exact(case, seed):
    """None where the result is bytes (trees, texels, 8-bit frames) or a tracer over a BVH is wanted."""
    if case["kind"] == "pick":
        return _exact_pick(case, int(seed))
    if case["kind"] == "frame" and case["scene"] == "implicit" and case["size"] <= 64:
        return _exact_frame(case, int(seed))
    return None
