"""The frames this renderer is timed on: what each stands for in use, how its
inputs are made, one pass through the public entry points, the bytes and
operations a pass cannot do without, and its depths in 64 bits.

Inputs are made on the GPU from a seed: soups as `scenes.soup_vertices` draws
them, the UV sphere and the displaced icosphere of `scenes` with a seeded
pose, relief and texture.  Vertices live in device buffers bound to the
renderer (uploaded each pass in the streaming case), and every state has
rendered and checked one frame, as a program past its first frame has.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(ROOT, "custom-gpgpu-rasterizer_gb300"), ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import gbr  # noqa: E402
import predictor  # noqa: E402
import scenes  # noqa: E402

SOUP, SPHERE, ICO, BATCH = "soup", "sphere", "icosphere", "batch"
# how a pass gives its frame: left on the device, or read back to pinned host
# memory; STREAM uploads the vertices first, TURN renders the next of TURNS
# views, BARE is the entry point that allocates nothing
DEVICE, TURN, STREAM, BARE = "device", "turn", "stream", "bare"
TURNS = 8

# one frame's settings; a case gives those it changes
BASE = {"kind": SOUP, "tris": 100_000, "width": 1280, "height": 720, "bin_w": 16, "bin_h": 16, "io": DEVICE,
        "binning": "exact", "wide": False, "cull": scenes.CULL_NONE, "sample": scenes.SAMPLE_POINT,
        "vis": scenes.VIS_PBR, "lit": False, "subdiv": 0, "lon": 0, "lat": 0, "texture": 0,
        "scenes": 0, "min_tris": 0, "chunk": 4096, "threads": 0}


def _case(**kw):
    return {**BASE, **kw}


def listed():
    return [
        # the smallest ordinary frame: the textured sphere of the smoke test, left on the device (latency, launches)
        _case(name="sphere_vga", kind=SPHERE, lon=64, lat=32, texture=512, width=640, height=480,
              cull=scenes.CULL_BACKFACE),
        # an interactive program: every pass another camera, the frame and its depth read back
        _case(name="sphere_vga_turntable", kind=SPHERE, lon=64, lat=32, texture=512, width=640, height=480,
              cull=scenes.CULL_BACKFACE, io=TURN),
        # a small frame of odd sizes: no extent is a multiple of anything, 56-byte vertices, bins of 24x20, culling
        _case(name="soup_30k_odd", tris=30_011, width=333, height=250, bin_w=24, bin_h=20, wide=True,
              cull=scenes.CULL_BACKFACE),
        # a host that may not allocate while it renders (latency of the synchronous entry point)
        _case(name="soup_20k_bare", tris=20_000, width=512, height=512, io=BARE),
        # an ordinary frame of overlapping triangles
        _case(name="soup_100k_720p", tris=100_000, width=1280, height=720),
        # the benchmark's frame
        _case(name="soup_1m_1080p", tris=1_000_000, width=1920, height=1080),
        # the same with learned bin capacities
        _case(name="soup_1m_1080p_learned", tris=1_000_000, width=1920, height=1080, binning="learned"),
        # the same end to end: new vertices from the host every frame, the framebuffer back to it
        _case(name="soup_1m_1080p_stream", tris=1_000_000, width=1920, height=1080, io=STREAM),
        # the largest single frame: 2M triangles over a 4K screen
        _case(name="soup_2m_4k", tris=2_000_000, width=3840, height=2160),
        # a dense mesh of sub-pixel triangles at 4K, four maps, bilinear filter and two lights
        _case(name="icosphere7_4k_lit", kind=ICO, subdiv=7, texture=2048, width=3840, height=2160,
              cull=scenes.CULL_BACKFACE, sample=scenes.SAMPLE_BILINEAR, lit=True),
        # a mesh of a few pixels a triangle with the reference's filter, shader and 8x8 bins
        _case(name="icosphere6_1080p", kind=ICO, subdiv=6, texture=1024, width=1920, height=1080, bin_w=8, bin_h=8,
              cull=scenes.CULL_BACKFACE, sample=scenes.SAMPLE_LINEAR),
        # a server's batch: 32 uneven scenes of the batch workload as one frame, with a configuration the tuner picks
        _case(name="batch_32_uneven", kind=BATCH, scenes=32, min_tris=1000, tris=500_000, width=1920, height=1080,
              bin_w=32, bin_h=32, chunk=2048, threads=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice([SOUP, SOUP, SOUP, SPHERE, ICO, BATCH])
    vis = rng.choice([scenes.VIS_PBR] * 3 + [scenes.VIS_NORMAL, scenes.VIS_DEPTH])
    bins = rng.choice([(8, 8), (16, 16), (16, 16), (32, 32), (24, 20)])
    if kind == SOUP:
        io = rng.choice([DEVICE, DEVICE, DEVICE, STREAM, BARE])
        tris = _log(rng, 1000, {BARE: 30_000, STREAM: 800_000}.get(io, 1_500_000))
        if io == BARE:
            w, h = rng.randint(200, 640), rng.randint(200, 640)
            bins = (16, 16)
        else:
            w, h = _log(rng, 300, 3840), _log(rng, 240, 2160)
        # a triangle meets some tens of 8x8 bins: those go with fewer triangles
        if tris > 500_000 and bins == (8, 8):
            bins = (16, 16)
        return _case(tris=tris, width=w, height=h, bin_w=bins[0], bin_h=bins[1], io=io, wide=io != STREAM and rng.random() < 0.3,
                     cull=rng.choice([scenes.CULL_NONE, scenes.CULL_BACKFACE]),
                     vis=scenes.VIS_PBR if rng.random() < 0.7 else vis,
                     binning="learned" if io == DEVICE and bins == (16, 16) and rng.random() < 0.3 else "exact")
    if kind == SPHERE:
        return _case(kind=SPHERE, lon=rng.randint(16, 300), lat=rng.randint(8, 150), texture=_log(rng, 64, 1024),
                     width=_log(rng, 300, 1920), height=_log(rng, 240, 1080), bin_w=bins[0], bin_h=bins[1],
                     cull=scenes.CULL_BACKFACE, sample=rng.randint(0, 2), vis=vis, lit=rng.random() < 0.3,
                     io=rng.choice([DEVICE, TURN]))
    if kind == ICO:
        return _case(kind=ICO, subdiv=rng.randint(5, 7), texture=_log(rng, 256, 2048), width=_log(rng, 1280, 3840),
                     height=_log(rng, 720, 2160), bin_w=bins[0], bin_h=bins[1], cull=scenes.CULL_BACKFACE,
                     sample=rng.randint(0, 2), vis=vis, lit=rng.random() < 0.5)
    # batches: from thumbnails to the uneven workload
    side = rng.choice([8, 16, 32])
    return _case(kind=BATCH, scenes=rng.randint(4, 31), min_tris=1000, tris=_log(rng, 4000, 400_000),
                 width=_log(rng, 256, 1920), height=_log(rng, 256, 1080), bin_w=side, bin_h=side,
                 chunk=rng.choice([128, 512, 2048]), threads=rng.choice([128, 256]))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rows(p, rgb, wide):
    """Vertex records as int32 words [n, 4 or 14] from positions [n, 3] (float32) and byte colours [n, 3]."""
    n = p.shape[0]
    if wide:
        v = torch.zeros(n, 14, dtype=torch.float32, device="cuda")
        v[:, 0:3] = p
        v[:, 11:14] = rgb.to(torch.float32) / 255.0
        return v.view(torch.int32)
    v = torch.empty(n, 4, dtype=torch.int32, device="cuda")
    v[:, 0:3] = p.contiguous().view(torch.int32)
    v[:, 3] = (rgb[:, 0] | (rgb[:, 1] << 8) | (rgb[:, 2] << 16) | (255 << 24)).to(torch.int32)
    return v


def _soup(n, width, height, seed, wide):
    """The soup of scenes.soup_vertices, drawn on the GPU: centroids uniform plus a 20% Gaussian blob, areas
    log-uniform in 0.5-4096 px^2, random orientation and winding, depths uniform in [0.1, 100], byte colours."""
    g = _gen(seed)

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    blob = torch.rand(n, generator=g, device="cuda") < 0.2
    near = 100.0 * torch.randn(n, 2, generator=g, device="cuda", dtype=torch.float64)
    cx = torch.where(blob, width / 2 + near[:, 0], uniform(0, width, n))
    cy = torch.where(blob, height / 2 + near[:, 1], uniform(0, height, n))
    area = torch.exp(uniform(math.log(0.5), math.log(4096.0), n))
    ang = (uniform(0, 2 * math.pi, n)[:, None] + torch.arange(3, device="cuda")[None, :] * (2 * math.pi / 3)
           + uniform(-0.6, 0.6, n, 3))
    ux, uy = torch.cos(ang), torch.sin(ang)
    unit = 0.5 * ((ux[:, 1] - ux[:, 0]) * (uy[:, 2] - uy[:, 0]) - (uy[:, 1] - uy[:, 0]) * (ux[:, 2] - ux[:, 0])).abs()
    r = torch.sqrt(area / unit.clamp_min(1e-6))
    x, y = cx[:, None] + r[:, None] * ux, cy[:, None] + r[:, None] * uy
    turn = (torch.rand(n, generator=g, device="cuda") < 0.5)[:, None]
    x = torch.where(turn, x[:, [0, 2, 1]], x)
    y = torch.where(turn, y[:, [0, 2, 1]], y)
    d = (uniform(0.1, 100.0, n)[:, None] * (1.0 + uniform(-0.01, 0.01, n, 3))).clamp(0.1, 100.0)
    p = torch.stack([2.0 * x / width - 1.0, 1.0 - 2.0 * y / height, (d - 0.1) / 99.9], -1)
    rgb = torch.randint(0, 256, (3 * n, 3), generator=g, device="cuda")
    return _rows(p.reshape(-1, 3).to(torch.float32), rgb, wide)


_ICOSPHERES = {}


def _unit_icosphere(subdiv):
    """Unit icosphere: positions [n, 3] float64 and triangles [m, 3] int32 (the same for every seed)."""
    if subdiv not in _ICOSPHERES:
        t = (1.0 + 5 ** 0.5) / 2.0
        v = np.array([(-1, t, 0), (1, t, 0), (-1, -t, 0), (1, -t, 0), (0, -1, t), (0, 1, t), (0, -1, -t), (0, 1, -t),
                      (t, 0, -1), (t, 0, 1), (-t, 0, -1), (-t, 0, 1)], np.float64)
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        near = [(a, b, c) for a in range(12) for b in range(a + 1, 12) for c in range(b + 1, 12)
                if max(np.linalg.norm(v[a] - v[b]), np.linalg.norm(v[b] - v[c]), np.linalg.norm(v[a] - v[c])) < 1.1]
        f = np.array([t if np.dot(np.cross(v[t[1]] - v[t[0]], v[t[2]] - v[t[0]]), v[t[0]]) > 0 else (t[0], t[2], t[1])
                      for t in near], np.int64)
        for _ in range(subdiv):
            m = len(f)
            e = np.sort(np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]), axis=1)
            key, at = np.unique(e[:, 0] * len(v) + e[:, 1], return_inverse=True)
            at = at.reshape(-1) + len(v)
            mid = v[key // len(v)] + v[key % len(v)]
            v = np.concatenate([v, mid / np.linalg.norm(mid, axis=1, keepdims=True)])
            a, b, c = at[:m], at[m:2 * m], at[2 * m:]
            f = np.concatenate([np.stack([f[:, 0], a, c], 1), np.stack([f[:, 1], b, a], 1),
                                np.stack([f[:, 2], c, b], 1), np.stack([a, b, c], 1)])
        _ICOSPHERES[subdiv] = v, f.astype(np.int32)
    return _ICOSPHERES[subdiv]


def _icosphere(subdiv, seed):
    """The icosphere with a seeded relief of about 5%: IVertex words [n, 14] and indices."""
    unit, faces = _unit_icosphere(subdiv)
    u = torch.from_numpy(unit).cuda()
    g = _gen(seed)
    k = 12.0 * torch.randn(8, 3, generator=g, device="cuda", dtype=torch.float64)
    phase = 2 * math.pi * torch.rand(8, generator=g, device="cuda", dtype=torch.float64)
    r = torch.ones(len(unit), dtype=torch.float64, device="cuda")
    slope = torch.zeros_like(u)
    for j in range(8):
        a = u[:, 0] * k[j, 0] + u[:, 1] * k[j, 1] + u[:, 2] * k[j, 2] + phase[j]
        r = r + 0.012 * torch.sin(a)
        slope = slope + 0.012 * torch.cos(a)[:, None] * k[j][None, :]
    slope = slope - (slope * u).sum(-1, keepdim=True) * u
    n = u - slope / r[:, None]
    n = n / n.norm(dim=-1, keepdim=True)
    t = torch.stack([n[:, 2], torch.zeros_like(r), -n[:, 0]], -1)
    long = t.norm(dim=-1, keepdim=True)
    t = torch.where(long > 1e-6, t / long.clamp_min(1e-12), torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64, device="cuda"))
    v = torch.zeros(len(unit), 14, dtype=torch.float32, device="cuda")
    v[:, 0:3] = u * r[:, None]
    v[:, 3] = 0.5 + torch.atan2(u[:, 2], u[:, 0]) / (2 * math.pi)
    v[:, 4] = torch.acos(u[:, 1].clamp(-1, 1)) / math.pi
    v[:, 5:8] = n
    v[:, 8:11] = t
    v[:, 11:14] = 1.0
    return v.view(torch.int32), torch.from_numpy(faces.reshape(-1)).cuda()


_SPHERES = {}


def _sphere(lon, lat):
    """scenes.uv_sphere_mesh as IVertex words and indices (its pose is what the seed changes)."""
    if (lon, lat) not in _SPHERES:
        _SPHERES.clear()
        _SPHERES[lon, lat] = scenes.uv_sphere_mesh(lon, lat)
    m = _SPHERES[lon, lat]
    words = np.frombuffer(m.vertices.tobytes(), np.int32).reshape(-1, 14).copy()
    return torch.from_numpy(words).cuda(), torch.from_numpy(m.indices.view(np.int32)).cuda()


def _texture(size, seed):
    """Smooth seeded noise, RGBA8 [size, size]."""
    g = _gen(seed)
    out = torch.zeros(3, size, size, device="cuda")
    for octave in range(4):
        cells = 8 << octave
        grid = torch.rand(1, 3, cells, cells, generator=g, device="cuda")
        out = out + 0.5 ** octave * torch.nn.functional.interpolate(grid, size=(size, size), mode="bilinear",
                                                                    align_corners=True)[0]
    c = (out / 1.875 * 255.0).clamp(0, 255).to(torch.int64)
    return (c[0] | (c[1] << 8) | (c[2] << 16) | (255 << 24)).cpu().numpy().astype(np.uint32)


def _pose(seed):
    """A seeded rotation as a world matrix (column-major float32)."""
    g = torch.Generator()
    g.manual_seed(seed)
    q = torch.randn(4, generator=g, dtype=torch.float64)
    w, x, y, z = (q / q.norm()).tolist()
    m = np.eye(4)
    m[:3, :3] = [[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                 [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                 [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]]
    return np.ascontiguousarray(m.T, np.float32).reshape(16)


def _scene(case, seed):
    """(vertex words, indices or None, world, cameras, textures, lights) of one frame."""
    w, h = case["width"], case["height"]
    if case["kind"] == SOUP:
        return (_soup(case["tris"], w, h, seed, case["wide"]), None, scenes.identity16(), [scenes.identity_camera()],
                [], [])
    if case["kind"] == SPHERE:
        verts, idx = _sphere(case["lon"], case["lat"])
        away = 3.0
    else:
        verts, idx = _icosphere(case["subdiv"], seed)
        away = 8.0
    shift = 0.4 * np.random.default_rng(seed).uniform(-1.0, 1.0, (TURNS, 2))
    cams = [scenes.perspective_camera((x, y, away), 60.0, w, h) for x, y in shift]
    n = case["texture"]
    maps = [_texture(n, seed + 1), scenes.bump_normal_texture(n), scenes.flat_texture(n, (40, 40, 40)),
            scenes.flat_texture(n, (128, 128, 128))]
    lights = []
    if case["lit"]:
        lights = [scenes.Light(scenes.LIGHT_DIRECTIONAL, (1.0, 0.95, 0.9), 4.0, (0.577, -0.577, -0.577)),
                  scenes.Light(scenes.LIGHT_POINT, (0.4, 0.6, 1.0), 30.0, (2.0, 1.5, 3.0))]
    return verts, idx, _pose(seed), cams if case["io"] == TURN else cams[:1], maps, lights


def _batch(case, seed):
    """(triangles, width, height, seed) of each scene of a batch: the workload's spread, up to the case's sizes."""
    rng = np.random.default_rng(seed)
    sizes = ((1.0, 1.0), (0.55, 0.7), (0.3, 0.5), (0.14, 0.25))
    # the sizes are the same for every seed (the work is the case's), the scenes are not
    fixed = np.random.default_rng(case["scenes"])
    out = []
    for _ in range(case["scenes"]):
        tris = int(math.exp(fixed.uniform(math.log(case["min_tris"]), math.log(case["tris"]))))
        fw, fh = sizes[int(fixed.integers(0, 4))]
        out.append((tris, max(64, int(case["width"] * fw)), max(64, int(case["height"] * fh)),
                    int(rng.integers(1 << 31))))
    return out


class Owner:
    """The renderers of a state with what they are bound to; closed when neither the state nor an output is left."""

    def __init__(self):
        self.renderers, self.keep = [], []
        self.batch = None

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for r in self.renderers:
            r.close()


class _Device:
    """A device buffer of a renderer's, seen by torch: the tensor keeps its owner."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _buffers(owner, r):
    colour, depth = r.device_buffers()
    shape = (r.height, r.width)
    return (torch.as_tensor(_Device(owner, colour, shape, "<i4"), device="cuda"),
            torch.as_tensor(_Device(owner, depth, shape, "<f4"), device="cuda"))


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


class State:
    """What a program keeps: its renderers, their device buffers, cameras and host buffers."""

    def __init__(self, case):
        self.case = case
        self.own = Owner()
        self.turn = 0


def _bind(own, r, verts, idx, world, tex_ids):
    fmt = scenes.VERTEX_IVERTEX56 if verts.shape[1] == 14 else scenes.VERTEX_POS3_RGBA8
    own.keep += [verts, idx]
    torch.cuda.synchronize()
    return r.bind_mesh_device(verts.data_ptr(), verts.shape[0], fmt, 0 if idx is None else idx.data_ptr(),
                              0 if idx is None else idx.numel(), 0, world, tex_ids)


def prepare(case, seed):
    s = State(case)
    own = s.own
    if case["kind"] == BATCH:
        own.batch = gbr.Batch()
        s.out = []
        for tris, w, h, sseed in _batch(case, seed):
            r = gbr.Renderer(w, h)
            own.renderers.append(r)
            _bind(own, r, _soup(tris, w, h, sseed, False), None, scenes.identity16(), (-1, -1, -1, -1))
            own.batch.add(r, scenes.identity_camera(), case["cull"], case["sample"], case["vis"])
            s.out += _buffers(own, r)
        own.batch.set_config(case["bin_w"], case["chunk"], 5, 0, case["threads"])
        for _ in range(2):   # the storage, the counters and the captured graph settle
            own.batch.render()
            own.batch.stats()
        return s

    w, h = case["width"], case["height"]
    verts, idx, world, cams, maps, lights = _scene(case, seed)
    s.cams = [gbr.make_camera(c) for c in cams]
    if case["io"] == BARE:
        own.keep = [verts]
        s.world = (ctypes.c_float * 16)(*[float(x) for x in world])
        s.out = [torch.empty(h, w, dtype=torch.int32, device="cuda"),
                 torch.empty(h, w, dtype=torch.float32, device="cuda"),
                 torch.empty(h, w, dtype=torch.int32, device="cuda")]
        torch.cuda.synchronize()
        run(s)
        return s
    r = gbr.Renderer(w, h)
    own.renderers.append(r)
    r.setup_bins(-(-w // case["bin_w"]), -(-h // case["bin_h"]), case["bin_w"], case["bin_h"], case["chunk"])
    tex = tuple(r.add_texture(t) for t in maps) if maps else (-1, -1, -1, -1)
    if case["io"] == STREAM:
        host = verts.cpu().numpy()
        s.mesh = r.add_mesh(host, scenes.VERTEX_IVERTEX56 if host.shape[1] == 14 else scenes.VERTEX_POS3_RGBA8)
        s.host = _pinned(host.shape, torch.int32)
        s.host[:] = host
    else:
        _bind(own, r, verts, idx, world, tex)
    r.set_lights(lights)
    if case["binning"] == "learned":
        predictor.install(r)
    if case["io"] in (TURN, STREAM):
        s.colour, s.depth = _pinned(w * h, torch.int32).view(np.uint32), _pinned(w * h, torch.float32)
    else:
        s.out = _buffers(own, r)
    r.render(s.cams[0], case["cull"], case["sample"], case["vis"])
    r.stats()
    return s


def run(s):
    c = s.case
    if s.own.batch is not None:
        s.own.batch.render()
        return s.out
    if c["io"] == BARE:
        verts, (colour, depth, ids) = s.own.keep[0], s.out
        gbr.check(gbr.lib().gbr_render_noalloc(
            ctypes.c_void_p(verts.data_ptr()), verts.shape[0],
            scenes.VERTEX_IVERTEX56 if verts.shape[1] == 14 else scenes.VERTEX_POS3_RGBA8, None, 0, 0, s.world,
            ctypes.byref(s.cams[0]), c["width"], c["height"], -(-c["width"] // c["bin_w"]),
            -(-c["height"] // c["bin_h"]), c["bin_w"], c["bin_h"], c["chunk"], c["cull"], c["sample"], c["vis"],
            ctypes.c_void_p(colour.data_ptr()), ctypes.c_void_p(depth.data_ptr()), ctypes.c_void_p(ids.data_ptr()),
            None))
        return s.out
    r = s.own.renderers[0]
    if c["io"] == STREAM:
        r.update_vertices(s.mesh, s.host.ctypes.data, s.host.shape[0])
    cam = s.cams[s.turn % len(s.cams)]
    s.turn += 1
    r.render(cam, c["cull"], c["sample"], c["vis"])
    if c["io"] in (TURN, STREAM):
        return list(r.readback(s.colour, s.depth))
    return s.out


# ---------------------------------------------------------------------------
# What a pass cannot do without, and its depths in 64 bits
# ---------------------------------------------------------------------------
def work(case):
    """Vertices, indices and the drawn pixels' texels read once; colour and depth (and ids where they are returned) written once.
    Operations: about 150 a triangle (three vertices, the cull test, the set-up) and 100 a pixel (interpolation and
    the shader)."""
    if case["kind"] == BATCH:
        specs = _batch(case, 0)
        tris, px = sum(t for t, _, _, _ in specs), sum(w * h for _, w, h, _ in specs)
        return {"bytes": 48.0 * tris + 8.0 * px, "flops": 150.0 * tris + 100.0 * px}
    px = case["width"] * case["height"]
    if case["kind"] == SOUP:
        tris, bytes_in = case["tris"], 3.0 * case["tris"] * (56 if case["wide"] else 16)
    else:
        tris = 20 * 4 ** case["subdiv"] if case["kind"] == ICO else 2 * case["lon"] * (case["lat"] - 1)
        verts = tris // 2 + 2 if case["kind"] == ICO else (case["lon"] + 1) * (case["lat"] + 1)
        away = 8.0 if case["kind"] == ICO else 3.0
        drawn = math.pi * (case["height"] / 2 / math.tan(math.pi / 6)) ** 2 / (away * away - 1)
        texels = 16.0 * min(case["texture"] ** 2, drawn) if case["vis"] == scenes.VIS_PBR else 0.0
        bytes_in = 56.0 * verts + 12.0 * tris + texels
    out = (12.0 if case["io"] == BARE else 8.0) * px
    return {"bytes": bytes_in + out, "flops": 150.0 * tris + 100.0 * px}


def _exact_depth(verts, idx, world, cam, w, h, cull):
    """Depth of the nearest covered fragment of each pixel (0 where none), in 64 bits: positions through world, view
    and projection, the edge functions at integer pixels (the covered winding, edges included), weights over the
    area, 0 <= z < 1."""
    dev = verts.device
    p = verts[:, 0:3].contiguous().view(torch.float32).to(torch.float64)

    def mat(m):
        return torch.from_numpy(np.asarray(m, np.float64).reshape(4, 4).T.copy()).to(dev)

    c = torch.cat([p, torch.ones_like(p[:, :1])], 1) @ (mat(cam.proj) @ mat(cam.view) @ mat(world)).T
    ndc = c[:, :3] / c[:, 3:4]
    tri = ndc.reshape(-1, 3, 3) if idx is None else ndc[idx.long()].reshape(-1, 3, 3)
    lo = torch.tensor([-1.0, -1.0, 0.0], dtype=torch.float64, device=dev)
    keep = ~((tri < lo).all(1) | (tri > 1.0).all(1)).any(-1)
    if cull != scenes.CULL_NONE:
        n = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
        keep &= n @ torch.from_numpy(np.asarray(cam.fwd, np.float64)).to(dev) > 0
    x, y, z = (tri[..., 0] + 1) / 2 * w, (1 - tri[..., 1]) / 2 * h, tri[..., 2]
    area = (x[:, 0] - x[:, 1]) * (y[:, 2] - y[:, 1]) - (y[:, 0] - y[:, 1]) * (x[:, 2] - x[:, 1])
    keep &= area > 0
    x, y, z, area = x[keep], y[keep], z[keep], area[keep]
    x0, x1 = x.amin(1).ceil().clamp_min(0).long(), x.amax(1).floor().clamp_max(w - 1).long()
    y0, y1 = y.amin(1).ceil().clamp_min(0).long(), y.amax(1).floor().clamp_max(h - 1).long()
    wide = (x1 - x0 + 1).clamp_min(0)
    n = wide * (y1 - y0 + 1).clamp_min(0)
    upto = n.cumsum(0)
    total = int(upto[-1]) if len(n) else 0
    best = torch.full((w * h,), 2.0, dtype=torch.float64, device=dev)
    step = 1 << 24
    for at in range(0, total, step):
        k = torch.arange(at, min(at + step, total), device=dev)
        t = torch.searchsorted(upto, k, right=True)
        k = k - (upto - n)[t]
        px, py = x0[t] + k % wide[t], y0[t] + k // wide[t]

        def edge(a, b):
            return (px - x[t, a]) * (y[t, b] - y[t, a]) - (py - y[t, a]) * (x[t, b] - x[t, a])

        e2, e0, e1 = edge(0, 1), edge(1, 2), edge(2, 0)
        d = (e0 * z[t, 0] + e1 * z[t, 1] + e2 * z[t, 2]) / area[t]
        ok = (e0 >= 0) & (e1 >= 0) & (e2 >= 0) & (d >= 0) & (d < 1)
        best.scatter_reduce_(0, (py * w + px)[ok], d[ok], "amin")
    return torch.where(best < 1.0, best, torch.zeros_like(best)).reshape(h, w)


def exact(case, seed):
    """Colours and ids are whole numbers; the depths have a value in 64 bits."""
    if case["kind"] == BATCH:
        out = []
        for tris, w, h, sseed in _batch(case, seed):
            out += [None, _exact_depth(_soup(tris, w, h, sseed, False), None, scenes.identity16(),
                                       scenes.identity_camera(), w, h, case["cull"])]
        return out
    verts, idx, world, cams, _, _ = _scene(case, seed)
    d = _exact_depth(verts, idx, world, cams[0], case["width"], case["height"], case["cull"])
    return [None, d, None] if case["io"] == BARE else [None, d]
