"""The block raster (gbr_raster.cu) where its split can go wrong, against the
oracle's fixed-point mode: bins that are not whole 8x4 blocks, bins of fewer
blocks than a CTA has warps and of many times more, items around one phase
(32 triangles) and around one sorted pass (1024 and 2048 entries), triangles
around and far above the extent that keeps 32-bit edge values, and triangles
on the float path.  Winners and depth bit-exact, colour within 1 LSB."""
import ctypes as C

import numpy as np
import pytest

import scenes
from oracle import mlp_oracle, oracle

pytestmark = pytest.mark.gpu


def triangles(kind, n, width, height, seed):
    v = scenes.soup_vertices(n, width, height, seed)
    if kind == "small":
        return v
    if kind == "inside":   # every triangle meets the screen
        v["p"][:, :2] = v["p"][:, :2].clip(-0.95, 0.95)
        return v
    rng = np.random.default_rng(seed)
    p = v["p"].reshape(-1, 3, 3)
    if kind == "vast":     # screen-filling triangles of 3000 to 8000 px
        reach = rng.uniform(1500.0, 4000.0, (n, 1, 1)) * 2.0 / np.array([width, height])
        angle = rng.uniform(0, 2 * np.pi, (n, 1)) - np.arange(3) * (2 * np.pi / 3)
        p[:, :, :2] = rng.uniform(-0.5, 0.5, (n, 1, 2)) + reach * np.stack([np.cos(angle), -np.sin(angle)], -1)
        v["p"] = p.reshape(-1, 3)
        return v
    # every fourth triangle's first vertex thrown out to the given distance:
    # extents around 128 to 1024 px (the 32-bit limit is 2^14 px over the
    # bin's width + height), thousands of px, or beyond the guard band
    far = {"wide": (100.0, 1100.0), "huge": (2000.0, 8000.0), "float": (8300.0, 50000.0)}[kind]
    k = np.arange(0, len(p), 4)
    angle, reach = rng.uniform(0, 2 * np.pi, len(k)), rng.uniform(*far, len(k))
    p[k, 0, 0] += (2.0 * reach * np.cos(angle) / width).astype(np.float32)
    p[k, 0, 1] += (2.0 * reach * np.sin(angle) / height).astype(np.float32)
    v["p"] = p.reshape(-1, 3)
    return v


@pytest.mark.parametrize("bw,bh,w,h,n,kind", [
    (1, 1, 40, 24, 60, "small"),           # one pixel a bin, eight warps on one block
    (1, 1, 40, 24, 60, "vast"),            # blocks that reach far past their bins
    (2, 3, 40, 24, 200, "vast"),
    (9, 5, 90, 61, 500, "vast"),
    (8, 4, 96, 60, 400, "small"),          # one block a bin
    (7, 5, 100, 61, 600, "wide"),          # ragged blocks, ragged last bins
    (8, 8, 128, 96, 33, "huge"),           # items of at most a phase
    (24, 20, 333, 250, 3000, "wide"),
    (16, 16, 640, 480, 4000, "huge"),
    (16, 16, 320, 240, 500, "float"),
    (64, 64, 300, 200, 9000, "wide"),      # 128 blocks a bin, several passes an item
    (64, 64, 64, 64, 32, "inside"),        # one bin: a whole phase, then one more
    (64, 64, 64, 64, 33, "inside"),
    (64, 64, 64, 64, 1024, "inside"),      # a whole pass of a 128-thread CTA, then one more
    (64, 64, 64, 64, 1025, "inside"),
    (64, 64, 64, 64, 2049, "inside"),      # one entry past a 256-thread CTA's pass
    (33, 17, 66, 34, 5000, "huge"),
    (8, 8, 640, 480, 3000, "wide"),        # many bins of two blocks: CTAs of 64 threads
    (16, 16, 1920, 1080, 2500, "wide"),    # many short items: CTAs of 64 threads, two pixels a lane
    (10, 12, 960, 1080, 2500, "huge"),     # the same, ragged
])
def test_block_raster_against_the_oracle(gbr_lib, cuda_device, bw, bh, w, h, n, kind):
    v = triangles(kind, n, w, h, seed=31)
    s = scenes.Scene(kind, w, h, bw, bh, scenes.identity_camera(), [scenes.Mesh(vertices=v)], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        for frame in range(3):   # without history, then with the CTAs and items the last frame calls for
            r.set_raster_params(16, (0, 4, 6)[frame])   # a phase below 32: never the small-triangle variant
            r.render_scene(s)
            colour, depth = r.readback()
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners differ"
            assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth differs"
            c, oc = colour.astype(np.int64), o["colour"].astype(np.int64)
            assert max(np.abs(((c >> k) & 255) - ((oc >> k) & 255)).max() for k in (0, 8, 16)) <= 1
            assert r.stats()["raster_lanes"] == 0


@pytest.mark.parametrize("n", [1 << 23, (1 << 23) + 1])
def test_list_entries_with_and_without_depth(gbr_lib, cuda_device, n):
    """Up to 2^23 triangles a list entry carries its depth bucket beside the
    primitive; one more and it does not.  Most of the frame's triangles lie
    off the screen, the drawn ones are the first and the last, so ids use
    every bit: bin lists and winners are the oracle's either way."""
    drawn = scenes.soup_vertices(1500, 320, 240, seed=9)
    off = np.zeros(3, scenes.POS3_RGBA8)
    off["p"] = [(5.0, 5.0, 0.5), (6.0, 5.0, 0.5), (5.0, 6.0, 0.5)]
    v = np.concatenate([drawn, off])
    ix = np.tile(np.arange(len(drawn), len(v), dtype=np.uint32), n).reshape(n, 3)
    d = np.arange(len(drawn), dtype=np.uint32).reshape(-1, 3)
    ix[:700], ix[-800:] = d[:700], d[700:]
    s = scenes.Scene("many", 320, 240, 16, 16, scenes.identity_camera(),
                     [scenes.Mesh(vertices=v, indices=ix.reshape(-1))], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    assert o["ids"][o["ids"] != 0xFFFFFFFF].max() >= n - 800
    with gbr_lib.Renderer(320, 240) as r:
        r.load_scene(s)
        for _ in range(2):
            r.render_scene(s)
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"])
            assert np.array_equal(r.readback_ids(), o["ids"])


@pytest.mark.parametrize("crowd", [10, 65, 129, 1500])
def test_short_items_beside_a_long_one(gbr_lib, cuda_device, crowd):
    """A frame of few, short items and one crowded bin: later frames split its
    list at twice the mean item (no less than 64 entries)."""
    w, h = 320, 240
    v = triangles("small", 500 + crowd, w, h, seed=8)
    p = v["p"].reshape(-1, 3, 3)
    p[500:, :, :2] = np.array([0.3, -0.2]) + 0.02 * (p[500:, :, :2] - p[500:, :1, :2])   # of a pixel, in one bin
    v["p"] = p.reshape(-1, 3)
    s = scenes.Scene("crowd", w, h, 16, 16, scenes.identity_camera(), [scenes.Mesh(vertices=v)], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        for frame in range(3):
            r.set_raster_params(16, 0)   # a phase below 32: never the small-triangle variant
            r.render_scene(s)
            _, depth = r.readback()
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"]), f"frame {frame}: lists"
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners"
            assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth"
            items = r.stats()["num_work_items"]
            first = items if frame == 0 else first
            if frame:   # the first frame has no mean to split at
                assert items == first if crowd == 10 else items >= first + (crowd > 1000) * 10


def small_beside_large(w, h, vertex_colours, px=3.5):
    rng = np.random.default_rng(3)
    n = 9000
    c = rng.uniform(-0.95, 0.95, (n, 1, 2))
    size = rng.uniform(0.2, px, (n, 1, 1)) * 2.0 / np.array([w, h])
    ang = rng.uniform(0, 2 * np.pi, (n, 1)) - np.arange(3) * (2 * np.pi / 3)
    v = np.zeros(3 * n, scenes.IVERTEX56)
    p = v["p"].reshape(-1, 3, 3)
    p[:, :, :2] = c + size * np.stack([np.cos(ang), -np.sin(ang)], -1)
    p[:, :, 2] = rng.uniform(0.05, 0.95, (n, 1))
    p[::1500, 0, :2] += rng.uniform(0.1, 0.5, (6, 2))
    p[5, 0, 0] = 60.0
    p[5, 2] = p[5, 0] + (0.0, 0.02, 0.0)
    v["p"] = p.reshape(-1, 3)
    v["uv"] = rng.uniform(0, 1, (3 * n, 2))
    v["n"] = (0, 0, 1)
    v["tan"] = (1, 0, 0)
    v["c"] = rng.uniform(0, 1, (3 * n, 3))
    m = scenes.Mesh(vertices=v)
    if not vertex_colours:
        m.textures = [scenes.checker_texture(64, 8), scenes.flat_texture(64, (128, 128, 255)), None, None]
    return m


@pytest.mark.parametrize("vertex_colours", [True, False])
@pytest.mark.parametrize("w,h,bw,bh", [(640, 480, 16, 16), (333, 250, 24, 20), (1024, 600, 8, 8)])
def test_direct_small_triangles_beside_large_ones(gbr_lib, cuda_device, w, h, bw, bh, vertex_colours):
    """A frame of small triangles, drawn by the set-up pass, around boxes of
    16 pixels (its limit) and among them a few large, very large and float-path
    triangles, drawn by the raster: lists, winners and depth are the oracle's
    (flat- and texture-shaded frames, one and two passes)."""
    m = small_beside_large(w, h, vertex_colours)
    s = scenes.Scene("direct", w, h, bw, bh, scenes.identity_camera(), [m], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    assert o["stats"]["num_float_path"] == 1
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        for frame in range(3):
            r.render_scene(s)
            colour, depth = r.readback()
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"]), f"frame {frame}: lists"
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners"
            assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth"
            c0, c1 = colour.astype(np.int64), o["colour"].astype(np.int64)
            assert max(np.abs(((c0 >> k) & 255) - ((c1 >> k) & 255)).max() for k in (0, 8, 16)) <= 1
            assert r.stats()["raster_lanes"] == (1 if frame else 0)


@pytest.mark.parametrize("per_bin", [29.0, 3.0])
@pytest.mark.parametrize("w,h,bin_size,px", [(640, 480, 16, 3.5), (2048, 1088, 8, 2.5)])   # bins within and beyond shared memory's rows
def test_direct_small_triangles_with_predicted_capacities(gbr_lib, cuda_device, w, h, bin_size, px, per_bin):
    """The same under predicted binning: capacities that hold every bin (the
    lists carry drawn and undrawn entries together), and capacities that
    overflow (the exact pass draws the small triangles once more)."""
    m = small_beside_large(w, h, True, px)
    s = scenes.Scene("direct", w, h, bin_size, bin_size, scenes.identity_camera(), [m], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    most = int(np.diff(o["offsets"].astype(np.int64)).max())
    assert 4 < most <= 29
    weights = np.zeros(mlp_oracle.NUM_PARAMS, np.float32)
    weights[mlp_oracle.OFF_B3] = per_bin
    w16 = mlp_oracle.f32_to_bf16(weights)
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        r.render_scene(s)
        r.stats()
        gbr_lib.check(r._lib.gbr_set_predictor(r.h, w16.ctypes.data_as(C.c_void_p), len(w16), C.c_float(0.0),
                                               C.c_float(0.0), C.c_float(0.0)))
        r.set_binning(gbr_lib.BINNING_PREDICTED)
        for frame in range(3):
            r.render_scene(s)
            _, depth = r.readback()
            st = r.stats()
            assert st["raster_lanes"] == 1 and st["predicted_overflow"] == (per_bin < most)
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"]), f"frame {frame}: lists"
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners"
            assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth"
