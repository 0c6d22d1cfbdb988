"""The block raster's CTA widths where the bins are odd or crowded, against the
oracle's fixed-point mode: CTAs of 128 threads (two pixels a lane) in ragged
and in large bins (of 64 in the smallest), with one bin of more than a sorted
pass (1024 entries);
CTAs of 64 in bins of two blocks with one, two and three passes (512 entries
each); the passes and splits that a small queue chunk asks of the raster with
bulk-copy staging, which honours it to the entry."""
import numpy as np
import pytest

import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def crowded_soup(n, crowd, w, h, seed):
    """A soup, and `crowd` triangles of a pixel or two in one bin."""
    v = scenes.soup_vertices(n + crowd, w, h, seed)
    p = v["p"].reshape(-1, 3, 3)
    p[n:, :, :2] = np.array([0.3, -0.2]) + 0.02 * (p[n:, :, :2] - p[n:, :1, :2])
    v["p"] = p.reshape(-1, 3)
    return v


def assert_frames(r, s, frames, check):
    o = oracle.render(s, oracle.RASTER_FIXED)
    for frame in range(frames):
        r.set_raster_params(16, 0)   # a phase below 32: no triangle is left to the set-up pass
        r.render_scene(s)
        _, depth = r.readback()
        assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners"
        assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth"
        check(frame, r.stats(), np.diff(o["offsets"].astype(np.int64)))


@pytest.mark.parametrize("bw,bh,w,h,n", [(24, 20, 960, 640, 9000), (33, 17, 1056, 510, 9000), (64, 64, 1536, 1280, 9000),
                                         (9, 5, 640, 480, 3000), (7, 5, 640, 480, 3000)])
def test_ragged_and_large_bins_in_many_items(gbr_lib, cuda_device, bw, bh, w, h, n):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    s = scenes.Scene("crowd", w, h, bw, bh, scenes.identity_camera(),
                     [scenes.Mesh(vertices=crowded_soup(n, 1300, w, h, 12))], cull=scenes.CULL_NONE)

    def check(frame, st, counts):
        assert counts.max() > 1024
        assert min(st["num_work_items"], (counts > 0).sum()) > 3 * sms   # else CTAs of 512 threads

    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        assert_frames(r, s, 3, check)


@pytest.mark.parametrize("crowd", [500, 1000, 1500])
def test_passes_of_ctas_of_64(gbr_lib, cuda_device, crowd):
    """The first frame's items hold up to 4096 entries: passes of 512."""
    w, h = 640, 480
    s = scenes.Scene("crowd", w, h, 8, 8, scenes.identity_camera(),
                     [scenes.Mesh(vertices=crowded_soup(3000, crowd, w, h, 13))], cull=scenes.CULL_NONE)

    def check(frame, st, counts):
        assert counts.max() > crowd - 50
        if frame == 0:
            assert st["num_work_items"] == (counts > 0).sum()

    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        assert_frames(r, s, 2, check)


@pytest.mark.parametrize("chunk", [1, 16, 100])
def test_small_queue_chunks_with_bulk_copy_staging(gbr_lib, cuda_device, chunk):
    w, h = 256, 192
    s = scenes.soup_scene(20000, w, h, seed=14)

    def check(frame, st, counts):
        if frame:   # items of at least 64 entries, sized from the first frame's pairs
            assert st["num_work_items"] > (counts > 0).sum()

    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s, chunk)
        r.set_raster_staging(True)
        assert_frames(r, s, 2, check)


@pytest.mark.parametrize("vertex_colours", [True, False])   # shaded in one pass, and in two
@pytest.mark.parametrize("w,h,n", [(512, 384, 150_000), (256, 192, 60_000)])   # the scan kernel, and the scan in the fill pass
def test_drawn_triangles_of_a_frame_that_outgrows_its_list(gbr_lib, cuda_device, vertex_colours, w, h, n):
    """The set-up pass draws before the scan finds the list too small: the
    shade passes empty the merge buffer again, and the next frame shows
    nothing of it."""
    rng = np.random.default_rng(4)
    ang = rng.uniform(0, 2 * np.pi, (n, 1)) - np.arange(3) * (2 * np.pi / 3)
    centre, turn = rng.uniform(-0.9, 0.9, (n, 1, 2)), np.stack([np.cos(ang), -np.sin(ang)], -1)
    z = rng.uniform(0.05, 0.95, (n, 1))

    def mesh(px, shift):
        v = np.zeros(3 * n, scenes.IVERTEX56)
        p = v["p"].reshape(-1, 3, 3)
        p[:, :, :2] = centre + shift + px * 2.0 / np.array([w, h]) * turn
        p[:, :, 2] = z
        v["p"] = p.reshape(-1, 3)
        v["n"], v["tan"], v["c"], v["uv"] = (0, 0, 1), (1, 0, 0), 0.5, 0.25
        m = scenes.Mesh(vertices=v)
        if not vertex_colours:
            m.textures = [scenes.checker_texture(64, 8), scenes.flat_texture(64, (128, 128, 255)), None, None]
        return m

    px = np.full((n, 1, 1), 0.6)
    small = mesh(px, 0.0)
    px[::2] = 12.0
    large = mesh(px, 0.05)   # every second one too large for the set-up pass to draw
    s = scenes.Scene("direct", w, h, 4, 4, scenes.identity_camera(), [small], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    s.meshes = [large]
    big = oracle.render(s, oracle.RASTER_FIXED)
    s.meshes = [small]
    assert o["stats"]["num_pairs"] < 4 * o["stats"]["num_visible"]               # the following frames are drawn by the set-up pass
    assert big["stats"]["num_pairs"] > max(8 * n, 5 * o["stats"]["num_pairs"] // 4, 1 << 20)   # more than the list holds
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        for _ in range(2):
            r.render_scene(s)
            assert np.array_equal(r.readback_ids(), o["ids"])
        assert r.stats()["raster_lanes"] == 1 and r.stats()["overflow_reruns"] == 0
        r.update_vertices(0, large.vertices.ctypes.data, 3 * n)
        r.render_scene(s)   # outgrows the list; not read back
        r.update_vertices(0, small.vertices.ctypes.data, 3 * n)
        r.render_scene(s)
        _, depth = r.readback()
        assert r.stats()["overflow_reruns"] == 0
        assert np.array_equal(r.readback_ids(), o["ids"])
        assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32))
        r.update_vertices(0, large.vertices.ctypes.data, 3 * n)
        r.render_scene(s)
        _, depth = r.readback()   # rendered again with a longer list
        assert r.stats()["overflow_reruns"] >= 1
        assert np.array_equal(r.readback_ids(), big["ids"])
        assert np.array_equal(depth.view(np.uint32), big["depth"].view(np.uint32))
