"""Renderers, batches and bare-pointer calls with bins of different sizes in one
process: the raster's kernels are shared, so setting one up for small bins must
not take from another the shared memory that its large bins need."""
import ctypes as C

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def bare_call(gbr, s, torch, dev):
    v = torch.from_numpy(s.meshes[0].vertices.view(np.uint8).copy()).to(dev)
    out = [torch.empty(s.width * s.height, dtype=torch.int32, device=dev) for _ in range(3)]
    cam, world = gbr.make_camera(s.camera), (C.c_float * 16)(*[float(x) for x in scenes.identity16()])
    p = [C.c_void_p(x.data_ptr()) for x in (v, *out)]
    gbr.check(gbr.lib().gbr_render_noalloc(p[0], len(s.meshes[0].vertices), s.meshes[0].vertex_format, None, 0, 0, world,
                                           C.byref(cam), s.width, s.height, s.num_bins_x, s.num_bins_y, s.bin_w, s.bin_h,
                                           256, s.cull, s.sample, s.vis, p[1], p[2], p[3], None))
    torch.cuda.synchronize()
    return out[2].cpu().numpy().view(np.uint32).reshape(s.height, s.width)


@pytest.mark.parametrize("tma", [False, True])
def test_small_bins_set_up_after_large_ones(gbr_lib, cuda_device, tma):
    import torch
    few = scenes.soup_scene(2000, 640, 480, 64, seed=3)       # CTAs of 512 threads
    many = scenes.soup_scene(20_000, 2048, 1600, 64, seed=4)  # of 128
    small = scenes.soup_scene(2000, 320, 240, 8, seed=5)
    with gbr_lib.Renderer(640, 480) as a, gbr_lib.Renderer(2048, 1600) as b, gbr_lib.Renderer(320, 240) as c:
        before = {}
        for r, s in ((a, few), (b, many)):
            r.set_raster_staging(tma)
            r.load_scene(s)
            r.render_scene(s)
            before[r] = r.readback_ids()
        c.load_scene(small)
        bare = bare_call(gbr_lib, small, torch, cuda_device)
        c.render_scene(small)
        assert np.array_equal(bare, c.readback_ids())
        for r, s in ((a, few), (b, many), (c, small), (a, few)):
            r.render_scene(s)
            if r in before:
                assert np.array_equal(r.readback_ids(), before[r])


def test_batches_of_small_and_large_bins(gbr_lib, cuda_device):
    s = scenes.soup_scene(5000, 320, 240, seed=6)
    with gbr_lib.Renderer(320, 240) as r, gbr_lib.Renderer(320, 240) as q, gbr_lib.Batch() as a, gbr_lib.Batch() as b:
        for x, batch, size in ((r, a, 64), (q, b, 32)):
            x.load_scene(s)
            batch.add_scene(x, s)
            batch.set_config(size, 64)
            batch.render()
            batch.stats()
        a.set_view(0, s.camera, s.cull, s.sample, scenes.VIS_NORMAL)   # captured anew
        a.render()
        assert np.array_equal(a.readback(0)[2], b.readback(0)[2])
