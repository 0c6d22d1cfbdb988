"""A frame captured into the caller's CUDA graph and replayed over vertices that
move: every replay shows what an ordinary frame of the same vertices does,
nothing of the replay before it (frames shaded in two passes leave bins that
stay clean untouched)."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def moving_sphere(textured):
    s = scenes.sphere_scene(640, 480)
    s.meshes[0].vertices["p"] *= 0.4
    if not textured:
        s.meshes[0].textures = [None] * 4
    return s


@pytest.mark.parametrize("textured,route", [(True, "fused scan"), (True, "scan kernel"), (True, "predicted"), (True, "tma"),
                                            (False, "fused scan")])   # shaded in two passes, and in one
def test_replays_over_moving_vertices(gbr_lib, cuda_device, textured, route):
    import ctypes as C
    import torch
    from oracle import mlp_oracle
    s = moving_sphere(textured)
    m = s.meshes[0]
    at = [(0.0, 0.0), (0.9, 0.3), (-0.9, -0.4), (0.2, 0.7), (0.0, 0.0)]

    def placed(dx, dy):
        v = m.vertices.copy()
        v["p"][:, 0] += dx
        v["p"][:, 1] += dy
        return torch.from_numpy(v.view(np.uint8).reshape(-1).copy()).to(cuda_device)

    ix = torch.from_numpy(np.ascontiguousarray(m.indices, np.uint32).view(np.int32)).to(cuda_device)

    def renderer(v):
        r = gbr_lib.Renderer(s.width, s.height)
        r.setup_bins(s.num_bins_x, s.num_bins_y, s.bin_w, s.bin_h)
        tex = [r.add_texture(t) if t is not None else -1 for t in m.textures]
        r.bind_mesh_device(v.data_ptr(), len(m.vertices), m.vertex_format, ix.data_ptr(), len(m.indices), m.topology,
                           m.world, tex)
        r.set_raster_staging(route == "tma")
        if route == "scan kernel":
            r.set_scan_wait(1 << 20, -1)
        if route == "predicted":
            weights = np.zeros(mlp_oracle.NUM_PARAMS, np.float32)
            weights[mlp_oracle.OFF_B3] = 512.0   # more than any bin holds
            w16 = mlp_oracle.f32_to_bf16(weights)
            gbr_lib.check(r._lib.gbr_set_predictor(r.h, w16.ctypes.data_as(C.c_void_p), len(w16), C.c_float(0.0),
                                                   C.c_float(0.0), C.c_float(0.0)))
            r.set_binning(gbr_lib.BINNING_PREDICTED)
        return r

    want = []
    for dx, dy in at:
        v = placed(dx, dy)
        with renderer(v) as r:
            r.render_scene(s)
            want.append([x.copy() for x in (*r.readback(), r.readback_ids())])
    assert not np.array_equal(want[0][2], want[1][2])
    v = placed(*at[0])
    with renderer(v) as r:
        for _ in range(3):
            r.render_scene(s)
            r.readback()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            r.render_scene(s, stream=torch.cuda.current_stream().cuda_stream)
        for k in (1, 2, 3, 0, 2):
            v.copy_(placed(*at[k]))
            g.replay()
            torch.cuda.synchronize()
            got = (*r.readback(), r.readback_ids())
            for x, y, what in zip(got, want[k], ("colour", "depth", "ids")):
                assert np.array_equal(x, y), f"place {k}: {what}"
        r.render_scene(s)   # and an ordinary frame after them
        assert np.array_equal(r.readback_ids(), want[2][2])
