"""The bin scan inside the fill pass around the limits of its rule (4096 bins,
2^16 triangles; the block-row path whatever its bins) and its 32-bin rows:
bin lists and winners of the frame are the oracle's, frame after frame (the
raster leaves the counts zero for the next)."""
import ctypes as C

import numpy as np
import pytest

import scenes
from oracle import mlp_oracle, oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,bin_size,n", [
    (16, 16, 16, 40),            # one bin (and a pair a triangle: taken for small triangles)
    (31 * 4, 4, 4, 300),         # one row of bins short of 32, whole, and one over
    (32 * 4, 4, 4, 300),
    (33 * 4, 4, 4, 300),
    (64, 64, 1, 200),            # 4096 bins: the last fused size on one counter a bin
    (241, 17, 1, 200),           # 4097: the scan kernel
    (320, 240, 16, 65536),       # the last triangle count, and one over
    (320, 240, 16, 65537),
    (512, 256, 4, 40000),        # 8192 bins in block rows
])
def test_fused_scan_against_the_oracle(gbr_lib, cuda_device, w, h, bin_size, n):
    import torch
    s = scenes.soup_scene(n, w, h, bin_size, seed=41)
    o = oracle.render(s, oracle.RASTER_FIXED)
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        for frame in range(3):
            r.render_scene(s)
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"]), f"frame {frame}"
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}"
            st = r.stats()
            assert st["num_pairs"] == o["stats"]["num_pairs"] and st["num_visible"] == o["stats"]["num_visible"]
            # later frames count in block rows (the first frame showed at
            # least a pair per (block, bin)), but for one of small triangles,
            # whose lists keep apart what the set-up pass has drawn
            blocks = min((n + 1023) // 1024, torch.cuda.get_device_properties(0).multi_processor_count)
            assert st["num_pairs"] >= s.num_bins_x * s.num_bins_y * blocks
            assert st["count_blocks"] == (blocks if frame and not st["raster_lanes"] else 0)


def test_bin_features_after_a_predicted_frame(gbr_lib, cuda_device):
    """The pre-pass counts its samples into the control block before a fused
    scan clears it: what a predicted frame left there must not count."""
    s = scenes.soup_scene(20_000, 640, 480, seed=5)
    s.bin_w = s.bin_h = 16
    nb = s.num_bins_x * s.num_bins_y
    weights = np.zeros(mlp_oracle.NUM_PARAMS, np.float32)
    weights[mlp_oracle.OFF_B3] = 60.0
    w16 = mlp_oracle.f32_to_bf16(weights)

    def features(predicted_first):
        with gbr_lib.Renderer(s.width, s.height) as r:
            r.load_scene(s)
            r.render_scene(s)
            r.stats()
            if predicted_first:
                gbr_lib.check(r._lib.gbr_set_predictor(r.h, w16.ctypes.data_as(C.c_void_p), len(w16), C.c_float(0.0),
                                                       C.c_float(0.0), C.c_float(0.0)))
                r.set_binning(gbr_lib.BINNING_PREDICTED)
                r.render_scene(s)
                r.stats()
            x, counts = np.zeros((nb, 12), np.float32), np.zeros(nb, np.uint32)
            cam = gbr_lib.make_camera(s.camera)
            gbr_lib.check(r._lib.gbr_collect_bin_features(r.h, C.byref(cam), s.cull, s.sample, s.vis,
                                                          x.ctypes.data_as(C.c_void_p), counts.ctypes.data_as(C.c_void_p), None))
            return x, counts

    x0, c0 = features(False)
    x1, c1 = features(True)
    assert np.array_equal(c0, c1)
    assert np.array_equal(x0[:, 11], x1[:, 11])   # the samples' density, of a whole number
