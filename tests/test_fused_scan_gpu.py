"""The bin scan inside the fill pass around the limits of its rule (4096 bins,
2^16 triangles; the block-row path whatever its bins) and its 32-bin rows:
bin lists and winners of the frame are the oracle's, frame after frame (the
raster leaves the counts zero for the next)."""
import numpy as np
import pytest

import scenes
from oracle import oracle

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
