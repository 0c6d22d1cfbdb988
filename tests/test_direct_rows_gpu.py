"""Frames of small triangles that count in block rows: lists with the drawn
entries behind the others, winners and depth are the oracle's, with the scan in
the fill pass and in a kernel of its own, in a frame of two meshes."""
import numpy as np
import pytest

import scenes
from oracle import oracle

pytestmark = pytest.mark.gpu


def small_triangles(n, w, h, px, seed):
    """n triangles of up to `px` px across, a few large ones and one beyond the
    guard band among them."""
    rng = np.random.default_rng(seed)
    v = np.zeros(3 * n, scenes.POS3_RGBA8)
    p = v["p"].reshape(-1, 3, 3)
    ang = rng.uniform(0, 2 * np.pi, (n, 1)) - np.arange(3) * (2 * np.pi / 3)
    size = rng.uniform(0.1 * px, px, (n, 1, 1)) / np.array([w, h])
    p[:, :, :2] = rng.uniform(-0.95, 0.95, (n, 1, 2)) + size * np.stack([np.cos(ang), -np.sin(ang)], -1)
    p[:, :, 2] = rng.uniform(0.05, 0.95, (n, 1))
    p[:: max(n // 12, 1), 0, :2] += 0.3
    p[7, 0, 0] = 60.0 * 2048 / w
    v["p"] = p.reshape(-1, 3)
    v["rgba"] = rng.integers(0, 2**32, 3 * n, dtype=np.uint64).astype(np.uint32)
    return v


@pytest.mark.parametrize("w,h,bw,bh,n,px", [
    (256, 256, 4, 4, 180_000, 3.8),      # 4096 bins: the last with the scan in the fill pass
    (260, 256, 4, 4, 180_000, 3.8),      # 4160: the scan kernel
    (64, 64, 64, 64, 70_000, 3.0),      # one bin
    (333, 250, 24, 20, 65_000, 3.0),    # ragged
])
def test_direct_frames_in_block_rows(gbr_lib, cuda_device, w, h, bw, bh, n, px):
    import torch
    v = small_triangles(n, w, h, px, seed=n + w)
    cut = 3 * (n // 3)
    s = scenes.Scene("two", w, h, bw, bh, scenes.identity_camera(),
                     [scenes.Mesh(vertices=v[:cut].copy()), scenes.Mesh(vertices=v[cut:].copy())], cull=scenes.CULL_NONE)
    o = oracle.render(s, oracle.RASTER_FIXED)
    blocks = min((n + 1023) // 1024, torch.cuda.get_device_properties(0).multi_processor_count)
    assert o["stats"]["num_pairs"] >= max(1 << 16, s.num_bins_x * s.num_bins_y * blocks)
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        for frame in range(3):
            r.render_scene(s)
            _, depth = r.readback()
            st = r.stats()
            assert (st["raster_lanes"], st["count_blocks"]) == ((1, blocks) if frame else (0, 0))
            assert st["num_visible"] == o["stats"]["num_visible"] and st["num_pairs"] == o["stats"]["num_pairs"]
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"]), f"frame {frame}: lists"
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners"
            assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth"
