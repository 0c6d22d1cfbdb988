"""Predicted binning whose blocks start late: while other work holds the SMs,
some blocks of the fused pass start after earlier ones have found a bin's
capacity exceeded and raised the overflow flag.  Such a block takes part with
all of its warps or with none (a part of them would store through counter
rows that nobody zeroed), and the exact pass that follows gives the oracle's
frame either way."""
import ctypes as C

import numpy as np
import pytest

import scenes
from oracle import mlp_oracle, oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,bin_size,n", [(640, 480, 16, 30_000),      # block rows in shared memory
                                            (2048, 1088, 8, 30_000)])    # more bins than they hold: an atomic a pair
def test_blocks_that_start_after_an_overflow(gbr_lib, cuda_device, w, h, bin_size, n):
    import torch
    s = scenes.soup_scene(n, w, h, bin_size, seed=29)
    o = oracle.render(s, oracle.RASTER_FIXED)
    weights = np.zeros(mlp_oracle.NUM_PARAMS, np.float32)
    weights[mlp_oracle.OFF_B3] = 2.0   # most bins hold more
    w16 = mlp_oracle.f32_to_bf16(weights)
    a = torch.randn(2048, 2048, device=cuda_device)
    busy = torch.cuda.Stream()
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        r.render_scene(s)
        r.stats()
        gbr_lib.check(r._lib.gbr_set_predictor(r.h, w16.ctypes.data_as(C.c_void_p), len(w16), C.c_float(0.0),
                                               C.c_float(0.0), C.c_float(0.0)))
        r.set_binning(gbr_lib.BINNING_PREDICTED)
        for frame in range(6):
            with torch.cuda.stream(busy):
                for _ in range(2 * frame):
                    b = a @ a
            r.render_scene(s)
            _, depth = r.readback()
            st = r.stats()
            assert st["predicted_overflow"] == 1
            assert st["num_visible"] == o["stats"]["num_visible"] and st["num_pairs"] == o["stats"]["num_pairs"]
            offsets, bins = r.get_bins()
            assert np.array_equal(offsets, o["offsets"]) and np.array_equal(bins, o["bins"]), f"frame {frame}: lists"
            assert np.array_equal(r.readback_ids(), o["ids"]), f"frame {frame}: winners"
            assert np.array_equal(depth.view(np.uint32), o["depth"].view(np.uint32)), f"frame {frame}: depth"
        torch.cuda.synchronize()
