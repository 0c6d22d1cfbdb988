"""A bin scan that gives up with more tiles than run at once: the tiles that
start after the flag was raised take part with all of their warps or with
none, and leave their bins' counts as they were.  The frame is reported as
GBR_ERR_TIMEOUT, and the next one counts from zero."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


def test_frame_after_a_scan_that_gave_up(gbr_lib, cuda_device):
    # 1024x1024 with 1x1 bins: 1,024 scan tiles, two a SM at once
    s = scenes.soup_scene(3000, 1024, 1024, 1, seed=19)
    with gbr_lib.Renderer(s.width, s.height) as r:
        r.load_scene(s)

        def frame():
            r.render_scene(s)
            _, depth = r.readback()
            offsets, bins = r.get_bins()
            return depth.copy(), r.readback_ids().copy(), offsets.copy(), bins.copy()

        good = frame()
        again = frame()   # the list holds the frame's entries from here on
        assert all(np.array_equal(x, y) for x, y in zip(good[:3], again[:3]))
        r.set_scan_wait(spin_limit=1, silent_tile=0)
        r.render_scene(s)
        with pytest.raises(gbr_lib.GbrError) as e:
            r.readback()
        assert e.value.status == 4, str(e.value)   # GBR_ERR_TIMEOUT
        r.set_scan_wait(0, -1)
        for _ in range(2):
            assert all(np.array_equal(x, y) for x, y in zip(again, frame()))
