"""A frame one of whose launches fails half-way, on the host (frame_on_host):
the next frame starts from zero counts, zero counters and an empty merge
buffer, whatever the failed one had already left there."""
import numpy as np
import pytest

from frame_on_host import Frames, load

EMPTY = 0xFFFFFFFF


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return load(tmp_path_factory.mktemp("frame_on_host"))


@pytest.mark.parametrize("small", [False, True])   # triangles drawn by the raster, or by the set-up pass
@pytest.mark.parametrize("nbx,nby", [(20, 15), (80, 60)])   # the scan in the fill pass, and in a kernel of its own
def test_frame_after_a_failed_launch(lib, nbx, nby, small):
    rng = np.random.default_rng(1)
    bins = rng.integers(1, 9, nbx * nby)
    visible = int(bins.sum()) if small else int(bins.sum()) // 8
    f = Frames(lib, nbx, nby, bins, visible)
    for _ in range(2):
        assert f.render() == 0
        good, ids = f.stats(), f.ids()
    assert f.last()["direct"] == small and f.last()["fused"] == (nbx * nby <= 4096)
    assert good["num_pairs"] == bins.sum() and good["num_visible"] == visible
    for nth in range(1, 6):
        lib.host_fail_launch(nth)
        failed = f.render() != 0
        lib.host_fail_launch(0)
        assert failed == (nth <= (4 if nbx * nby <= 4096 else 5))
        for _ in range(2):
            assert f.render() == 0
            st = f.stats()
            assert all(st[k] == good[k] for k in ("num_pairs", "num_visible", "num_work_items")), nth
            assert np.array_equal(f.ids(), ids), nth
    f.close()
