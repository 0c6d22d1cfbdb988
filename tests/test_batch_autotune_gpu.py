"""The batch autotuner times what runs differently once: queue chunks that give
the raster the same pass are one configuration (every configuration is
captured anew), reported as the first of them."""
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads,chunks,same_as,best", [
    (128, (32, 64, 4096), (32,), {32}),                        # CTAs of 128 sort 1024 entries at once, whatever is asked
    (256, (64, 2048, 1024, 4096), (1024, 2048), {64, 2048}),   # CTAs of 256: 1024 to 2048
])
def test_autotune_times_equal_chunks_once(gbr_lib, cuda_device, threads, chunks, same_as, best):
    s = scenes.soup_scene(20000, 320, 240, seed=2)

    def tuned(chunk_list):
        with gbr_lib.Renderer(320, 240) as r, gbr_lib.Batch() as b:
            r.load_scene(s)
            b.add_scene(r, s)
            got = b.autotune(bin_sizes=(8, 16), chunks=chunk_list, raster_ctas=(4, 0), frames=1, raster_threads=(threads,))
            assert b.config() == got
            captures = b.stats()["graph_captures"]
            b.render()
            return got, captures, b.readback(0)[2]

    got, captures, ids = tuned(chunks)
    _, least, ids2 = tuned(same_as)
    assert got["queue_chunk"] in best and got["raster_ctas"] == 4   # 0: 4
    # the winner is captured once more unless it was timed last, and a bin
    # size's first frame may be captured again for its counters
    assert captures <= 2 * len(same_as) + 3 and least <= 2 * len(same_as) + 3
    assert (ids == ids2).all()
