"""How a frame's work items follow from the frame before it: the same scene,
rendered and checked again and again, settles by its third frame on one CTA
width and one item size, also where cutting the long lists takes the items' number
over the limit (three a SM) by which the width is chosen."""
import numpy as np
import pytest

import scenes
from frame_on_host import Frames, load


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return load(tmp_path_factory.mktemp("frame_on_host"))


def uneven_counts(bins, long_items, seed):
    """Entries of each bin: 20 to 90, and a few of 400."""
    n = np.random.default_rng(seed).integers(20, 91, bins)
    n[:: max(bins // max(long_items, 1), 1)][:long_items] = 400
    return n


@pytest.mark.parametrize("nbx,nby", [(20, 19), (21, 20), (43, 10), (25, 18), (38, 12), (457, 1), (50, 12)])   # 152 SMs: 456 is the limit
@pytest.mark.parametrize("long_items", [0, 10, 40])
@pytest.mark.parametrize("pairs_each", [8.0, 2.1])   # triangles that cover their bins 40 times over, and less than 3 times
def test_a_scene_settles(lib, nbx, nby, long_items, pairs_each):
    bins = uneven_counts(nbx * nby, long_items, seed=nbx)
    f = Frames(lib, nbx, nby, bins, int(bins.sum() / pairs_each))
    seen = []
    for _ in range(10):
        assert f.render() == 0
        st = f.stats()
        assert st["num_pairs"] == bins.sum() and st["raster_lanes"] == 0
        seen.append((f.last()["threads"], f.last()["chunk"], st["num_work_items"]))
    assert len(set(seen[2:])) == 1, seen
    assert (seen[-1][0] == 512) == (nbx * nby <= 456)
    few_layers = bins.sum() / pairs_each * (16 * (pairs_each - 1) - 4) ** 2 / 8 < 3.0 * 256 * len(bins)
    assert few_layers or pairs_each > 3 or long_items == 40
    mean = int(bins.sum()) // len(bins)
    assert seen[-1][1] == (64 if few_layers else max(2 * mean, 64) if seen[-1][0] == 512 and mean <= 64 else 512)
    f.close()


@pytest.mark.gpu
@pytest.mark.parametrize("route", ["fused scan", "scan kernel", "predicted"])
@pytest.mark.parametrize("nbx,nby", [(24, 18), (19, 24)])
def test_a_scene_settles_on_the_gpu(gbr_lib, cuda_device, nbx, nby, route):
    import ctypes as C
    from oracle import mlp_oracle
    w, h = 16 * nbx, 16 * nby
    counts = uneven_counts(nbx * nby, 10, seed=2)
    bin_of = np.repeat(np.arange(nbx * nby), counts)
    rng = np.random.default_rng(3)
    at = np.stack([bin_of % nbx, bin_of // nbx], -1) * 16.0 + 8.0   # a triangle some 11 px across in the middle of its bin
    ang = rng.uniform(0, 2 * np.pi, (len(at), 1)) - np.arange(3) * (2 * np.pi / 3)
    px = at[:, None, :] + 5.5 * np.stack([np.cos(ang), np.sin(ang)], -1)
    v = np.zeros(3 * len(at), scenes.POS3_RGBA8)
    v["p"][:, 0] = (2.0 * px[..., 0] / w - 1.0).reshape(-1)
    v["p"][:, 1] = (1.0 - 2.0 * px[..., 1] / h).reshape(-1)
    v["p"][:, 2] = np.repeat(rng.uniform(0.1, 0.9, len(at)), 3)
    s = scenes.Scene("uneven", w, h, 16, 16, scenes.identity_camera(), [scenes.Mesh(vertices=v)], cull=scenes.CULL_NONE)
    with gbr_lib.Renderer(w, h) as r:
        r.load_scene(s)
        r.set_raster_params(16, 0)   # a phase below 32: no triangle is left to the set-up pass
        if route == "scan kernel":
            r.set_scan_wait(1 << 20, -1)
        if route == "predicted":
            weights = np.zeros(mlp_oracle.NUM_PARAMS, np.float32)
            weights[mlp_oracle.OFF_B3] = 512.0
            w16 = mlp_oracle.f32_to_bf16(weights)
            gbr_lib.check(r._lib.gbr_set_predictor(r.h, w16.ctypes.data_as(C.c_void_p), len(w16), C.c_float(0.0),
                                                   C.c_float(0.0), C.c_float(0.0)))
            r.set_binning(gbr_lib.BINNING_PREDICTED)
        items = []
        for _ in range(10):
            r.render_scene(s)
            st = r.stats()
            assert st["num_pairs"] == counts.sum() and st["predicted_overflow"] == 0
            items.append(st["num_work_items"])
        assert len(set(items[2:])) == 1, items
        assert items[-1] == (-(-counts // 64)).sum()   # a layer of triangles: items of 64 entries


@pytest.mark.gpu
@pytest.mark.parametrize("bin_size", [16, 64])
def test_batches_of_few_layers_cut_their_lists(gbr_lib, cuda_device, bin_size):
    """Spheres cover their bins once or twice: items of 64 entries from the
    second frame on.  Soups cover them many times: items of 2048."""
    for make, chunk in ((lambda k: scenes.sphere_scene(320, 240, lon=64, lat=32 + k), 64),
                        (lambda k: scenes.soup_scene(20_000, 320, 240, seed=k), 2048)):
        sl = [make(k) for k in range(3)]
        with gbr_lib.Batch() as b:
            rs = []
            for s in sl:
                r = gbr_lib.Renderer(s.width, s.height)
                r.load_scene(s)
                b.add_scene(r, s)
                rs.append(r)
            b.set_config(bin_size, 4096)
            first = None
            for frame in range(4):
                b.render()
                counts = np.concatenate([np.diff(b.get_bins(i)[0].astype(np.int64)) for i in range(len(sl))])
                now = [b.readback(i)[2] for i in range(len(sl))]
                first = first or now
                assert all(np.array_equal(x, y) for x, y in zip(first, now))
                st = b.stats()
                assert st["num_work_items"] == (-(-counts // (chunk if frame else 2048))).sum()
            assert b.stats()["graph_captures"] <= 2
            b.close()
            for i, r in enumerate(rs):
                r.load_scene(sl[i])
                r.render_scene(sl[i])
                assert np.array_equal(r.readback_ids(), first[i])
                r.close()
