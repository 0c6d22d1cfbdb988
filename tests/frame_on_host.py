"""The frame's host path (gbr_api.cu) on host memory, for tests without a GPU:
builds tests/cpp/*_on_host.* against the library's own object file."""
import ctypes as C
import os
import subprocess

import numpy as np

import build as gbr_build
import gbr
import scenes


def load(tmp_dir) -> C.CDLL:
    gbr_build.build(force=not os.path.exists(os.path.join(gbr_build.OUT_DIR, "gbr_api.o")))
    lib = os.path.join(str(tmp_dir), "frame_on_host.so")
    src = [os.path.join(gbr_build.ROOT, "tests", "cpp", f) for f in ("frame_on_host.cu", "cuda_on_host.cpp")]
    subprocess.run([gbr_build.nvcc(), "-shared", "-cudart", "none", "-std=c++17", "-O1", *gbr_build.ARCH, "-Xcompiler",
                    "-fPIC", "-Xlinker", "-Bsymbolic", "-I", gbr_build.CSRC, *src, os.path.join(gbr_build.OUT_DIR, "gbr_api.o"), "-o", lib], check=True)
    return C.CDLL(lib)


class Frames:
    """A renderer of one mesh over bins of 16x16 pixels; render() and stats()
    as the library answers them for the bins' entry counts in `bins`."""

    def __init__(self, lib, nbx, nby, bins, visible):
        self.lib, self.bins = lib, np.asarray(bins, np.uint32)
        assert len(self.bins) == nbx * nby
        lib.host_set_bins(self.bins.ctypes.data_as(C.c_void_p), C.c_uint32(len(self.bins)), C.c_uint32(visible))
        self.w, self.h = 16 * nbx, 16 * nby
        self.r = C.c_void_p()
        self.check(lib.gbr_create(C.c_uint32(self.w), C.c_uint32(self.h), C.byref(self.r)))
        self.check(lib.gbr_setup_bins(self.r, *(C.c_uint32(x) for x in (nbx, nby, 16, 16, 4096))))
        v = np.zeros(3 * visible, scenes.POS3_RGBA8)
        world = (C.c_float * 16)(*np.eye(4, dtype=np.float32).reshape(16))
        self.check(lib.gbr_mesh_upload(self.r, v.ctypes.data_as(C.c_void_p), C.c_uint32(len(v)), C.c_uint32(1), None,
                                       C.c_uint32(0), C.c_uint32(0), world, None, None))
        self.cam = gbr.make_camera(scenes.identity_camera())

    @staticmethod
    def check(status):
        assert status == 0, status

    def render(self):
        return self.lib.gbr_render(self.r, C.byref(self.cam), C.c_uint32(2), C.c_uint32(0), C.c_uint32(0), None)

    def stats(self):
        st = gbr.Stats()
        self.check(self.lib.gbr_get_stats(self.r, C.byref(st), None))
        return {k: getattr(st, k) for k, _ in gbr.Stats._fields_}

    def ids(self):
        out = np.zeros(self.w * self.h, np.uint32)
        self.check(self.lib.gbr_readback_ids(self.r, out.ctypes.data_as(C.c_void_p), None))
        return out

    def last(self):
        out = (C.c_uint32 * 4)()
        self.lib.host_last_frame(out)
        return dict(zip(("chunk", "threads", "direct", "fused"), out))

    def close(self):
        self.lib.gbr_destroy(self.r)
