"""A request that does not fit the device's memory leaves nothing behind: the next one works."""

from __future__ import annotations

import ctypes

import pytest
import torch

from torchhull_gb300 import build, scenes

pytestmark = pytest.mark.gpu

FLOAT32, OUT_OF_MEMORY = 7, 4
# more views and pixels than fit: the allocations fail before anything is read
VIEWS, SIDE = 512, 1 << 15


class HullArgs(ctypes.Structure):
    _fields_ = [("masks", ctypes.c_void_p), ("masks_dtype", ctypes.c_int32), ("batch", ctypes.c_int64), ("height", ctypes.c_int64),
                ("width", ctypes.c_int64), ("transforms", ctypes.c_void_p), ("transforms_dtype", ctypes.c_int32),
                ("level", ctypes.c_int32), ("corner", ctypes.c_float * 3), ("length", ctypes.c_float), ("partial", ctypes.c_int32),
                ("opengl", ctypes.c_int32), ("unique", ctypes.c_int32)]


class HullInfo(ctypes.Structure):
    _fields_ = [("num_verts", ctypes.c_int64), ("num_faces", ctypes.c_int64), ("num_corners", ctypes.c_int64),
                ("num_levels", ctypes.c_int32), ("reserved", ctypes.c_int32), ("level_sizes", ctypes.c_int64 * 13)]


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("call", ["hull", "batch", "blur"])
def test_next_request_works(th, cuda, call):
    lib = ctypes.CDLL(str(build.LIB))
    ctx = ctypes.c_void_p()
    assert lib.th_context_create(ctypes.c_int32(0), ctypes.byref(ctx)) == 0
    r = scenes.make_request(5, 6, 128, 5, False, device="cpu")
    masks, transforms = r.masks.to(cuda), r.transforms.to(cuda)
    want = th.visual_hull(masks, transforms, r.level, r.cube_corner_bfl, r.cube_length, False, "opengl", True)
    blurred = th.gaussian_blur(masks, 9, 2.0)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def hull(views, side, name):
        a = HullArgs(masks.data_ptr(), FLOAT32, views, side, side, transforms.data_ptr(), FLOAT32, r.level,
                     (ctypes.c_float * 3)(*r.cube_corner_bfl), r.cube_length, 0, 1, 1)
        info = HullInfo()
        if name == "hull":
            return lib.th_visual_hull(ctx, ctypes.byref(a), stream, ctypes.byref(info)), info
        return lib.th_visual_hull_batch(ctx, ctypes.byref(a), ctypes.c_int32(1), stream, ctypes.byref(info)), info

    def blur(views, side, out):
        return lib.th_gaussian_blur(ctx, ptr(masks), ctypes.c_int32(FLOAT32), ctypes.c_int64(views), ctypes.c_int64(side),
                                    ctypes.c_int64(side), ctypes.c_int32(3 if views == VIEWS else 9), ctypes.c_float(2.0),
                                    ctypes.c_int32(1), ptr(out), ctypes.c_int32(FLOAT32), stream)

    try:
        out = torch.full_like(masks, -7.0)
        status = blur(VIEWS, SIDE, out) if call == "blur" else hull(VIEWS, SIDE, call)[0]
        assert status == OUT_OF_MEMORY
        if call == "blur":
            assert blur(6, 128, out) == 0
            assert torch.equal(out, blurred)
        else:
            status, info = hull(6, 128, call)
            assert status == 0 and (info.num_verts, info.num_faces) == (len(want[0]), len(want[1]))
            v, f = torch.empty_like(want[0]), torch.empty_like(want[1])
            export = (ctx, ptr(v), ptr(f), stream) if call == "hull" else (ctx, ctypes.c_int32(0), ptr(v), ptr(f), stream)
            assert (lib.th_visual_hull_export if call == "hull" else lib.th_visual_hull_batch_export)(*export) == 0
            assert torch.equal(v, want[0]) and torch.equal(f, want[1])
        torch.cuda.synchronize()
    finally:
        lib.th_context_destroy(ctx)
