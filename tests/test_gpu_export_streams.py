"""Exports of one result on several streams of the C ABI: the next request waits for all of them."""

from __future__ import annotations

import ctypes

import pytest
import torch

from torchhull_gb300 import build, scenes

pytestmark = pytest.mark.gpu

FLOAT32 = 7
SLEEP = 100_000_000  # clock cycles: about 50 ms


class HullArgs(ctypes.Structure):
    _fields_ = [("masks", ctypes.c_void_p), ("masks_dtype", ctypes.c_int32), ("batch", ctypes.c_int64), ("height", ctypes.c_int64),
                ("width", ctypes.c_int64), ("transforms", ctypes.c_void_p), ("transforms_dtype", ctypes.c_int32),
                ("level", ctypes.c_int32), ("corner", ctypes.c_float * 3), ("length", ctypes.c_float), ("partial", ctypes.c_int32),
                ("opengl", ctypes.c_int32), ("unique", ctypes.c_int32)]


class HullInfo(ctypes.Structure):
    _fields_ = [("num_verts", ctypes.c_int64), ("num_faces", ctypes.c_int64), ("num_corners", ctypes.c_int64),
                ("num_levels", ctypes.c_int32), ("reserved", ctypes.c_int32), ("level_sizes", ctypes.c_int64 * 13)]


class McArgs(ctypes.Structure):
    _fields_ = [("sparse", ctypes.c_int32), ("dtype", ctypes.c_int32), ("depth", ctypes.c_int64), ("height", ctypes.c_int64),
                ("width", ctypes.c_int64), ("volume", ctypes.c_void_p), ("indices", ctypes.c_void_p), ("values", ctypes.c_void_p),
                ("nnz", ctypes.c_int64), ("isolevel", ctypes.c_float), ("local", ctypes.c_int32), ("unique", ctypes.c_int32)]


class McInfo(ctypes.Structure):
    _fields_ = [("num_verts", ctypes.c_int64), ("num_faces", ctypes.c_int64)]


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def on(stream):
    return ctypes.c_void_p(stream.cuda_stream)


@pytest.fixture
def context(cuda):
    lib = ctypes.CDLL(str(build.LIB))
    ctx = ctypes.c_void_p()
    assert lib.th_context_create(ctypes.c_int32(0), ctypes.byref(ctx)) == 0
    yield lib, ctx
    lib.th_context_destroy(ctx)


def mesh(verts, faces, cuda):
    return (torch.full((verts, 3), -7.0, device=cuda), torch.full((faces, 3), -7, dtype=torch.int64, device=cuda))


def equal(made, want):
    return all(torch.equal(a, b) for a, b in zip(made, want))


@pytest.mark.parametrize("depth", [60, 1 << 19])  # the second: rows of two points and more than 2^27 words, slab by slab
def test_marching_cubes(th, context, cuda, depth):
    lib, ctx = context
    shape = (1, depth, 60, 70) if depth == 60 else (1, depth, 300, 2)
    g = torch.Generator(device=cuda).manual_seed(3)
    volumes = []
    for i in range(2):
        v = torch.ones(shape, device=cuda)
        v[:, 20:50, 20:50] = torch.rand((1, 30, 30, shape[3]), generator=g, device=cuda) - 0.3 - 0.2 * i
        volumes.append(v)
    want = [th.marching_cubes(v, 0.0, False) for v in volumes]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()

    def count(v, stream):
        args = McArgs(0, FLOAT32, *shape[1:], v.data_ptr(), None, None, 0, 0.0, 0, 1)
        info = McInfo()
        assert lib.th_marching_cubes(ctx, ctypes.byref(args), on(stream), ctypes.byref(info)) == 0
        made = mesh(info.num_verts, info.num_faces, cuda)
        torch.cuda.synchronize()
        return made

    def export(made, stream):
        assert lib.th_marching_cubes_export(ctx, ptr(made[0]), ptr(made[1]), on(stream)) == 0

    first = count(volumes[0], streams[0])
    again = tuple(torch.empty_like(t) for t in first)
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(SLEEP)
    export(first, streams[0])
    export(again, streams[1])
    other = count(volumes[1], streams[2])
    export(other, streams[2])
    torch.cuda.synchronize()
    assert equal(first, want[0]) and equal(again, want[0]) and equal(other, want[1])


def test_hull(th, context, cuda):
    lib, ctx = context
    reqs = [scenes.make_request(90 + i, 6, 128, 6, False, device=cuda) for i in range(2)]
    want = [th.visual_hull_with_candidate_voxels(**r.kwargs()) for r in reqs]
    streams = [torch.cuda.Stream() for _ in range(4)]
    torch.cuda.synchronize()

    def run(r, stream):
        masks, transforms = r.masks.contiguous(), r.transforms.contiguous()
        args = HullArgs(masks.data_ptr(), FLOAT32, *masks.shape[:3], transforms.data_ptr(), FLOAT32, r.level,
                        (ctypes.c_float * 3)(*r.cube_corner_bfl), r.cube_length, int(r.masks_partial),
                        int(r.transforms_convention == "opengl"), int(r.unique_verts))
        info = HullInfo()
        assert masks.dtype == transforms.dtype == torch.float32
        assert lib.th_visual_hull(ctx, ctypes.byref(args), on(stream), ctypes.byref(info)) == 0
        made = mesh(info.num_verts, info.num_faces, cuda)
        leaves = [torch.full((info.level_sizes[r.level],), -7, dtype=torch.int64, device=cuda) for _ in range(2)]
        torch.cuda.synchronize()
        return made, leaves

    made, leaves = run(reqs[0], streams[0])
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(SLEEP)
    assert lib.th_visual_hull_export(ctx, ptr(made[0]), ptr(made[1]), on(streams[0])) == 0
    for i in range(2):  # both write the leaf list out
        assert lib.th_visual_hull_export_candidates(ctx, ctypes.c_int32(reqs[0].level), ptr(leaves[i]), on(streams[1 + i])) == 0
    other, _ = run(reqs[1], streams[3])
    assert lib.th_visual_hull_export(ctx, ptr(other[0]), ptr(other[1]), on(streams[3])) == 0
    torch.cuda.synchronize()
    assert equal(made, want[0][:2]) and equal(other, want[1][:2])
    assert all(torch.equal(x, want[0][2][reqs[0].level]) for x in leaves)
