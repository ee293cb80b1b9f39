"""What the mesh stages number with 32 bits is refused beyond them, not wrapped."""

from __future__ import annotations

import ctypes
import os
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent / "probe"
CORNERS, INDICES = 2, 4  # OverflowBits


@pytest.fixture(scope="module")
def probe():
    lib = HERE / "_build" / "libmesh_probe.so"
    lib.parent.mkdir(parents=True, exist_ok=True)
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    subprocess.run([str(nvcc) if nvcc.exists() else (shutil.which("nvcc") or "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O1", "-std=c++20", "-shared", "-Xcompiler", "-fPIC", "-o", str(lib), str(HERE / "mesh_probe.cu")],
                   check=True, capture_output=True)
    made = ctypes.CDLL(str(lib))
    made.counters_bytes.restype = ctypes.c_longlong
    return made


def count_corners(probe, cuda, level, full_rows, last_points, room):
    """Overflow bits and corners when the first full_rows rows of a level's bitmap hold all their points, and the next one
    its first last_points; room for `room` corners."""
    r = (1 << level) + 1
    wr = (r + 63) // 64
    bitmap = torch.zeros((full_rows + 1, wr), dtype=torch.int64, device=cuda)
    bitmap[:full_rows, : r // 64] = -1
    bitmap[:full_rows, r // 64] = (1 << r % 64) - 1
    bitmap[full_rows, : last_points // 64] = -1
    if last_points % 64:
        bitmap[full_rows, last_points // 64] = (1 << last_points % 64) - 1
    rowbits = torch.zeros(((r * r + 31) // 32 + 3) // 4 * 4, dtype=torch.int32, device=cuda)
    touched = full_rows + (last_points > 0)
    rowbits[: touched // 32] = -1
    if touched % 32:
        rowbits[touched // 32] = (1 << touched % 32) - 1
    ints = lambda n: torch.zeros(n, dtype=torch.int32, device=cuda)  # noqa: E731
    rows, row_slot, row_place, row_cnt = ints(r * r), ints(r * r), ints(12 * (touched + 1)), ints(2 * (touched + 1))
    corners = torch.zeros(room, dtype=torch.int64, device=cuda)
    counters = torch.zeros(probe.counters_bytes(level), dtype=torch.uint8, device=cuda)
    result = (ctypes.c_longlong * 2)()
    torch.cuda.synchronize()
    at = [ctypes.c_void_p(t.data_ptr()) for t in (bitmap, rowbits, rows, row_slot, row_place, row_cnt, corners)]
    rc = probe.corners_probe(ctypes.c_int(level), *at, ctypes.c_longlong(room), ctypes.c_void_p(counters.data_ptr()), result)
    assert rc == 0
    return result[0], result[1], corners


@pytest.mark.parametrize("extra", [-4097 * 4, 0, 3000])
def test_corner_count_beyond_32_bits(probe, cuda, extra):
    """Level 12, 2^32 + extra corners, room for 4096."""
    full_rows, last = divmod((1 << 32) + extra, 4097)
    overflow, corners, _ = count_corners(probe, cuda, 12, full_rows, last, 4096)
    assert overflow & (CORNERS if extra < 0 else INDICES)
    assert corners == 0


def test_corners_that_fit(probe, cuda):
    overflow, _, corners = count_corners(probe, cuda, 12, 2, 100, 3 * 4097)
    assert not overflow & (CORNERS | INDICES)
    x = torch.arange(4097, device=cuda)
    want = torch.cat([x, x + (1 << 21), x[:100] + (2 << 21)])
    assert torch.equal(corners[: len(want)], want)


@pytest.mark.parametrize("words", [1000, (1 << 32) // 372, (1 << 32) // 372 + 1, 12_000_000])
def test_triangle_corners_beyond_32_bits(probe, cuda, words):
    """31 cells of 12 triangle corners in each word."""
    ints = lambda n: torch.zeros(n, dtype=torch.int32, device=cuda)  # noqa: E731
    cnt, cells, tiles = ints(words), ints(words), ints(2 * (words // 1024 + 1))
    counters = torch.zeros(2 * probe.counters_bytes(1), dtype=torch.uint8, device=cuda)
    result = (ctypes.c_longlong * 2)()
    torch.cuda.synchronize()
    at = [ctypes.c_void_p(t.data_ptr()) for t in (cnt, cells, tiles, counters)]
    rc = probe.triangles_probe(ctypes.c_longlong(words), *at, result)
    assert rc == 0
    assert bool(result[0] & INDICES) == (words * 372 >= 1 << 32)
    if not result[0]:
        assert result[1] == words * 372
