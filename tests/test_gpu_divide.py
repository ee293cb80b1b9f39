"""The projection's shared-reciprocal division equals the IEEE division, bit for bit."""

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


@pytest.fixture(scope="module")
def probe():
    lib = HERE / "_build" / "libdivide_probe.so"
    src = HERE / "divide_probe.cu"
    lib.parent.mkdir(parents=True, exist_ok=True)
    nvcc = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "bin" / "nvcc"
    subprocess.run([str(nvcc) if nvcc.exists() else (shutil.which("nvcc") or "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a",
                    "-O3", "-std=c++20", "-shared", "-Xcompiler", "-fPIC", "-o", str(lib), str(src)], check=True,
                   capture_output=True)
    return ctypes.CDLL(str(lib))


def floats(n, seed, cuda, low, high):
    """Random signs and mantissas with exponents in [low, high)."""
    g = torch.Generator(device=cuda).manual_seed(seed)
    mant = torch.randint(0, 1 << 23, (n,), generator=g, device=cuda, dtype=torch.int64)
    expo = torch.randint(127 + low, 127 + high, (n,), generator=g, device=cuda, dtype=torch.int64)
    sign = torch.randint(0, 2, (n,), generator=g, device=cuda, dtype=torch.int64)
    bits = (sign << 31) | (expo << 23) | mant
    return (bits - ((bits >= 1 << 31).to(torch.int64) << 32)).to(torch.int32).view(torch.float32)


@pytest.mark.parametrize("low,high", [(-2, 3), (-30, 30)])
def test_divide_pair(probe, cuda, low, high):
    n = 1 << 24
    a, b, d = (floats(n, s, cuda, low, high) for s in (1, 2, 3))
    d = d.abs()
    # exact quotients, equal and neighbouring operands, and divisors outside the fast range
    a[:1000] = d[:1000]
    a[1000:2000] = d[1000:2000] * 3
    a[2000:3000] = torch.nextafter(d[2000:3000], torch.full_like(d[2000:3000], 1e30))
    d[3000:3100] = 0.0
    d[3100:3200] = float("inf")
    d[3200:3300] = -1.5
    d[3300:3400] = 1e-30
    differ = torch.zeros(1, dtype=torch.int64, device=cuda)
    torch.cuda.synchronize()
    rc = probe.divide_probe(ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), ctypes.c_void_p(d.data_ptr()),
                            ctypes.c_longlong(n), ctypes.c_void_p(differ.data_ptr()))
    assert rc == 0 and differ.item() == 0
