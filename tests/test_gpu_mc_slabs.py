"""Dense volumes whose words need too much scratch go through slab by slab: the mesh is that of the whole volume."""

from __future__ import annotations

import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu

# 12000 words a plane, more than 2^27 words in all: the first slab ends at plane 11182
SIZES = (12000, 12000, 3)
# planes with a surface: at the start, across the slabs' border, behind it, at the end
PARTS = [(0, 30), (11150, 11210), (11300, 11303), (11980, 12000)]
Y = slice(7500, 7560)


@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32, torch.float64])
def test_slabs(th, cuda, dtype, unique):
    g = torch.Generator().manual_seed(31)
    volume = torch.ones((1, *SIZES), dtype=dtype, device=cuda)
    verts, faces, count = [], [], 0
    for z0, z1 in PARTS:
        part = (torch.rand((1, z1 - z0, 60, 3), generator=g) - 0.4).to(dtype)
        part[:, :, 0] = part[:, :, -1] = 1.0
        if z0 > 0:
            part[:, 0] = 1.0
        if z1 < SIZES[0]:
            part[:, -1] = 1.0
        volume[:, z0:z1, Y] = part.to(cuda)
        v, f = oracle.marching_cubes(part, 0.0, False, unique)
        verts.append(torch.as_tensor(v) + torch.tensor([0.0, Y.start, z0]))
        faces.append(torch.as_tensor(f) + count)
        count += len(v)
    got_verts, got_faces = th.marching_cubes(volume, 0.0, False, unique)
    assert torch.equal(got_faces.cpu(), torch.cat(faces))
    # coordinates below 2^14: two roundings of half a unit in the last place each
    torch.testing.assert_close(got_verts.cpu(), torch.cat(verts).float(), rtol=0, atol=2.0**-9)
