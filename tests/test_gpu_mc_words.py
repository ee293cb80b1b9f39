"""Marching cubes over words of 32 points: row lengths around a word, and sparse volumes on both sides of the word rule."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def check(th, cuda, sdf, iso, unique, keep=None):
    if keep is None:
        ref = oracle.marching_cubes(sdf, iso, False, unique)
        vol = torch.from_numpy(sdf).to(cuda)
    else:
        idx = np.stack(np.nonzero(keep)).astype(np.int64)
        vals = sdf[keep]
        ref = oracle.marching_cubes(None, iso, False, unique, indices=idx, values=vals, size=sdf.shape)
        vol = torch.sparse_coo_tensor(torch.from_numpy(idx), torch.from_numpy(vals), sdf.shape).coalesce().to(cuda)
    v, f = th.marching_cubes(vol, iso, False, unique)
    assert np.array_equal(v.cpu().numpy(), ref[0])
    assert np.array_equal(f.cpu().numpy(), ref[1])
    return f.shape[0]


@pytest.mark.parametrize("width", [2, 31, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("kind", ["dense", "sparse", "holes"])
def test_rows_around_a_word(th, cuda, width, unique, kind):
    rng = np.random.default_rng(width)
    sdf = rng.normal(0.2, 0.5, size=(1, 6, 9, width)).astype(np.float32)
    sdf[rng.random(sdf.shape) < 0.05] = 0.3  # values on the isolevel
    keep = None if kind == "dense" else rng.random(sdf.shape) < (1.0 if kind == "sparse" else 0.9)
    n = check(th, cuda, sdf, 0.3, unique, keep)
    assert n > 0 or width == 2


def test_not_a_number_counts_as_above(th, cuda):
    sdf = np.full((1, 4, 5, 40), 1.0, dtype=np.float32)
    sdf[0, 2, 2, 30:34] = -1.0
    nan = sdf.copy()
    nan[0, 2, 2, 36] = np.nan
    a = th.marching_cubes(torch.from_numpy(sdf).to(cuda), 0.0, False)
    b = th.marching_cubes(torch.from_numpy(nan).to(cuda), 0.0, False)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("side", [20, 60])
def test_few_entries_in_a_large_volume(th, cuda, side, unique):
    """A small band far from the origin of a volume of 327,680 words: at side 20 the hash table is used, at 60 words."""
    sdf = np.full((1, 256, 256, 160), 5.0, dtype=np.float32)
    z, y, x = np.meshgrid(*[np.arange(side, dtype=np.float32) - (side - 1) / 2] * 3, indexing="ij")
    ball = np.sqrt(x * x + y * y + z * z) - 0.43 * side
    at = slice(150, 150 + side), slice(101, 101 + side), slice(90, 90 + side)
    sdf[0][at] = ball
    keep = np.zeros(sdf.shape, dtype=bool)
    keep[0][at] = np.abs(ball) <= (2 if side == 20 else 6)
    assert check(th, cuda, sdf, 0.0, unique, keep) > 100
