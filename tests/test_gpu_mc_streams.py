"""Marching cubes of one context on several streams share its buffers: each mesh is its own."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def volumes(kind, cuda):
    """Four volumes of one size with different surfaces."""
    g = torch.Generator().manual_seed(23)
    out = []
    for i in range(4):
        v = (torch.rand((1, 60, 70, 80), generator=g) - 0.3 - 0.1 * i).to(cuda)
        if kind == "dense":
            out.append(v)
            continue
        if kind == "words":
            held = torch.rand(v.shape, generator=g).to(cuda) < 0.98
            index = held.nonzero().T.contiguous()
            out.append(torch.sparse_coo_tensor(index, v[tuple(index)], v.shape).coalesce())
            continue
        # single cells in a volume with very many words for its entries
        at = (torch.rand(v.shape, generator=g) < 0.0005).nonzero().T.to(cuda)
        index = torch.cat([at + torch.tensor([[0], [z], [y], [x]], device=cuda) for z in (0, 1) for y in (0, 1) for x in (0, 1)], 1)
        values = torch.rand(index.shape[1], generator=g).to(cuda) - 0.5
        out.append(torch.sparse_coo_tensor(index, values, (1, 600, 700, 800)).coalesce())
    return out


@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("kind", ["dense", "words", "hash"])
def test_interleaved_streams(th, cuda, kind, unique):
    inputs = volumes(kind, cuda)
    want = [th.marching_cubes(v, 0.0, False, unique) for v in inputs]
    assert all(len(w[1]) > 0 for w in want)
    streams = [torch.cuda.Stream() for _ in inputs]
    torch.cuda.synchronize()
    got = [[] for _ in inputs]
    for _ in range(8):
        for i, (v, s) in enumerate(zip(inputs, streams)):
            with torch.cuda.stream(s):
                got[i].append(th.marching_cubes(v, 0.0, False, unique))
    torch.cuda.synchronize()
    for w, made in zip(want, got):
        for m in made:
            assert torch.equal(w[0], m[0]) and torch.equal(w[1], m[1])
