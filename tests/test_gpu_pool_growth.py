"""Requests that outgrow the pools a context starts with run again: their own result and the ones after it are as ever."""

from __future__ import annotations

import functools

import numpy as np
import pytest
import torch

from oracle import oracle
from torchhull_gb300 import scenes

pytestmark = pytest.mark.gpu

CORNER, LENGTH = (-1.0, -1.0, -1.0), 2.0


def request(masks, transforms, level, partial=False):
    return masks, transforms, level, CORNER, LENGTH, partial, "opengl", True


def views(*rows):
    """Transforms whose pixel coordinates are the given rows (x row, y row) of the world point."""
    t = torch.zeros((len(rows), 4, 4))
    for i, (x, y) in enumerate(rows):
        t[i, 0], t[i, 1], t[i, 3, 3] = torch.tensor(x), torch.tensor(y), 1.0
    return t


def full(swap):
    """Level 8, every cell refined: 19.2 M nodes and 17.0 M corners where the pools start at 16.8 M.  One view sees the
    whole cube, the other a quarter of it, so that view masks are set."""
    g = torch.Generator().manual_seed(41)
    masks = 0.3 + 0.1 * torch.rand((2, 400, 400, 1), generator=g)
    masks[:, 150:230, 130:220] = 0.9
    wide, near = ((0.8, 0.0, 0.0, 0.0), (0.0, 0.8, 0.0, 0.0)), ((0.0, 0.0, 1.6, 0.4), (0.0, 1.6, 0.0, 0.4))
    return request(masks, views(*((near, wide) if swap else (wide, near))), 8, True)


def planes(at):
    """Level 10, planes x = const: nearly every row of the grid holds corners, 35.7 M words where there is room for 33.5."""
    masks = torch.zeros((1, 16, 2048, 1))
    for x in at:
        masks[:, :, x : x + 6] = 1.0
    return request(masks, views(((0.5, 0.0, 0.0, 0.0), (0.0, 0.5, 0.0, 0.0))), 10)


def small(seed, level=5):
    r = scenes.make_request(seed, 5, 96, level, False, device="cpu")
    return request(r.masks, r.transforms, level)


REQUESTS = {"full": functools.partial(full, False), "full, views swapped": functools.partial(full, True),
            "plane": functools.partial(planes, (900,)), "planes": functools.partial(planes, (700, 1300)),
            "small": functools.partial(small, 51, 8)}
REQUESTS.update({f"small {i}": functools.partial(small, 60 + i) for i in range(8)})


@functools.cache
def expected(name):
    return oracle.visual_hull(*REQUESTS[name]())


def on(cuda, name):
    masks, transforms, *rest = REQUESTS[name]()
    return (masks.to(cuda), transforms.to(cuda), *rest)


def same(got, name):
    want = expected(name)
    assert len(want.faces) > 0
    return np.array_equal(got[0].cpu().numpy(), want.verts) and np.array_equal(got[1].cpu().numpy(), want.faces)


@pytest.mark.parametrize("names", [("full", "full, views swapped", "small"), ("plane", "small", "planes")])
def test_plain(th, cuda, names):
    ctx = th._C.HullContext(0)
    for name in names:
        before = ctx.device_bytes()
        assert same(ctx.visual_hull(*on(cuda, name)), name)
        if name == names[0]:
            once = ctx.device_bytes()
            assert same(ctx.visual_hull(*on(cuda, name)), name) and ctx.device_bytes() == once > before


# ten requests on eight streams: the last two run on the first two's streams and pools, and run again with them
@pytest.mark.parametrize("names", [("full", "plane", *(f"small {i}" for i in range(6)), "small", "full, views swapped"),
                                   ("planes", "small")])
def test_batch(th, cuda, names):
    ctx = th._C.HullContext(0)
    for order in (names, names[::-1]):
        for name, got in zip(order, ctx.visual_hull_batch([on(cuda, name) for name in order])):
            assert same(got, name), name
