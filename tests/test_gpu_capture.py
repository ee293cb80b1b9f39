"""Blurs and integral images recorded into a CUDA graph keep their own scratch."""

from __future__ import annotations

import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def images(seed, b, h, w, cuda):
    g = torch.Generator().manual_seed(seed)
    return (torch.rand((b, h, w, 1), generator=g) < 0.5).float().to(cuda)


CALLS = {
    "sparse blur": lambda th, m: th.gaussian_blur(m, 9, 2.0),
    "dense blur": lambda th, m: th.gaussian_blur(m, 9, 2.0, sparse=False),
    "integral image": lambda th, m: th.integral_image(m),
}


def record(call):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    return graph, out


@pytest.mark.parametrize("name", list(CALLS))
@pytest.mark.parametrize("shape", [(3, 70, 90), (2, 300, 5000)])  # the second is wider than 4096
def test_replays_beside_larger_calls(th, cuda, name, shape):
    call = CALLS[name]
    m = images(1, *shape, cuda)
    call(th, m)
    torch.cuda.synchronize()
    graph, out = record(lambda: call(th, m))
    # larger calls outside the graph: the context's buffer grows, and its contents change
    other = images(2, 4 * shape[0], 2 * shape[1], shape[2], cuda)
    want_other = call(th, other)
    m.copy_(images(3, *shape, cuda))
    want = call(th, m)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    for _ in range(6):
        graph.replay()
        with torch.cuda.stream(side):
            got.append(call(th, other))
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert all(torch.equal(o, want_other) for o in got)


@pytest.mark.parametrize("name", list(CALLS))
def test_first_call_in_a_graph(th, cuda, name):
    """Without a call before it, and larger than all before: recorded as any other."""
    call = CALLS[name]
    m = images(4, 9, 400, 900, cuda)
    torch.cuda.synchronize()
    graph, out = record(lambda: call(th, m))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, call(th, m))


def test_scratch_of_dropped_graphs_is_reused(th, cuda):
    m = images(5, 3, 200, 300, cuda)
    th.gaussian_blur(m, 9, 2.0)
    torch.cuda.synchronize()
    sizes = []
    for _ in range(6):
        graph, out = record(lambda: th.gaussian_blur(m, 9, 2.0))
        graph.replay()
        torch.cuda.synchronize()
        sizes.append(th._C.device_pool_bytes(0))
        del graph, out
        time.sleep(0.3)  # a graph's objects are destroyed on a thread of the driver
    assert sizes[-1] == sizes[1]
