"""The calls whose speed this project looks after, through its public entry points.

The cases run from the smallest request, where launches and latency count, to
the largest one the server meets, over the mask types, camera conventions and
output forms that users combine, and over the public blur and marching cubes.
Hull inputs are the seeded scenes of ``torchhull_gb300.scenes``: unions of
ellipsoids (and thin capsules where the masks are partial) seen by cameras
around them.  Volumes are the sphere distance fields of torchhull's own
marching-cubes benchmark, with the centre and the radius drawn from the seed.

Meshes and fields go into buffers of a fixed size that the caller keeps (a
renderer's vertex and index buffers): how many vertices come depends on the
scene.  The rest of a buffer stays zero.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import torchhull_gb300 as th
from torchhull_gb300 import scenes

DEVICE = "cuda:0"
CORNER, LENGTH = (-1.0, -1.0, -1.0), 2.0
ELEMENT = {"uint8": 1, "float16": 2, "float32": 4, "float64": 8}


def _hull(views, height, width, level, partial=False, convention="opengl", dtype="float32", unique=True, kind="hull",
          blur=0):
    # capsules are slow to render: large partial scenes have fewer of them
    capsules = 0 if not partial else 20 if views * height * width <= 1 << 25 else 4
    return {"kind": kind, "views": views, "height": height, "width": width, "level": level, "partial": partial,
            "convention": convention, "dtype": dtype, "unique": unique, "blur": blur,
            "ellipsoids": 8 if partial else 3, "capsules": capsules}


def _blur(views, height, width, dtype, kernel, sparse):
    return {"kind": "blur", "views": views, "height": height, "width": width, "dtype": dtype, "kernel": kernel,
            "sparse": sparse}


def _mc(depth, height, width, dtype, sparse, local, unique=True):
    return {"kind": "mc", "depth": depth, "height": height, "width": width, "dtype": dtype, "sparse": sparse,
            "local": local, "unique": unique}


def listed():
    return [
        # a preview while someone moves a camera: launches and latency are all there is
        dict(_hull(6, 128, 128, 5), name="hull 6x128 l5"),
        # torchhull's small benchmark scene, an interactive reconstruction
        dict(_hull(8, 256, 256, 6), name="hull 8x256 l6"),
        # masks of a segmentation network: bytes, odd image sizes, a plain triangle soup
        dict(_hull(13, 437, 611, 7, True, "opencv", "uint8", False), name="soup 13x437x611 l7"),
        # torchhull's blur benchmark: silhouettes smoothed first, then carved (the masks are no longer 0/1)
        dict(_hull(24, 512, 512, 8, False, "opencv", blur=9), name="blurred hull 24x512 l8"),
        # the field itself, for a renderer or a solver that goes on from the sparse tensor
        dict(_hull(16, 640, 480, 8, False, "opengl", "float16", kind="field"), name="field 16x640x480 l8"),
        # the headline scene: a capture stage whose cameras stand close to the object
        dict(_hull(32, 1024, 1024, 9, True), name="hull 32x1024 l9"),
        # the large request of the served mix
        dict(_hull(64, 2048, 2048, 10), name="hull 64x2048 l10"),
        # what a batch worker hands over at once: requests of mixed size and mode
        {"kind": "batch", "count": 16, "mix": 4, "name": "batch of 16"},
        # smoothing the masks of a capture stage, the usual sparse form
        dict(_blur(32, 1024, 1024, "float32", 9, True), name="sparse blur 32x1024 k9"),
        # every pixel smoothed, in half, at an odd size and with a wider kernel
        dict(_blur(24, 501, 723, "float16", 13, False), name="dense blur 24x501x723 k13"),
        # a distance field from elsewhere turned into a mesh
        dict(_mc(400, 400, 400, "float32", False, False), name="mesh of 400^3"),
        # the same from a narrow band, as a coalesced COO tensor
        dict(_mc(400, 400, 400, "float32", True, True), name="mesh of a 400^3 band"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["hull", "hull", "hull", "hull", "field", "batch", "blur", "mc"])
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(2, 20), "mix": rng.randrange(1 << 20)}
    if kind == "mc":
        side = _log_int(rng, 24, 400)
        sizes = [max(16, int(side * rng.uniform(0.7, 1.0))) for _ in range(3)]
        return _mc(*sizes, rng.choice(["float16", "float32", "float32", "float64"]), rng.random() < 0.4,
                   rng.random() < 0.5, rng.random() < 0.8)
    height = _log_int(rng, 64, 1536)
    width = max(64, int(height * rng.uniform(0.8, 1.4)))
    views = _log_int(rng, 3, 48)
    if kind == "blur":
        return _blur(views, height, width, rng.choice(["uint8", "float16", "float32", "float32", "float64"]),
                     rng.choice([3, 5, 9, 9, 13, 17]), rng.random() < 0.7)
    partial = rng.random() < 0.3
    blurred = kind == "hull" and rng.random() < 0.25
    dtype = rng.choice(["float16", "float32"]) if blurred else rng.choice(["uint8", "float16", "float32", "float32"])
    return _hull(views, height, width, rng.randint(4, 9), partial, rng.choice(["opengl", "opencv"]), dtype,
                 rng.random() < 0.8, kind, rng.choice([5, 9]) if blurred else 0)


def _batch_shapes(case):
    """The requests of a batch: the mixed distribution of ``scenes.batched_requests``."""
    rng = np.random.default_rng(case["mix"])
    return [(int(rng.integers(4, 49)), int(rng.choice([256, 512, 768, 1024])), int(rng.integers(6, 10)),
             bool(rng.random() < 0.3)) for _ in range(case["count"])]


def _masks(seed, views, height, width, ellipsoids, capsules, partial, convention, dtype):
    scene = scenes.make_scene(seed, ellipsoids, capsules)
    cams = scenes.make_cameras(seed, views, 1.4 if partial else 2.5, 50.0 if partial else 40.0, height, width, convention)
    masks = scenes.render_masks(scene, cams, device=DEVICE, dtype=getattr(torch, dtype))
    return masks, torch.as_tensor(cams.transforms, dtype=torch.float32).to(DEVICE)


def _volume(case, seed):
    """Signed distance to a sphere, in voxels: radius 0.87 of the half extent, both a little off."""
    rng = np.random.default_rng(seed)
    sizes = [case["depth"], case["height"], case["width"]]
    radius = 0.8731945 * min(sizes) / 2 * rng.uniform(0.95, 1.0)
    square = torch.zeros((1, 1, 1), dtype=torch.float64, device=DEVICE)
    for axis, size in enumerate(sizes):
        at = torch.arange(size, dtype=torch.float64, device=DEVICE) - ((size - 1) / 2 + rng.uniform(-1, 1))
        square = square + (at * at).reshape([-1 if a == axis else 1 for a in range(3)])
    return (square.sqrt() - radius).to(getattr(torch, case["dtype"]))[None]


def _band(volume):
    """The entries within two voxels of the surface."""
    index = (volume.abs() <= 2).nonzero().T.contiguous()
    return index, volume[tuple(index)]


def _room(level, partial):
    """Vertices of a level's mesh that there is room for: about three times what these scenes have (1.1 per cell of one
    face of the cube, 12 where frames cut the object and capsules are part of it)."""
    return (40 if partial else 3) * 4**level + 1024


def _mc_verts(case, radius):
    """Lattice edges that a sphere of that radius crosses: its silhouette's area twice per axis."""
    return int(6 * math.pi * (radius * min(case["depth"], case["height"], case["width"]) / 2) ** 2)


def _mc_room(case):
    return _mc_verts(case, 0.9) + 1024


def _mesh_buffers(verts, unique):
    faces = 2 * verts
    return (torch.zeros((verts if unique else 3 * faces, 3), dtype=torch.float32, device=DEVICE),
            torch.zeros((faces, 3), dtype=torch.int64, device=DEVICE))


def _keep(buffer, made):
    n = min(len(buffer), len(made))
    buffer[:n].copy_(made[:n])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        requests, buffers = [], []
        for i, (views, side, level, partial) in enumerate(_batch_shapes(case)):
            r = scenes.make_request(1000 * seed + i, views, side, level, partial, n_capsules=4 if partial else 0, device=DEVICE)
            requests.append((r.masks, r.transforms, r.level, r.cube_corner_bfl, r.cube_length, r.masks_partial,
                             r.transforms_convention, r.unique_verts))
            buffers.append(_mesh_buffers(_room(level, partial), True))
        return {"kind": kind, "requests": requests, "buffers": buffers}
    if kind == "mc":
        volume = _volume(case, seed)
        if case["sparse"]:
            index, values = _band(volume)
            volume = torch.sparse_coo_tensor(index, values, volume.shape).coalesce()
        return {"kind": kind, "volume": volume, "local": case["local"], "unique": case["unique"],
                "buffers": _mesh_buffers(_mc_room(case), case["unique"])}
    if kind == "blur":
        masks, _ = _masks(seed, case["views"], case["height"], case["width"], 3, 0, False, "opengl", case["dtype"])
        return {"kind": kind, "masks": masks, "kernel": case["kernel"], "sparse": case["sparse"],
                "dtype": torch.float32 if case["dtype"] == "uint8" else None}
    masks, transforms = _masks(seed, case["views"], case["height"], case["width"], case["ellipsoids"], case["capsules"],
                               case["partial"], case["convention"], case["dtype"])
    args = (case["level"], CORNER, LENGTH, case["partial"], case["convention"])
    if kind == "field":
        points = 3 * _room(case["level"], case["partial"])
        buffers = (torch.zeros((4, points), dtype=torch.int64, device=DEVICE),
                   torch.zeros(points, dtype=torch.float32, device=DEVICE))
    else:
        buffers = _mesh_buffers(_room(case["level"], case["partial"]), case["unique"])
    return {"kind": kind, "masks": masks, "transforms": transforms, "args": args, "unique": case["unique"],
            "blur": case["blur"], "buffers": buffers}


def run(state):
    kind = state["kind"]
    if kind == "blur":
        return th.gaussian_blur(state["masks"], state["kernel"], 2.0, state["sparse"], state["dtype"])
    buffers = state["buffers"]
    if kind == "batch":
        for (verts, faces), kept in zip(th._C.visual_hull_batch(state["requests"]), buffers):
            _keep(kept[0], verts)
            _keep(kept[1], faces)
        return buffers
    if kind == "mc":
        made = th.marching_cubes(state["volume"], 0.0, state["local"], state["unique"])
    elif kind == "field":
        field = th.sparse_visual_hull_field(state["masks"], state["transforms"], *state["args"])
        n = min(field.values().numel(), len(buffers[1]))
        buffers[0][:, :n].copy_(field.indices()[:, :n])
        buffers[1][:n].copy_(field.values()[:n])
        return buffers
    else:
        masks = state["masks"]
        if state["blur"]:
            masks = th.gaussian_blur(masks, state["blur"], 2.0)
        made = th.visual_hull(masks, state["transforms"], *state["args"], state["unique"])
    _keep(buffers[0], made[0])
    _keep(buffers[1], made[1])
    return buffers


def _mesh_bytes(verts, unique):
    """A closed mesh of that many vertices has twice as many triangles of three int64 indices; the soup has three
    vertices of its own for each."""
    return 2 * verts * 24 + (verts if unique else 6 * verts) * 12


def _hull_bytes(views, height, width, element, level, partial, unique=True):
    return views * (height * width * element + 64) + _mesh_bytes((12 if partial else 1.1) * 4**level, unique)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        return {"bytes": sum(_hull_bytes(v, s, s, 4, level, p) for v, s, level, p in _batch_shapes(case)), "flops": 0}
    if kind == "mc":
        points, verts = case["depth"] * case["height"] * case["width"], _mc_verts(case, 0.85)
        if case["sparse"]:
            points = 4 * verts * 2 / 3  # the band is four voxels thick: 4 pi r^2 of each
        entry = ELEMENT[case["dtype"]] + (32 if case["sparse"] else 0)
        return {"bytes": points * entry + _mesh_bytes(verts, case["unique"]), "flops": 0}
    pixels, size = case["views"] * case["height"] * case["width"], ELEMENT[case["dtype"]]
    if kind == "blur":
        out = 4 if case["dtype"] == "uint8" else size
        # the boundary tiles are a few percent of the pixels
        return {"bytes": pixels * (size + out), "flops": 2 * case["kernel"] ** 2 * pixels * (0.03 if case["sparse"] else 1)}
    if kind == "field":
        # about 3 (30) lattice points per cell of one face of the cube, with four indices and a value each
        return {"bytes": pixels * size + 64 * case["views"] + 36 * (30 if case["partial"] else 3) * 4 ** case["level"],
                "flops": 0}
    return {"bytes": _hull_bytes(case["views"], case["height"], case["width"], size, case["level"], case["partial"],
                                 case["unique"]), "flops": 0}


def _exact_blur(case, seed):
    state = prepare(case, seed)
    kernel, r = case["kernel"], case["kernel"] // 2
    images = state["masks"][..., 0].double()
    height, width = images.shape[1:]
    padded = torch.nn.functional.pad(images[:, None], (r, r, r, r), mode="reflect")[:, 0]
    blurred = torch.zeros_like(images)
    total = 0.0
    for i in range(kernel):
        for j in range(kernel):
            weight = math.exp(-((i - r) ** 2 + (j - r) ** 2) / (2 * 2.0**2))
            total += weight
            blurred.add_(padded[:, i : i + height, j : j + width], alpha=weight)
    blurred /= total
    if case["sparse"]:
        # only the tiles of r x r pixels next to one that holds an edge are smoothed
        edge = torch.zeros_like(images, dtype=torch.bool)
        edge[:, :, :-1] |= images[:, :, :-1] != images[:, :, 1:]
        edge[:, :-1] |= images[:, :-1] != images[:, 1:]
        up = (height // r + 1) * r - height, (width // r + 1) * r - width
        tiles = torch.nn.functional.pad(edge[:, None].float(), (0, up[1], 0, up[0]))
        tiles = torch.nn.functional.max_pool2d(tiles, r)
        tiles = torch.nn.functional.max_pool2d(tiles, 3, stride=1, padding=1)
        near = tiles[:, 0].repeat_interleave(r, 1).repeat_interleave(r, 2)[:, :height, :width] > 0
        blurred = torch.where(near, blurred, images)
    return blurred[..., None]


def _exact_vertices(case, seed):
    """Vertices of the unique mesh, by their edge's lower end point, then by axis."""
    volume = _volume(case, seed)
    if case["sparse"]:
        index, values = _band(volume)
        held = torch.zeros(volume.shape, dtype=torch.bool, device=DEVICE)
        held[tuple(index)] = True
        held = held[0]
    volume = volume[0]
    below = volume < 0.0
    sizes = volume.shape
    crossed = torch.zeros((*sizes, 3), dtype=torch.bool, device=DEVICE)  # x, y, z edges
    cells = None
    if case["sparse"]:
        # an edge counts only where a cell with all its eight corners holds it
        cells = held.clone()
        for axis in range(3):
            moved = torch.zeros_like(cells)
            n = sizes[axis] - 1
            moved.narrow(axis, 0, n).copy_(cells.narrow(axis, 1, n))
            cells &= moved
    for axis in range(3):
        along, n = 2 - axis, sizes[2 - axis] - 1
        change = below.narrow(along, 0, n) != below.narrow(along, 1, n)
        if cells is not None:
            use = cells.clone()
            for other in (0, 1, 2):
                if other != along:
                    m = sizes[other] - 1
                    shifted = use.clone()
                    shifted.narrow(other, 1, m).logical_or_(use.narrow(other, 0, m))
                    use = shifted
            change = change & use.narrow(along, 0, n)
        crossed[..., axis].narrow(along, 0, n).copy_(change)
    z, y, x, axis = crossed.nonzero(as_tuple=True)
    lower = torch.stack([x, y, z], 1)
    step = torch.nn.functional.one_hot(axis, 3)
    upper = lower + step
    v1 = volume[z, y, x].double()
    v2 = volume[upper[:, 2], upper[:, 1], upper[:, 0]].double()
    t = -v1 / (v2 - v1)
    t = torch.where((v1 - v2).abs() < 1e-5, torch.zeros_like(t), t)
    t = torch.where(v2.abs() < 1e-5, torch.ones_like(t), t)
    t = torch.where(v1.abs() < 1e-5, torch.zeros_like(t), t)
    verts = lower.double() + t[:, None] * step
    if case["local"]:
        verts = verts * 2 / (torch.tensor([case["width"], case["height"], case["depth"]], device=DEVICE).double() - 1) - 1
    kept = torch.zeros((_mc_room(case), 3), dtype=torch.float64, device=DEVICE)
    _keep(kept, verts)
    return kept


def exact(case, seed):
    if case["kind"] == "blur":
        return _exact_blur(case, seed)
    if case["kind"] == "mc" and case["unique"]:
        return [_exact_vertices(case, seed), None]
    # a hull's octree, its lattice and its mesh follow from 32-bit decisions: in 64 bits it is another set of cells
    return None
