"""Frames drawn from the direct lists (cell_lists.cu: one entry per splat and patch of 1, 2 or 4 cells
a side, filtered by the composite) against the same frames drawn from the stable (cell, splat) sort:
the image bit for bit, the (splat, cell) pairs and the list records the composite read. Targets at
the edges of the patch sizes (320 patches, odd cells and tiles), beyond the direct lists' 4096
patches, and splats of many patches (several staging windows, whole-warp walks)."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for


def draw(cloud, frames, w, h, mode):
    r = sk.Renderer(w, h, image_format=sk.FORMAT_RGBA32F)
    r.set_binning(mode)
    r.upload_world(cloud, cloud.sh_degree)
    out = []
    for frame in frames:
        r.draw(frame)
        image = r.read_image(sk.FORMAT_RGBA32F)
        s = r.stats()
        out.append((image, s["draw_count"], s["instances"], s["instances_read"]))
    r.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n,w,h,log_scale", [
    (60_000, 640, 512, -3.0),     # 20 x 16 = 320 cells: the most for single-cell patches
    (60_000, 641, 512, -2.5),     # one column more: patches of 2 x 2 cells
    (80_000, 1279, 1021, -2.0),   # odd cells and tiles, 2 x 2
    (40_000, 1281, 1025, -1.0),   # just above: 4 x 4 patches that hang over the target
    (150_000, 3840, 2160, -2.5),  # 4 x 4, 510 patches
    (300, 8224, 8096, 0.0),       # 65 x 64 patches: both modes sort
    (2_500, 1280, 720, 0.5),      # boxes of hundreds of cells, several windows per warp
    (1, 33, 17, -1.0),
])
def test_direct_frames_equal_the_sorted_frames(cuda_device, n, w, h, log_scale):
    cloud = synthetic.random_cloud(n, seed=17, sh_degree=0, log_scale_mean=log_scale)
    frames = frames_for(cloud, w, h, (11, 52))
    for (ia, va, pa, ra), (ib, vb, pb, rb) in zip(draw(cloud, frames, w, h, "auto"),
                                                  draw(cloud, frames, w, h, "sorted")):
        assert (va, pa, ra) == (vb, pb, rb)
        assert np.array_equal(ia, ib)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [255, 256, 257, 512, 513, 151_552, 151_553, 152_065])
def test_direct_frames_at_the_edges_of_a_blocks_ranks(cuda_device, n):
    """Count and emission blocks of 256 ranks up to 151,552 sources, of 512 above."""
    w, h = 500, 400
    cloud = synthetic.random_cloud(n, seed=23, sh_degree=0, log_scale_mean=-3.5)
    frames = frames_for(cloud, w, h, (11,))
    for (ia, va, pa, ra), (ib, vb, pb, rb) in zip(draw(cloud, frames, w, h, "auto"),
                                                  draw(cloud, frames, w, h, "sorted")):
        assert (va, pa, ra) == (vb, pb, rb)
        assert np.array_equal(ia, ib)


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,log_scale", [(31, -1.0), (1023, -2.0), (1024, 0.5), (1025, -2.5), (20_000, -1.0)])
def test_batches_of_small_targets_equal_the_sorted_frames(cuda_device, n, log_scale, mixed):
    """Single-cell patches of every view (blocks of 1024 ranks, boxes of more than 64 cells, several
    windows), and beside a view of larger patches (the general emission)."""
    sizes = [(640, 480), (33, 17), (512, 640)] + [(1280, 720)] * mixed
    cloud = synthetic.random_cloud(n, seed=29, sh_degree=0, log_scale_mean=log_scale)
    r = sk.Renderer(64, 64)
    r.set_binning("sorted")
    r.upload_world(cloud, 0)
    frames = [frames_for(cloud, w, h, (11 + 9 * i,))[0] for i, (w, h) in enumerate(sizes)]
    with sk.Batch(lanes=1, max_views=4) as batch:
        t = batch.submit([sk.BatchView(r, f, w, h) for f, (w, h) in zip(frames, sizes)])
        images = [batch.read_image(t, i) for i in range(len(sizes))]
        assert batch.stats(t)["device_error"] == 0
    for frame, (w, h), image in zip(frames, sizes, images):
        r.resize(w, h)
        r.draw(frame)
        assert np.array_equal(image, r.read_image(sk.FORMAT_RGBA8))
    r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(8192, 8192), (8224, 8224), (16384, 4160)])
def test_sorted_lists_of_65536_cells_and_more(cuda_device, w, h):
    """Cell ids of more than 16 bits: every pair is in one list, and the lists are those of the cells: a
    splat's list entries form the rows and columns of a box."""
    cloud = synthetic.random_cloud(200, seed=31, sh_degree=0, log_scale_mean=-1.0)
    frame = frames_for(cloud, w, h, (11,))[0]
    with sk.Renderer(w, h) as r:
        r.set_binning("sorted")
        r.upload_world(cloud, 0)
        r.draw(frame)
        ranges, values = r.read_tile_lists()
        order = r.read_order()
        assert r.stats()["instances"] == len(values) == int((ranges[:, 1] - ranges[:, 0]).sum())
    rank = np.empty(int(order.max()) + 1, np.int64)
    rank[order] = np.arange(len(order))
    columns, seen = (w + 31) // 32, {}
    for cell in np.flatnonzero(ranges[:, 1] > ranges[:, 0]):
        entries = values[ranges[cell, 0]:ranges[cell, 1]]
        assert (np.diff(rank[entries]) > 0).all()  # front to back, each splat once
        for v in entries:
            seen.setdefault(int(v), []).append((cell // columns, cell % columns))
    for cells in seen.values():  # convex: every row of a splat's cells is one run, in adjacent rows
        rows = {}
        for y, x in cells:
            rows.setdefault(y, []).append(x)
        assert max(rows) - min(rows) + 1 == len(rows)
        for xs in rows.values():
            assert max(xs) - min(xs) + 1 == len(xs)
