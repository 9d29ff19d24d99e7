"""The entries the direct lists' kernels write (per patch: projected index and cell bits, in depth order),
filtered by cell on the host, against the lists the stable (cell, splat) sort gives for the same frame.
sk_read_tile_lists makes its answer by that sort for a direct frame too, and an image does not show
what lies behind early termination; these do."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for

pytestmark = pytest.mark.gpu


def cell_lists(lists, w, h):
    """The patch lists as (ranges, values) per cell."""
    shift, patches_x, ranges, values, masks = lists
    cells_x, cells_y, edge = (w + 31) // 32, (h + 31) // 32, 1 << shift
    out, starts, at = [], np.zeros((cells_x * cells_y, 2), np.uint32), 0
    for cell in range(cells_x * cells_y):
        x, y = cell % cells_x, cell // cells_x
        a, b = ranges[(y >> shift) * patches_x + (x >> shift)]
        bit = (y % edge) * edge + x % edge
        own = values[a:b][(masks[a:b] >> bit) & 1 == 1]
        out.append(own)
        starts[cell] = at, at + len(own)
        at += len(own)
    return starts, np.concatenate(out)


@pytest.mark.parametrize("n,w,h,log_scale,shift", [
    (30_000, 640, 480, -2.5, 0),
    (2_000, 640, 512, 0.5, 0),       # 320 patches; boxes of more than 64 cells, several windows
    (60_000, 641, 512, -2.5, 1),
    (1_500, 1279, 1021, 0.5, 1),     # patches that hang over the target, several windows
    (80_000, 1920, 1080, -2.5, 2),
    (3_000, 1920, 1080, 0.7, 2),     # boxes of hundreds of cells
    (200_000, 3840, 2160, -2.0, 2),  # more than 151,552 sources: blocks of 512 ranks
    (160_000, 400, 300, -3.0, 0),
    (160_000, 640, 480, -3.0, 1),    # larger patches from 145 cells, and from 81 patches of 2 x 2, up
    (151_553, 384, 384, -2.5, 0),    # 144 cells
    (151_553, 385, 384, -2.0, 1),
    (151_553, 640, 512, -1.0, 1),    # 80 patches; several windows
    (151_553, 641, 512, -2.5, 2),
    (1, 33, 17, -1.0, 0),
])
def test_patch_lists_hold_the_cells_lists(cuda_device, n, w, h, log_scale, shift):
    cloud = synthetic.random_cloud(n, seed=37, sh_degree=0, log_scale_mean=log_scale)
    with sk.Renderer(w, h) as r:
        r.upload_world(cloud, 0)
        for frame in frames_for(cloud, w, h, (11, 52)):
            r.draw(frame)
            r.wait_idle()
            lists = r.testing_read_patch_lists()
            assert lists[0] == shift
            assert lists[2][0, 0] == 0 and np.array_equal(lists[2][1:, 0], lists[2][:-1, 1])  # back to back
            assert lists[2][-1, 1] == len(lists[3])
            ranges, values = cell_lists(lists, w, h)
            want_ranges, want_values = r.read_tile_lists()
            assert len(want_values) == r.stats()["instances"]
            assert np.array_equal(ranges, want_ranges) and np.array_equal(values, want_values)


@pytest.mark.parametrize("n,w,h,log_scale", [(60_000, 500, 400, -2.0), (60_000, 1000, 700, -2.0), (60_000, 1920, 1080, -1.5)])
def test_images_without_early_termination(cuda_device, n, w, h, log_scale):
    cloud = synthetic.random_cloud(n, seed=38, sh_degree=0, log_scale_mean=log_scale)
    frame, got = frames_for(cloud, w, h, (11,))[0], []
    for mode in ("auto", "sorted"):
        with sk.Renderer(w, h, image_format=sk.FORMAT_RGBA32F) as r:
            r.apply_render_policy(sk.Policy(enable_early_termination=False))
            r.set_binning(mode)
            r.upload_world(cloud, 0)
            r.draw(frame)
            image, s = r.read_image(sk.FORMAT_RGBA32F), r.stats()
            got.append((image, s["instances"], s["instances_read"], s["fragments"]))
    assert got[0][1:] == got[1][1:]
    assert got[0][2] >= got[0][1]  # every pair was read, by each of its cell's tiles
    assert np.array_equal(got[0][0], got[1][0])


@pytest.mark.parametrize("sizes", [[(640, 480), (33, 17), (512, 640)],  # single cells
                                   [(640, 480), (1280, 720), (33, 17), (3840, 2160)]])  # beside larger patches
@pytest.mark.parametrize("n,log_scale", [(1_025, 0.5), (40_000, -2.0)])
def test_batches_without_early_termination(cuda_device, n, log_scale, sizes):
    cloud = synthetic.random_cloud(n, seed=39, sh_degree=0, log_scale_mean=log_scale)
    with sk.Renderer(64, 64) as r, sk.Batch(lanes=1, max_views=4) as batch:
        r.upload_world(cloud, 0)
        batch.apply_render_policy(sk.Policy(enable_early_termination=False))
        views = [sk.BatchView(r, frames_for(cloud, w, h, (11 + 9 * i,))[0], w, h) for i, (w, h) in enumerate(sizes)]
        got = []
        for sorted_lists in (0, 1):
            batch.set_tuning(1, 4096, 1, sorted_lists)
            t = batch.submit(views)
            got.append(([batch.read_image(t, i) for i in range(len(views))], batch.stats(t)))
    for key in ("instances", "fragments", "visible"):
        assert got[0][1][key] == got[1][1][key]
    assert all(np.array_equal(a, b) for a, b in zip(got[0][0], got[1][0]))
