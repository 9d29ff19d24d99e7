"""A submission that fails at any of its device allocations leaves its lane drawing as before: buffers that
moved by then are cleared, and no captured graph points at the old ones. Nor does one after the
pinned view table of the lists has moved."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for
from test_gpu_half_failed_uploads import fails_at

pytestmark = pytest.mark.gpu


def view_of(r, cloud, w, h, step=11):
    frame = frames_for(cloud, w, h, (step,))[0]
    if r.lod:
        frame.ranges = []
    return sk.BatchView(r, frame, w, h)


def images_of(batch, views):
    t = batch.submit(views)
    out = [batch.read_image(t, i) for i in range(len(views))]
    assert batch.stats(t)["device_error"] == 0
    return out


@pytest.fixture(scope="module")
def worlds(cuda_device):
    small, large = (synthetic.random_cloud(n, seed=91, sh_degree=0) for n in (40_000, 150_000))
    made = []
    for cloud, lod in ((small, False), (large, False), (small, True)):
        r = sk.Renderer(64, 64)
        if lod:
            r.upload_lod_world(sk.build_lod_tree(cloud), 0, 4_000_000)
        else:
            r.upload_world(cloud, 0)
        r.lod = lod
        made.append((r, cloud))
    yield made
    for r, _ in made:
        r.close()


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("lod", [False, True])
def test_the_lane_draws_as_before(worlds, graphs, lod):
    before = [view_of(*worlds[0], 320, 240), view_of(*worlds[2 if lod else 0], 200, 150)]
    grown = [view_of(*worlds[1], 1280, 720), view_of(*worlds[2 if lod else 1], 640, 480)] * 3
    allocation = 0
    while True:
        with sk.Batch(lanes=1, max_views=8, use_graphs=graphs) as batch:
            want = images_of(batch, before)
            if not fails_at(lambda: batch.submit(grown), allocation):
                break
            for _ in range(2):
                assert all(np.array_equal(a, b) for a, b in zip(images_of(batch, before), want))
        allocation += 1
    assert allocation > 12


def test_a_graph_after_the_view_table_has_moved(worlds):
    one = [view_of(*worlds[0], 320, 240)]
    four = [view_of(*worlds[2], 200, 150, step) for step in (3, 9, 20, 31)]  # LOD views: not captured
    with sk.Batch(lanes=1, max_views=8, use_graphs=True) as batch:
        batch.set_tuning(1, 4096, 1, 1)
        images_of(batch, four)  # the lane knows four views, its lists' table does not
        batch.set_tuning(1, 4096, 1, 0)
        want = images_of(batch, one)
        images_of(batch, four)
        assert np.array_equal(images_of(batch, one)[0], want[0])
