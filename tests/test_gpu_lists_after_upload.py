"""sk_read_tile_lists makes a direct frame's per-cell lists from the spans and the order the frame left
behind. Once a world's upload has put other memory in their place there is nothing to make them from:
the call returns no entries. Where the upload leaves the buffers alone, the lists stay the frame's."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for
from test_gpu_half_failed_uploads import fails_at

pytestmark = pytest.mark.gpu

W, H = 480, 320


def world(n, seed=71):
    return synthetic.random_cloud(n, seed=seed, sh_degree=0, log_scale_mean=-2.0)


def put(r, into, n):
    if into == "world":
        r.upload_world(world(n, 72), 0)
    elif into == "slab":
        r.create_slab(n, 0)
    else:
        r.upload_lod_world(sk.build_lod_tree(world(n, 72)), 0, 4_000_000)


def drawn(r, cloud, mode="auto"):
    """A frame's lists, and the same frame drawn again with its lists not read."""
    r.set_binning(mode)
    r.upload_world(cloud, 0)
    frame = frames_for(cloud, W, H, (11,))[0]
    r.draw(frame)
    lists = r.read_tile_lists()
    r.draw(frame)
    r.wait_idle()
    return lists


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("mode", ["auto", "sorted"])
@pytest.mark.parametrize("into", ["world", "slab", "lod"])
def test_a_larger_world_leaves_no_lists(cuda_device, into, mode):
    with sk.Renderer(W, H) as r:
        assert len(drawn(r, world(20_000), mode)[1]) > 20_000
        put(r, into, 60_000)
        ranges, values = r.read_tile_lists()
        assert len(values) == 0 and not ranges.any()
        # the next frame has its own
        cloud = world(50_000, 73)
        want = drawn(r, cloud, "sorted")[1]
        assert np.array_equal(drawn(r, cloud)[1], want)


@pytest.mark.parametrize("into", ["world", "slab", "lod"])
def test_a_smaller_world_leaves_the_lists(cuda_device, into):
    with sk.Renderer(W, H) as r:
        want = drawn(r, world(60_000))
        put(r, into, 9_000)
        assert same(r.read_tile_lists(), want)


def test_lists_whose_own_buffers_stay_are_kept(cuda_device):
    """Worlds of up to 128 splats share the first list buffers: only the spans move."""
    with sk.Renderer(W, H) as r:
        want = drawn(r, world(60))
        assert len(want[1]) > 0
        r.upload_world(world(120, 72), 0)
        assert same(r.read_tile_lists(), want)


def test_a_larger_target_leaves_the_lists(cuda_device):
    with sk.Renderer(W, H) as r:
        want = drawn(r, world(20_000))[1]
        r.resize(8 * W, 8 * H)
        assert np.array_equal(r.read_tile_lists()[1], want)


@pytest.mark.parametrize("into", ["world", "slab"])
def test_an_upload_that_fails_half_way(cuda_device, into):
    """Whichever allocation fails, the lists are the frame's or none."""
    kept, gone, allocation = 0, 0, 0
    while True:
        with sk.Renderer(W, H) as r:
            want = drawn(r, world(20_000))
            if not fails_at(lambda: put(r, into, 60_000), allocation):
                break
            got = r.read_tile_lists()
            if len(got[1]) == 0:
                assert not got[0].any()
                gone += 1
            else:
                assert same(got, want)
                kept += 1
        allocation += 1
    assert kept > 2 and gone > 5
