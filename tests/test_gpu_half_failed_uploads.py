"""An upload that fails at any of its device allocations keeps the world before it, and that world draws
as before: buffers that had already grown by then are cleared as a frame expects them."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for

pytestmark = pytest.mark.gpu

W, H = 320, 240


def fails_at(call, allocation):
    """Whether the call runs out of memory when its allocation number `allocation` (from 0) fails."""
    sk.testing_fail_device_allocations(1, after=allocation)
    try:
        call()
        return False
    except sk.SplatError as err:
        assert err.status == sk.SK_E_OOM
        return True
    finally:
        sk.testing_fail_device_allocations(0)


@pytest.mark.parametrize("mode", ["auto", "sorted"])
@pytest.mark.parametrize("into", ["world", "slab"])
def test_the_previous_world_draws_as_before(cuda_device, into, mode):
    small = synthetic.random_cloud(40_000, seed=61, sh_degree=0)
    large = synthetic.random_cloud(90_000, seed=62, sh_degree=0)
    frame = frames_for(small, W, H, (5,))[0]
    failed = 0
    while True:  # a context of its own for each allocation that fails: the buffers before it have grown
        with sk.Renderer(W, H) as r:
            r.set_binning(mode)
            r.upload_world(small, 0)
            r.draw(frame)
            want = r.read_image()
            grow = (lambda: r.upload_world(large, 0)) if into == "world" else (lambda: r.create_slab(large.count, 0))
            if not fails_at(grow, failed):
                break
            assert r.world() == (small.count, 0)
            r.draw(frame)
            assert np.array_equal(r.read_image(), want)
            assert r.stats()["device_error"] == 0
        failed += 1
    assert failed > 10  # the world's, then the frame buffers'
