"""A band's launch, a band's copy or a batch view's copy that fails: the call returns the error with nothing
of it left running (the caller's buffers are the caller's again), and what follows is right."""
from __future__ import annotations

import time

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_bands import buffer_for
from test_gpu_cell_lists import frames_for

pytestmark = pytest.mark.gpu

W, H = 3840, 2160  # eight bands


@pytest.fixture(scope="module")
def cloud(cuda_device):
    return synthetic.random_cloud(400_000, seed=95, sh_degree=0, log_scale_mean=-1.0)


def fails(call):
    with pytest.raises(sk.SplatError) as err:
        call()
    assert err.value.status == sk.SK_E_OOM


@pytest.mark.parametrize("band", [0, 2, 7])
def test_a_failed_band(cloud, band):
    a, b = frames_for(cloud, W, H, (11, 52))
    with sk.Renderer(W, H) as r:
        r.upload_world(cloud, 0)
        out = buffer_for(r, W, H, sk.FORMAT_RGBA8)
        want = []
        for frame in (a, b):
            r.draw(frame)
            want.append(r.read_image(out=out).copy())
        # the copy of a band: the rows before it land before the call returns, none after
        r.draw(a)
        out.fill(0)
        sk.testing_fail_image_step(band)
        fails(lambda: r.read_image(out=out))
        left = out.copy()
        time.sleep(0.05)
        assert np.array_equal(out, left)
        assert left.any() == (band > 0)
        assert np.array_equal(r.read_image(out=out), want[0])
        # the launch of a band: the frame after the failed one, on the same stream, is right
        sk.testing_fail_image_step(band)
        fails(lambda: r.draw(a))
        r.draw(b)
        assert np.array_equal(r.read_image(out=out), want[1])
        assert r.stats()["device_error"] == 0 and not r.gpu_failed()


@pytest.mark.parametrize("copy", [0, 2])
def test_a_failed_copy_of_a_served_image(cloud, copy):
    """The requests of the batch complete with an error and nothing writes their images after that."""
    frames = frames_for(cloud, W, H, (11, 52, 40, 80))
    with sk.Renderer(64, 64) as r:
        r.upload_world(cloud, 0)
        server = sk.Server(lanes=1, max_batch_views=4, max_batch_splats=4_000_000)
        scene = server.add_scene(r)
        images = [sk.HostImage(W, H) for _ in frames]
        requests = [sk.Request(scene, f, W, H, i) for f, i in zip(frames, images)]

        def burst():
            for q in requests:
                server.submit(q)
            server.drain()
            return [c["status"] for c in sorted(server.take_completions(), key=lambda c: c["id"])]

        assert burst() == [0] * 4
        want = [i.array.copy() for i in images]
        for i in images:
            i.array.fill(0)
        sk.testing_fail_image_step(copy)
        status = burst()
        assert sk.SK_E_OOM in status and set(status) <= {0, sk.SK_E_OOM}
        left = [i.array.copy() for i in images]
        time.sleep(0.05)
        assert all(np.array_equal(i.array, x) for i, x in zip(images, left))
        assert burst() == [0] * 4
        assert all(np.array_equal(i.array, x) for i, x in zip(images, want))
        server.close()
