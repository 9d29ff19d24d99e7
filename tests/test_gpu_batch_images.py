"""Submissions whose images are composited by several launches (each launch's views copied to the host
while the next ones are drawn) against the plain frames, bit for bit: direct and sorted lists, replayed
graphs, two lanes in flight, and server requests with pageable and with no image buffers."""
from __future__ import annotations

import math

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import camera as skcam
from splatkit_b200 import synthetic

SIZES = [(1920, 1080), (333, 97), (2048, 1040), (64, 64), (1919, 1081), (640, 480), (2560, 1440)]


@pytest.fixture(scope="module")
def world(cuda_device):
    cloud = synthetic.random_cloud(30_000, seed=71, sh_degree=1)
    r = sk.Renderer(64, 64)
    r.upload_world(cloud, 1)
    yield r, cloud
    r.close()


def frame_of(cloud, i, w, h):
    view, eye = skcam.orbit_view(7 * i + 2, radius=15.0)
    return sk.Frame(view, skcam.perspective(math.radians(60.0), w / h, 0.05, 200.0), eye, [(0, cloud.count)], 1)


def plain(r, frame, w, h):
    r.resize(w, h)
    r.draw(frame)
    return r.read_image(sk.FORMAT_RGBA8)


@pytest.mark.gpu
@pytest.mark.parametrize("graphs,sorted_lists", [(False, 0), (True, 0), (False, 1)])
def test_images_of_several_composite_launches(world, graphs, sorted_lists):
    r, cloud = world
    views = [[sk.BatchView(r, frame_of(cloud, i + 10 * k, w, h), w, h) for i, (w, h) in enumerate(SIZES)]
             for k in range(3)]
    with sk.Batch(lanes=2, max_views=8, use_graphs=graphs) as batch:
        batch.set_tuning(1, 4096, 2, sorted_lists)
        tickets = [batch.submit(v) for v in views[:2]]
        images = [[batch.read_image(t, i) for i in range(len(SIZES))] for t in tickets]
        t = batch.submit(views[2])  # a lane's second submission (a replayed graph)
        images.append([batch.read_image(t, i) for i in range(len(SIZES))])
        assert batch.stats(t)["device_error"] == 0
    for v, got in zip(views, images):
        for view, image in zip(v, got):
            assert np.array_equal(image, plain(r, view.frame, view.width, view.height))


class Pageable:
    def __init__(self, w, h):
        self.array = np.zeros((h, w, 4), np.uint8)
        self.ptr = self.array.ctypes.data


@pytest.mark.gpu
def test_served_images_land_in_any_buffer(world):
    r, cloud = world
    with sk.Server(lanes=1, max_batch_views=16, max_batch_splats=4_000_000) as server:
        server.add_scene(r)
        requests = []
        for i in range(12):
            w, h = SIZES[i % len(SIZES)]
            image = None if i % 4 == 3 else (Pageable(w, h) if i % 4 == 1 else sk.HostImage(w, h))
            requests.append(sk.Request(0, frame_of(cloud, i, w, h), w, h, image))
        for q in requests:
            server.submit(q)
        server.drain()
        assert all(c["status"] == 0 for c in server.take_completions())
    for q in requests:
        if q.image is not None:
            assert np.array_equal(q.image.array, plain(r, q.frame, q.width, q.height))
