"""Frames drawn in bands (several composite launches, each band's rows copied to the host while the next are
drawn) against the same frames in one launch (captured ones), bit for bit: sizes around the bands' edges,
ragged last rows, both pixel formats, sorted lists, LOD cuts, a frame whose lists overflow and is drawn again,
and frames that are not read at once."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from scenes import lod_camera
from test_gpu_cell_lists import frames_for
from test_gpu_lod_one_launch import fan_tree


def banded(r, frame, fmt):
    r.draw(frame)
    return r.read_image(fmt)


def captured(r, frame, out):
    ticket = r.capture_next_frame(out)
    r.draw(frame)
    return np.array(r.wait_capture(ticket))


def buffer_for(r, w, h, fmt):
    import torch
    dtype = torch.float32 if fmt == sk.FORMAT_RGBA32F else torch.uint8
    return torch.zeros((h, w, 4), dtype=dtype, pin_memory=True).numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,fmt,mode", [
    (1023, 592, sk.FORMAT_RGBA8, "auto"),     # 64 x 37 = 2368 tiles: two bands
    (1008, 592, sk.FORMAT_RGBA8, "auto"),     # 63 x 37: one launch
    (1280, 720, sk.FORMAT_RGBA8, "auto"),     # three bands
    (1919, 1081, sk.FORMAT_RGBA32F, "auto"),  # six, ragged
    (1920, 1080, sk.FORMAT_RGBA8, "sorted"),
    (3839, 2161, sk.FORMAT_RGBA8, "auto"),    # eight
    (8192, 40, sk.FORMAT_RGBA8, "auto"),      # one band of three rows of tiles
    (40, 8192, sk.FORMAT_RGBA8, "auto"),
])
def test_bands_equal_one_launch(cuda_device, w, h, fmt, mode):
    cloud = synthetic.random_cloud(40_000, seed=41, sh_degree=0, log_scale_mean=-2.0)
    frames = frames_for(cloud, w, h, (11, 52))
    with sk.Renderer(w, h, image_format=fmt) as r:
        r.set_binning(mode)
        r.upload_world(cloud, 0)
        got = [banded(r, f, fmt) for f in frames]
        out = buffer_for(r, w, h, fmt)
        want = [captured(r, f, out) for f in frames]
        again = banded(r, frames[0], fmt)  # after captures: two images
        r.draw(frames[1])                  # drawn, waited for, read later
        r.wait_idle()
        late = r.read_image(fmt)
        r.draw(frames[0])
        r.draw(frames[1])                  # two in flight, the newest read
        second = r.read_image(fmt)
    for a, b in zip(got + [again, late, second], want + [want[0], want[1], want[1]]):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_bands_of_a_frame_drawn_again(cuda_device):
    """Splats of many patches overflow the first guess of the lists' size."""
    w, h = 1920, 1080
    cloud = synthetic.random_cloud(6_000, seed=43, sh_degree=0, log_scale_mean=0.5)
    frame = frames_for(cloud, w, h, (11,))[0]
    with sk.Renderer(w, h) as r:
        r.set_binning("sorted")
        r.upload_world(cloud, 0)
        first = banded(r, frame, sk.FORMAT_RGBA8)
        assert r.stats()["instances"] > 8 * cloud.count  # more than the guess
        second = banded(r, frame, sk.FORMAT_RGBA8)
        want = captured(r, frame, buffer_for(r, w, h, sk.FORMAT_RGBA8))
    assert np.array_equal(first, want) and np.array_equal(second, want)


@pytest.mark.gpu
def test_bands_of_a_lod_frame(cuda_device):
    w, h = 1920, 1080
    tree = fan_tree(8, 4)
    view, proj, pos = lod_camera(0.0)
    images = []
    for capture in (False, True):  # fresh worlds: the threshold adapts from frame to frame
        with sk.Renderer(w, h) as r:
            r.upload_lod_world(tree, 0, 100_000)
            frame = sk.Frame(view, proj, pos, [], 0)
            out = buffer_for(r, w, h, sk.FORMAT_RGBA8)
            images.append([captured(r, frame, out) if capture else banded(r, frame, sk.FORMAT_RGBA8)
                           for _ in range(2)])
    for a, b in zip(*images):
        assert np.array_equal(a, b)
    assert images[0][0].any()
