"""Which frames are drawn in bands: a context's first and those after a read into pinned memory, whose rows are
copied band by band. Into pageable memory an image of fewer than 5 million pixels goes in one copy, and the
frame after it is drawn in one launch (no step of theirs meets the hook that makes a band's launch or copy
fail). The images are the same bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_bands import buffer_for, captured
from test_gpu_cell_lists import frames_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,fmt,mode", [
    (1023, 592, sk.FORMAT_RGBA8, "auto"),     # two bands
    (1280, 720, sk.FORMAT_RGBA8, "auto"),
    (1919, 1081, sk.FORMAT_RGBA32F, "auto"),  # six, ragged
    (1920, 1080, sk.FORMAT_RGBA8, "sorted"),
    (2559, 1441, sk.FORMAT_RGBA8, "auto"),    # eight
])
def test_bands_by_the_memory_read_into(cuda_device, w, h, fmt, mode):
    cloud = synthetic.random_cloud(40_000, seed=45, sh_degree=0, log_scale_mean=-2.0)
    a, b = frames_for(cloud, w, h, (11, 52))
    with sk.Renderer(w, h, image_format=fmt) as r:
        r.set_binning(mode)
        r.upload_world(cloud, 0)
        out = buffer_for(r, w, h, fmt)
        want = [captured(r, f, out) for f in (a, b)]
    with sk.Renderer(w, h, image_format=fmt) as r:
        r.set_binning(mode)
        r.upload_world(cloud, 0)

        def same(frame, into):
            into.fill(0)
            r.draw(frame)
            assert np.array_equal(r.read_image(fmt, out=into), want[0 if frame is a else 1])

        try:
            r.draw(a)  # in bands, but read into pageable memory
            sk.testing_fail_image_step(0)
            assert np.array_equal(r.read_image(fmt, out=np.zeros_like(out)), want[0])
            same(b, np.zeros_like(out))
            same(a, out)  # drawn in one launch, read into pinned memory: the next one is drawn in bands
            with pytest.raises(sk.SplatError) as err:
                r.draw(b)
            assert err.value.status == sk.SK_E_OOM
            same(b, out)
            r.draw(a)
            sk.testing_fail_image_step(0)
            assert np.array_equal(r.read_image(fmt, out=np.zeros_like(out)), want[0])
            same(b, np.zeros_like(out))
        finally:
            sk.testing_fail_image_step(0xFFFFFFFF)  # none
        same(b, out)
        same(a, out)
        same(b, out)
        assert r.stats()["device_error"] == 0 and not r.gpu_failed()


def test_very_large_images_go_in_bands_into_any_memory(cuda_device):
    w, h = 2500, 2000
    cloud = synthetic.random_cloud(40_000, seed=46, sh_degree=0, log_scale_mean=-2.0)
    a, b = frames_for(cloud, w, h, (11, 52))
    with sk.Renderer(w, h) as r:
        r.upload_world(cloud, 0)
        out = buffer_for(r, w, h, sk.FORMAT_RGBA8)
        want = [captured(r, f, out) for f in (a, b)]
        for frame, image in ((a, want[0]), (b, want[1])):
            r.draw(frame)
            assert np.array_equal(r.read_image(), image)
        sk.testing_fail_image_step(0)
        with pytest.raises(sk.SplatError):
            r.draw(a)
