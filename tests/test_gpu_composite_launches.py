"""The composite launched after the emission (all tiles on the chip at once, many records) and chained behind
it: frames and a batch at the edges of both rules, against the same frames from the sorted lists."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for


@pytest.mark.gpu
@pytest.mark.parametrize("w,h", [(17, 9), (592, 512), (593, 512)])  # 2, 1184 and 1216 tiles
@pytest.mark.parametrize("n", [75_776, 75_777, 160_000])
def test_frames_at_the_edges(cuda_device, n, w, h):
    cloud = synthetic.random_cloud(n, seed=43, sh_degree=0, log_scale_mean=-2.5)
    frames, got = frames_for(cloud, w, h, (11, 52, 11)), {}
    for mode in ("auto", "sorted"):
        with sk.Renderer(w, h) as r, sk.Batch(lanes=1, max_views=2) as batch:
            r.set_binning(mode)
            r.upload_world(cloud, 0)
            images = []
            for frame in frames:
                r.draw(frame)
                images.append(r.read_image())
                t = batch.submit([sk.BatchView(r, frame, w, h)])
                assert np.array_equal(batch.read_image(t, 0), images[-1])
            got[mode] = images
    assert all(np.array_equal(a, b) for a, b in zip(got["auto"], got["sorted"]))
    assert np.array_equal(got["auto"][0], got["auto"][2])
