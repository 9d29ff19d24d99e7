"""The cull at the edges of its tiles (256 splats; beyond 592 tiles a block takes several), against the
oracle: survivors, keys and records bit for bit, for record counts around a tile and around 592 of
them, opacities over the whole 8-bit range, merged opacities above 1 and colours that saturate binary16."""
from __future__ import annotations

import math

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import camera as skcam
from splatkit_b200 import synthetic

W, H = 640, 360


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree", [(1, 3), (255, 0), (256, 1), (257, 2), (4 * 148 * 256, 0), (4 * 148 * 256 + 1, 1),
                                      (4 * 148 * 256 + 1023, 0)])
@pytest.mark.parametrize("bits", [16, 32])
def test_counts_around_the_tiles(cuda_device, oracle, n, degree, bits):
    cloud = synthetic.random_cloud(n, seed=n, sh_degree=degree)
    if n > 2:
        cloud.alphas[:: 3] = (np.arange(len(cloud.alphas[:: 3])) % 256) / 255.0
        cloud.alphas[1:: 7] = 1.5  # stored beside the 8-bit opacity, as merged LOD splats are
        if degree:
            cloud.sh[::11] = 6e4
    view, eye = skcam.orbit_view(9, radius=15.0)
    proj = skcam.perspective(math.radians(60.0), W / H, 0.05, 200.0)
    with sk.Renderer(W, H) as r:
        r.apply_render_policy(sk.Policy(sort_depth_bits=bits))
        r.upload_world(cloud, degree)
        r.draw(sk.Frame(view, proj, eye, [(0, n)], degree))
        keys, projected = r.read_visible()
    cam = oracle.camera(view, proj, eye, W, H, 1.0)
    okeys, oproj = oracle.visibility(cam, sk.pack_splats(cloud), sk.pack_sh(cloud, degree),
                                     sk.sh_device_stride(degree), degree, bits, [(0, n)], threads=8)
    assert np.array_equal(keys, okeys)
    assert projected.tobytes() == oproj.tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 2, 15, 16, 17, 40])
def test_ranges_passed_with_the_launch_and_in_memory(cuda_device, oracle, count):
    """Up to 16 ranges are scanned in the kernel's parameters, more are searched in memory: empty ones,
    gaps, ranges out of order and the world's last splat."""
    n, rng = 3001, np.random.default_rng(count)
    cuts = np.sort(rng.integers(0, n + 1, 2 * count))
    ranges = [(int(a), int(b - a)) for a, b in zip(cuts[::2], cuts[1::2])]
    ranges[0] = (ranges[0][0], ranges[0][1] // 2)
    if count > 2:
        ranges[1] = (n, 0)
        ranges[-1] = (n - 7, 7) if ranges[-1][1] >= 7 else (n - 1, min(ranges[-1][1], 1))
        rng.shuffle(ranges)
        ranges = [(int(a), int(b)) for a, b in ranges]
    cloud = synthetic.random_cloud(n, seed=5, sh_degree=1)
    view, eye = skcam.orbit_view(9, radius=15.0)
    proj = skcam.perspective(math.radians(60.0), W / H, 0.05, 200.0)
    with sk.Renderer(W, H) as r:
        r.upload_world(cloud, 1)
        r.draw(sk.Frame(view, proj, eye, ranges, 1))
        keys, projected = r.read_visible()
    cam = oracle.camera(view, proj, eye, W, H, 1.0)
    okeys, oproj = oracle.visibility(cam, sk.pack_splats(cloud), sk.pack_sh(cloud, 1), sk.sh_device_stride(1), 1, 16,
                                     ranges, threads=8)
    assert np.array_equal(keys, okeys)
    assert projected.tobytes() == oproj.tobytes()
