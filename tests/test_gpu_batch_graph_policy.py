"""A replayed batch graph draws under the batch's current policy: a background or early termination changed
between two submissions of the same views on the same lane."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from test_gpu_cell_lists import frames_for

SIZES = [(320, 240), (97, 61)]


@pytest.mark.gpu
@pytest.mark.parametrize("policy", [sk.Policy(background=(0.9, 0.1, 0.4)),
                                    sk.Policy(enable_early_termination=False),
                                    sk.Policy(subpixel_threshold=3.0)])
def test_a_replayed_graph_draws_under_the_new_policy(cuda_device, policy):
    cloud = synthetic.random_cloud(60_000, seed=81, sh_degree=0, log_scale_mean=-1.5)
    with sk.Renderer(64, 64) as r, sk.Batch(lanes=1, max_views=4, use_graphs=True) as graphs, \
            sk.Batch(lanes=1, max_views=4) as plain:
        r.upload_world(cloud, 0)
        views = [sk.BatchView(r, frames_for(cloud, w, h, (11,))[0], w, h) for w, h in SIZES]
        results = {}
        for batch in (graphs, plain):
            for p in (sk.Policy(), policy, sk.Policy()):  # captured, then replayed or captured anew
                batch.apply_render_policy(p)
                t = batch.submit(views)
                results.setdefault(batch, []).append(
                    ([batch.read_image(t, i) for i in range(len(views))], batch.stats(t)["fragments"],
                     [batch.view_visible(t, i) for i in range(len(views))]))
        for (ia, fa, va), (ib, fb, vb) in zip(results[graphs], results[plain]):
            assert all(np.array_equal(a, b) for a, b in zip(ia, ib))
            assert (fa, va) == (fb, vb)
        first, second = results[plain][0], results[plain][1]
        assert first[1:] != second[1:] or not np.array_equal(first[0][0], second[0][0])
