"""The LOD selection in one launch (lod.cu lodWalkKernel) against the oracle, cut and counters, on trees
whose rounds are smaller, equal to and larger than the cluster's blocks and threads, with and without
budgets that deny splits, packets of more than 32 leaves and frustum culling; and the round-by-round
kernels that trees with larger frontiers keep."""
from __future__ import annotations

import numpy as np
import pytest

import splatkit_b200 as sk
from splatkit_b200 import synthetic

from scenes import lod_camera, uniform_nodes


def tree_of(nodes, layout, leaf_count):
    tree = sk.LodTree(nodes, layout, leaf_count)
    tree.clusters, tree.leaves = sk.build_lod_selection(tree)
    return tree


def fan_tree(fan, levels):
    """A complete tree of `fan` children per node, breadth first."""
    inner = sum(fan ** k for k in range(levels))
    total = inner + fan ** levels
    layout = np.zeros(total, sk.LOD_NODE_DTYPE)
    layout["position"] = (0, 0, -2)
    layout["size"] = 0.02
    layout["child_start"][:inner] = 1 + fan * np.arange(inner)
    layout["child_count"][:inner] = fan
    nodes = uniform_nodes(total)
    nodes.positions[:, 0] = np.linspace(-1.5, 1.5, total)
    return tree_of(nodes, layout, fan ** levels)


def check(oracle, tree, budget, pixels, cull, distance=0.0):
    view, proj, pos = lod_camera(distance)
    proj = proj.copy()
    proj[0] = proj[5] = 1.0
    r = sk.Renderer(1000, 1000)
    r.apply_render_policy(sk.Policy(lod_error_pixels=pixels, enable_frustum_culling=cull))
    r.upload_lod_world(tree, 0, budget)
    r.draw(sk.Frame(view, proj, pos, [], 0))
    cut, stats = r.read_cut()
    assert r.stats()["device_error"] == 0
    r.close()
    cam = oracle.camera(view, proj, pos, 1000, 1000, 0.0)
    ocut, ostats = oracle.lod_select(cam, tree.clusters, tree.leaves,
                                     sk.lod_depth(tree.layout, tree.leaf_count) + 1,
                                     min(budget, 4_000_000, tree.leaf_count), pixels, 4.0, cull)
    assert np.array_equal(stats, ostats)
    assert np.array_equal(cut, ocut)
    return len(cut)


@pytest.mark.gpu
@pytest.mark.parametrize("fan,levels", [(2, 15), (8, 4), (3, 9), (40, 3), (513, 1)])
def test_complete_trees_at_every_kind_of_budget(oracle, cuda_device, fan, levels):
    tree = fan_tree(fan, levels)
    full = fan ** levels
    for budget in {1, 2, fan, fan + 1, full // 3 + 1, full - 1, full, 10 * full}:
        check(oracle, tree, budget, 1e-6, False)
    assert check(oracle, tree, full, 1e-6, False) == full


@pytest.mark.gpu
@pytest.mark.parametrize("budget,pixels", [(4_000_000, 0.5), (4_000_000, 2.0), (9_000, 0.5), (37, 0.1)])
def test_clustered_tree_with_culling(oracle, cuda_device, budget, pixels):
    cloud = synthetic.clustered_cloud(clusters=60, per_cluster=800, seed=8, half_extent=15.0)
    tree = sk.build_lod_tree(cloud, cluster_leaves=40)
    for distance in (0.0, 10.0, 60.0):
        check(oracle, tree, budget, pixels, True, distance)


@pytest.mark.gpu
def test_a_frontier_beyond_the_one_launch_walk(oracle, cuda_device):
    tree = fan_tree(2, 21)  # 2,097,151 clusters: the rounds' own kernels
    check(oracle, tree, 4_000_000, 1e-6, False)
    check(oracle, tree, 1_500_000, 1e-6, False)
