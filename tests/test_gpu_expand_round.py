"""The expand round's splits where they could go wrong: one split, thousands in
a batch (past what k_deep_split keeps in shared memory), a node pool and an
arena that run out inside a round, every pass limit; the whole tree equals the
oracle's, and another batch builds on it."""
import numpy as np
import pytest

from gpu_helpers import (build_gpu, build_oracle, compare_accums, compare_grids, compare_nodes, compare_points,
                         compare_stats, compare_voxels)

pytestmark = pytest.mark.gpu


# limits from one split to several thousand nodes in the first batch
@pytest.mark.parametrize("limit", [60_000, 9_000, 300, 60])
@pytest.mark.parametrize("iters", [20, 3])
def test_whole_tree(c1_cloud, limit, iters):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::16][:120_000])
    cfg = dict(max_points_per_node=limit, max_expand_iters=iters)
    ctx, _ = build_gpu(cloud, bmin, bmax, 80_000, backlog_capacity=10_000_000, store_capacity=12 << 30, **cfg)
    tree = build_oracle(cloud, bmin, bmax, 80_000, persistent_capacity=12 << 30, **cfg)
    tree.accumulate(2)
    nodes = compare_nodes(ctx, tree)
    compare_stats(ctx, tree)
    compare_points(ctx, tree, nodes)
    compare_accums(ctx, tree)
    if limit >= 300:
        compare_voxels(ctx, tree, nodes)
        compare_grids(ctx, tree, nodes)
    ctx.close()
    tree.close()


@pytest.mark.parametrize("max_nodes", [9, 17, 100, 1001, 5000])
def test_node_pool_runs_out_inside_a_round(c1_cloud, max_nodes):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::16][:120_000])
    cfg = dict(max_points_per_node=200, max_nodes=max_nodes)
    ctx, _ = build_gpu(cloud, bmin, bmax, 80_000, backlog_capacity=10_000_000, store_capacity=4 << 30, **cfg)
    tree = build_oracle(cloud, bmin, bmax, 80_000, persistent_capacity=4 << 30, **cfg)
    nodes = compare_nodes(ctx, tree)
    compare_points(ctx, tree, nodes)
    assert ctx.stats().node_capacity_reached == int(len(nodes) + 8 > max_nodes)  # 5,000 hold the whole tree
    ctx.close()
    tree.close()
