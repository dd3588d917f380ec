"""Colour filtering where its units, tables and chains could go wrong: chunks of
one point and longer than a unit, a root that never split, queues of nested
nodes and of leaves without voxels, points past the declared box, a capacity
that admits part of the queue."""
import numpy as np
import pytest

from gpu_helpers import build_gpu, build_oracle, compare_nodes, compare_voxels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,ppc,limit,shrink,capacity", [
    (900, 1000, 1000, 1.0, 0), (1_100, 1, 1000, 1.0, 0), (50_001, 7, 300, 1.0, 0), (50_001, 5000, 12_000, 1.0, 0),
    (200_000, 1000, 700, 1.0, 0), (200_000, 1000, 700, 0.8, 0), (200_000, 1000, 5000, 1.0, 20_000)])
def test_filtered_colours_equal_the_oracle(c1_cloud, points, ppc, limit, shrink, capacity):
    from remobench_b200.lod import make_frame
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::len(cloud) // points][:points])
    bmax = (np.asarray(bmax) * np.float32(shrink)).astype(np.float32)
    cfg = dict(points_per_chunk=ppc, max_points_per_node=limit)
    ctx, _ = build_gpu(cloud, bmin, bmax, 20_011, store_capacity=4 << 30, refine_voxel_capacity=capacity, **cfg)
    tree = build_oracle(cloud, bmin, bmax, 20_011, persistent_capacity=4 << 30, **cfg)
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.3, pitch=-0.5, radius_scale=0.5)
    ctx.analyze(f, min_points=1, frontier_only=False, queue_capacity=16_384)
    queue = ctx.queue()
    cap = capacity or 2_097_152
    for budget in (1, len(queue) // 3, len(queue)):
        r = ctx.refine_colors(budget)
        m, nv = tree.refine_colors(queue[:budget], capacity=cap)
        assert (r.nodes_filtered, r.voxels_filtered) == (m, nv)
        nodes = ctx.nodes()
        compare_voxels(ctx, tree, nodes)
        # every stored point once per filtered node above it (or its own)
        above = np.zeros(len(nodes), dtype=np.int64)
        taken = np.zeros(len(nodes), dtype=np.int64)
        taken[queue[:m]] = 1
        for i in np.argsort(nodes["level"], kind="stable"):
            above[i] += taken[i]
            kids = nodes["child"][i]
            above[kids[kids >= 0]] += above[i]
        assert r.points_visited == int((above * nodes["num_points"])[nodes["is_leaf"] == 1].sum())
    ctx.close()
    tree.close()


def test_points_visited_where_chunks_are_missing(c1_cloud):
    """A batch larger than the arena: the points without a chunk are dropped and
    not counted as visited."""
    from remobench_b200.lod import make_frame
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(np.concatenate([cloud, cloud[:900_000]]))
    ctx, _ = build_gpu(cloud, bmin, bmax, len(cloud), store_capacity=1 << 20, safety_margin=0)
    s = ctx.stats()
    assert s.overflow_flags & 8 and 0 < s.dropped_points < len(cloud)
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.3, pitch=-0.5, radius_scale=0.5)
    ctx.analyze(f, min_points=int(0.6 * len(cloud)), frontier_only=False)
    assert ctx.queue().tolist() == [0]
    r = ctx.refine_colors(1)
    assert r.nodes_filtered == 1 and r.points_visited == len(cloud) - s.dropped_points
    ctx.close()


# 25,000 voxels' sums are exactly as long as the list of 100,000 spilled points
@pytest.mark.parametrize("capacity", [25_000, 25_001])
def test_sums_in_the_spill_list_and_beside_it(c1_cloud, capacity):
    """Batches before, between and after filterings equal the oracle's."""
    from remobench_b200.lod import DeviceRing, make_frame
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::16])
    cfg = dict(max_points_per_node=2000)
    step = 30_000
    ctx, _ = build_gpu(cloud[:step], bmin, bmax, step, spilled_capacity=100_000, refine_voxel_capacity=capacity, **cfg)
    tree = build_oracle(cloud[:step], bmin, bmax, step, **cfg)
    ring = DeviceRing(cloud, step, slots=ctx.cfg.ring_slots, slot_capacity=step)
    ring.upload_window(0)
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.3, pitch=-0.5, radius_scale=0.5)
    for k in range(1, 4):
        ctx.analyze(f, min_points=1, frontier_only=False)
        queue = ctx.queue()
        r = ctx.refine_colors(len(queue))
        assert (r.nodes_filtered, r.voxels_filtered) == tree.refine_colors(queue, capacity=capacity)
        assert r.voxels_filtered > 0
        ctx.build(ring.ring, ring.sizes, k + 1, ring.num_batches)
        tree.add_batch(cloud[k * step:(k + 1) * step])
        tree.sweep()
        nodes = compare_nodes(ctx, tree)
        compare_voxels(ctx, tree, nodes)
    ctx.close()
    tree.close()


@pytest.mark.parametrize("points,limit,shrink", [(60_001, 300, 1.0), (60_001, 300, 0.8), (200_000, 5000, 1.0)])
def test_cloud_that_fills_its_volume(c1_cloud, points, limit, shrink):
    """Few points a voxel: the points go to their entries one by one."""
    from remobench_b200.lod import make_frame
    _, cloud, bmin, bmax = c1_cloud
    cloud = cloud[:points].copy()
    rng = np.random.default_rng(3)
    for k, a in enumerate("xyz"):
        cloud[a] = rng.uniform(bmin[k], bmax[k], points)
    bmax = (np.asarray(bmax) * np.float32(shrink)).astype(np.float32)
    cfg = dict(max_points_per_node=limit)
    # more new cells a batch than the default list holds
    ctx, _ = build_gpu(cloud, bmin, bmax, 20_011, store_capacity=4 << 30, backlog_capacity=1_000_000, **cfg)
    tree = build_oracle(cloud, bmin, bmax, 20_011, persistent_capacity=4 << 30, **cfg)
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.3, pitch=-0.5, radius_scale=0.5)
    ctx.analyze(f, min_points=1, frontier_only=False, queue_capacity=16_384)
    queue = ctx.queue()
    for budget in (1, len(queue)):
        r = ctx.refine_colors(budget)
        assert (r.nodes_filtered, r.voxels_filtered) == tree.refine_colors(queue[:budget])
        nodes = compare_nodes(ctx, tree)
        compare_voxels(ctx, tree, nodes)
    with_voxels = nodes["num_voxels"][queue] > 0
    assert r.points_visited < 4 * r.voxels_filtered + int(nodes["num_points"][queue[~with_voxels]].sum())
    ctx.close()
    tree.close()


def test_one_cell_of_17_million_points():
    """More points in a chunk, and in one cell, than 32-bit sums of colours hold."""
    from remobench_b200.lod import make_frame
    n, box = 17_000_000, (np.zeros(3, np.float32), np.full(3, 128.0, np.float32))
    cloud = np.zeros(n, dtype=np.dtype([("x", "<f4"), ("y", "<f4"), ("z", "<f4"), ("color", "<u4")]))
    for k, a in enumerate("xyz"):
        cloud[a] = 0.5
        # in another octant, so that the root splits; near its corner, as the others
        cloud[a][-100_000:] = np.random.default_rng(k).uniform(0.0, 1.0, 100_000) + (65.0 if k == 0 else 0.0)
    cloud["color"] = 0xFF00FFFF
    cloud["color"][0] = 0xFF000000  # the voxel's own colour, of the lowest index
    ctx, _ = build_gpu(cloud, *box, n, points_per_chunk=20_000_000, max_points_per_node=16_950_000, backlog_capacity=200_000,
                       store_capacity=4 << 30)

    def colour():
        v = ctx.node_voxels(0)
        return v["color"][v["x"] == 0.5].tolist()
    ctx.analyze(make_frame(*box, 1920, 1080, yaw=1.3, pitch=-0.5, radius_scale=0.5), min_points=1, frontier_only=False)
    queue = ctx.queue()
    assert 0 in queue and colour() == [0xFF000000]
    ctx.refine_colors(len(queue))
    assert colour() == [0xFF00FFFF]
    ctx.close()
