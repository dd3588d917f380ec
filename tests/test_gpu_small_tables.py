"""The cell tables at their smallest: colour filtering and the batch's list of
new cells take as many cells as they are sized for, at capacities of a few
cells and with the list just full."""
import numpy as np
import pytest

from gpu_helpers import build_oracle, compare_grids, compare_nodes, compare_stats, compare_voxels
from oracle import binding as ob

BOX = (np.zeros(3, np.float32), np.full(3, 128.0, np.float32))  # a root cell is one unit wide


def _points(xyz, rng):
    p = np.zeros(len(xyz), dtype=ob.POINT_DTYPE)
    for k, a in enumerate("xyz"):
        p[a] = xyz[:, k]
    p["color"] = rng.integers(0, 1 << 32, len(xyz), dtype=np.uint64).astype(np.uint32)
    return p


def _cells(n, rng, flat):
    """n distinct root cells of a surface or of the whole cube, not all in one octant."""
    while True:
        c = rng.integers(0, 128, (n, 3))
        if flat:
            c[:, 2] = 40 + c[:, 0] // 16
        if len(np.unique(c, axis=0)) == n and len(np.unique(c // 64, axis=0)) > 1:
            return c


def filter_cloud(cells, seed):
    """Three points of random colours in each of `cells` root cells: a root that
    splits (above 3 cells - 1 points) keeps that many voxels."""
    rng = np.random.default_rng(seed)
    c = np.repeat(_cells(cells, rng, seed % 2 == 0), 3, axis=0)
    return _points((c + rng.uniform(0.1, 0.9, c.shape)).astype(np.float32), rng)


def _prefix(pts, batch, new_cells, limit):
    """The points before the first batch that makes more than `new_cells` new
    cells, and the most that one of theirs makes."""
    made, keep, most = 0, 0, 0
    tree = ob.Tree(max_points_per_node=limit)
    tree.reset(*BOX)
    while keep < len(pts):
        tree.add_batch(pts[keep:keep + batch])
        v = int(tree.node_table()["num_voxels"].sum())
        if v - made > new_cells:
            break
        most, made, keep = max(most, v - made), v, keep + batch
    tree.close()
    return most, keep


def batch_cloud(seed, slot, new_cells, limit):
    """A cloud whose batches fill the list of new cells as far as some batch size
    up to `slot` can without passing it: (points, batch, the most cells of a batch)."""
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0.0, 128.0, (100 + 4 * slot, 3))
    if seed % 2 == 0:
        xyz[:, 2] = 40.0 + xyz[:, 0] / 16.0
    pts = _points(xyz.astype(np.float32), rng)
    sizes = np.unique(np.linspace(1, min(slot, new_cells), 12).astype(int))
    (most, keep), batch = max((_prefix(pts, int(b), new_cells, limit), int(b)) for b in sizes)
    return np.ascontiguousarray(pts[:keep]), batch, most


def _context(slot, points, **cfg):
    from remobench_b200.lod import Context
    ctx = Context(slot_capacity=slot, time_budget_ms=0.0, max_nodes=20_000, **cfg)
    ctx.allocate(points, *BOX)
    return ctx


def _rebuild(ctx, pts, batch):
    """The cloud through the context's device ring, into a tree started anew."""
    from remobench_b200.lod import DeviceRing
    ctx.reset()
    ring = DeviceRing(pts, batch, slots=ctx.cfg.ring_slots, slot_capacity=ctx.cfg.slot_capacity)
    consumed = 0
    while consumed < ring.num_batches:
        ring.upload_window(consumed)
        r = ctx.build(ring.ring, ring.sizes, ring.uploaded, ring.num_batches)
        assert r.batches_this_call > 0
        consumed = r.batches_consumed


@pytest.mark.gpu
@pytest.mark.parametrize("capacity", [2, 3, 4, 8, 16, 32, 64])
def test_colour_filter_takes_its_capacity(capacity):
    from remobench_b200.lod import make_frame
    n = 3 * capacity
    ctx = _context(n, n, max_points_per_node=n - 1, refine_voxel_capacity=capacity)
    f = make_frame(*BOX, 1920, 1080, yaw=1.3, pitch=-0.5, radius_scale=0.5)
    for seed in range(30):
        pts = filter_cloud(capacity, seed)
        _rebuild(ctx, pts, n)
        tree = build_oracle(pts, *BOX, n, max_points_per_node=n - 1)
        ctx.analyze(f, min_points=1, frontier_only=False)
        queue = ctx.queue()
        assert 0 in queue
        r = ctx.refine_colors(len(queue))
        m, nv = tree.refine_colors(queue, capacity=capacity)
        assert (r.nodes_filtered, r.voxels_filtered) == (m, nv)
        assert nv == capacity  # the table is as full as it gets
        nodes = compare_nodes(ctx, tree)
        compare_voxels(ctx, tree, nodes)
        tree.close()
    ctx.close()


# (slot_capacity, backlog_capacity, points per node); the list holds
# backlog_capacity cells, or two per point of a slot rounded up to a power of two
CASES = [(1, 0, 1), (2, 0, 1), (4, 0, 2), (8, 0, 4), (16, 0, 8), (32, 0, 16), (64, 0, 32), (4, 10, 4), (16, 5, 2),
         (64, 20, 6)]


def batch_clouds(slot, backlog, limit):
    new_cells = backlog or 2 * slot
    return new_cells, [batch_cloud(seed, slot, new_cells, limit) for seed in range(24)]


@pytest.mark.gpu
@pytest.mark.parametrize("slot,backlog,limit", CASES)
def test_batches_take_their_list(slot, backlog, limit):
    _, clouds = batch_clouds(slot, backlog, limit)
    ctx = _context(slot, 1000, max_points_per_node=limit, backlog_capacity=backlog)
    for pts, batch, _ in clouds:
        _rebuild(ctx, pts, batch)
        tree = build_oracle(pts, *BOX, batch, max_points_per_node=limit)
        nodes = compare_nodes(ctx, tree)
        compare_stats(ctx, tree)
        compare_voxels(ctx, tree, nodes)
        compare_grids(ctx, tree, nodes)
        tree.close()
    ctx.close()


@pytest.mark.parametrize("slot,backlog,limit", CASES)
def test_batches_fill_their_list(slot, backlog, limit):
    """The batches above reach the size of the list without passing it."""
    new_cells, clouds = batch_clouds(slot, backlog, limit)
    assert max(most for _, _, most in clouds) == new_cells
    assert all(len(pts) for pts, _, _ in clouds)
