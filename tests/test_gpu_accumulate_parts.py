"""Accumulate's items and its watermark where they could go wrong: chunks of one
point, of sizes that four does not divide and longer than a warp's share, folds
on either side of the size that cuts chunks into parts, points past the box and
boxes whose size takes the plain division; sums, counts and the Morton
watermark equal the oracle's and the points'."""
import numpy as np
import pytest

from gpu_helpers import build_gpu, build_oracle, compare_accums, compare_nodes, quant28

pytestmark = pytest.mark.gpu


def _watermark(cloud, bmin, bmax):
    """The largest Morton code of the points' 20-bit coordinates, clamped to the grid."""
    size = np.max(np.asarray(bmax, dtype=np.float32) - np.asarray(bmin, dtype=np.float32))
    code = np.zeros(len(cloud), dtype=np.uint64)
    for k, a in enumerate("xyz"):
        v = np.minimum(quant28(cloud[a], bmin[k], size) >> 8, (1 << 20) - 1).astype(np.uint64)
        for bit in range(20):
            code |= ((v >> np.uint64(bit)) & np.uint64(1)) << np.uint64(3 * bit + 2 - k)
    return int(code.max())


def _check(cloud, bmin, bmax, batch, **cfg):
    # finely split small batches make more new cells than the default list holds
    ctx, _ = build_gpu(cloud, bmin, bmax, batch, per_call=2, backlog_capacity=10_000_000, **cfg)
    cfg.pop("store_capacity", None)
    tree = build_oracle(cloud, bmin, bmax, batch, persistent_capacity=4 << 30, **cfg)
    nb = (len(cloud) + batch - 1) // batch
    tree.accumulate(nb)
    g = ctx.accumulate(nb)
    compare_nodes(ctx, tree)
    compare_accums(ctx, tree)
    assert g.morton_watermark == _watermark(cloud, bmin, bmax)
    assert g.num_accumulated >= len(cloud) and g.sum_leaf_counts == len(cloud)
    assert (g.points_folded, g.num_leaves_folded, g.inner_with_sums) == (0, 0, 0)
    ctx.close()
    tree.close()


@pytest.mark.parametrize("ppc,limit", [(1, 300), (3, 300), (1000, 50_000), (1023, 5000), (6000, 20_000)])
def test_items_of_any_chunk_size(c1_cloud, ppc, limit):
    _, cloud, bmin, bmax = c1_cloud
    _check(np.ascontiguousarray(cloud[:60_001]), bmin, bmax, 9_001, points_per_chunk=ppc, max_points_per_node=limit,
           store_capacity=4 << 30)


def test_fold_above_the_fine_limit(c1_cloud):
    _, cloud, bmin, bmax = c1_cloud
    _check(np.ascontiguousarray(np.concatenate([cloud, cloud])), bmin, bmax, 2_000_000, store_capacity=4 << 30)


# 0.9: a tenth of the tile lies past the box; the others scale it to sizes of about 1e-9, 7 and 1e14 metres
@pytest.mark.parametrize("shrink,scale", [(0.9, 1.0), (1.0, 5e-12), (1.0, 0.035), (1.0, 5e11)])
def test_boxes(c1_cloud, shrink, scale):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::30])
    for a in "xyz":
        cloud[a] *= np.float32(scale)
    bmax = (np.asarray(bmax) * np.float32(scale) * np.float32(shrink)).astype(np.float32)
    _check(cloud, bmin, bmax, 20_011, max_points_per_node=2000, store_capacity=4 << 30)


def test_any_batch_index(c1_cloud):
    """What a caller gives as the batch index is what the touched leaves record."""
    _, cloud, bmin, bmax = c1_cloud
    ctx, _ = build_gpu(np.ascontiguousarray(cloud[:9_001]), bmin, bmax, 9_001, accumulate=0)
    ctx.accumulate(0xFFFFFFFF)
    sums = ctx.accums()
    assert int(sums["count"].sum()) == 9_001
    assert np.all(sums["last_touched_batch"][sums["count"] > 0] == 0xFFFFFFFF)
    ctx.close()


@pytest.mark.parametrize("ppc,limit", [(1000, 1_743_378_284), (10, 1_853_000_612)])
def test_memory_of_a_context(ppc, limit):
    """What a context of the default sizes takes for 2M points with whole chunks as
    work items and colour filtering's sums outside the spill list; no more now."""
    from remobench_b200.lod import Context
    ctx = Context(points_per_chunk=ppc)
    ctx.allocate(2_000_000, (0, 0, 0), (1, 1, 1))
    assert ctx.stats().bytes_allocated <= limit
    ctx.close()


# the smallest chunks that are cut are of 128 points, in folds of under 3,000 chunks
@pytest.mark.parametrize("ppc,limit", [(5, 300), (127, 300), (128, 300), (129, 1000), (130, 50_000)])
def test_items_around_the_smallest_cut_chunk(c1_cloud, ppc, limit):
    _, cloud, bmin, bmax = c1_cloud
    _check(np.ascontiguousarray(cloud[:80_003]), bmin, bmax, 9_001, points_per_chunk=ppc, max_points_per_node=limit,
           store_capacity=4 << 30)


def test_fold_above_the_fine_limit_of_small_chunks(c1_cloud):
    _, cloud, bmin, bmax = c1_cloud
    _check(np.ascontiguousarray(cloud), bmin, bmax, 300_001, points_per_chunk=128, max_points_per_node=5000,
           store_capacity=8 << 30)
