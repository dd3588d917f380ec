"""The one-launch roll-up and the queue's radix select at the trees and queue
lengths where they could go wrong: a root that never split, one split, deep and
wide trees, sibling groups that a collapse detached; queues of one entry, of
every eligible node and of more than there are."""
import numpy as np
import pytest

from gpu_helpers import build_gpu, build_oracle

pytestmark = pytest.mark.gpu


def _analyzed(cloud, bmin, bmax, batch, limit, **kw):
    from remobench_b200.lod import make_frame
    ctx, _ = build_gpu(cloud, bmin, bmax, batch, max_points_per_node=limit, store_capacity=4 << 30)
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.2, pitch=-0.5, radius_scale=0.5)
    return ctx, f, ctx.analyze(f, frontier_only=False, **kw)


@pytest.mark.parametrize("points,limit,nodes", [(700, 1000, 1), (1300, 1000, 9), (60_001, 300, None), (262_144, 2000, None)])
def test_rollup_equals_the_oracle(c1_cloud, points, limit, nodes):
    cfg, cloud, bmin, bmax = c1_cloud
    step = max(1, len(cloud) // points)
    cloud = np.ascontiguousarray(cloud[::step][:points])
    ctx, f, _ = _analyzed(cloud, bmin, bmax, 20_011, limit)
    tree = build_oracle(cloud, bmin, bmax, 20_011, max_points_per_node=limit, persistent_capacity=4 << 30)
    tree.accumulate((points + 20_010) // 20_011)
    g = ctx.rollup()
    assert nodes is None or len(g) == nodes
    assert np.array_equal(g, tree.rolled_sums()[0])
    ctx.analyze(f)  # the arrival counters are back at zero
    assert np.array_equal(ctx.rollup(), g)
    ctx.close()
    tree.close()


def test_rollup_skips_detached_groups(c1_cloud):
    cfg, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[:200_000])
    ctx, f, _ = _analyzed(cloud, bmin, bmax, 50_000, 1000)
    nodes = ctx.nodes()
    kids = nodes["child"]
    twigs = [i for i in range(1, len(nodes)) if not nodes["is_leaf"][i] and np.all(nodes["is_leaf"][kids[i]] == 1)]
    assert ctx.refine_collapse(twigs[::2], max_points=1_000_000).nodes_collapsed == len(twigs[::2])
    ctx.analyze(f)
    g = ctx.rollup()
    assert g[0, 0] == len(cloud)
    after = ctx.nodes()
    for i in np.nonzero(after["is_leaf"] == 0)[0]:
        assert g[i, 0] == g[after["child"][i], 0].sum(), i
    assert np.all(g[after["is_leaf"] == 1, 0] == after["num_points"][after["is_leaf"] == 1])
    ctx.close()


@pytest.mark.parametrize("k", [1, 2, 31, 1000, 16_384])
def test_queue_is_the_top_k(c1_cloud, k):
    cfg, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[:400_000])
    ctx, f, r = _analyzed(cloud, bmin, bmax, 100_000, 1000, queue_capacity=k)
    for _ in range(2):  # the histogram is back at zero after a call
        a, q = ctx.analysis(), ctx.queue()
        ids = np.nonzero(a["score"] > 0)[0]
        order = ids[np.lexsort((ids, -a["score"][ids]))]
        assert r.eligible == len(ids) > 1000
        assert r.overflow == 0 and np.array_equal(q, order[:k])
        r = ctx.analyze(f, frontier_only=False, queue_capacity=k)
    ctx.close()


def test_mask_is_the_queue_prefix_on_a_changed_tree(c1_cloud):
    """The mask marks the queue's prefix, and nothing else: after an analysis of
    a larger tree whose keys are still there, and when the tree grew since."""
    import torch
    from remobench_b200.lod import Context, DeviceRing, make_frame
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[:400_000])
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.2, pitch=-0.5, radius_scale=0.5)
    ctx = Context(slot_capacity=100_000, max_points_per_node=1000, time_budget_ms=0.0, max_batches_per_build=1,
                  store_capacity=4 << 30)
    ctx.allocate(len(cloud), bmin, bmax)
    ring = DeviceRing(cloud, 100_000, slots=ctx.cfg.ring_slots, slot_capacity=100_000)
    ring.upload_window(0)
    mask = torch.empty(ctx.cfg.max_nodes, dtype=torch.uint8, device="cuda")
    for upto in (4, 1):  # a large tree first, then a small one after a reset
        ctx.reset()
        for k in range(upto):
            ctx.build(ring.ring, ring.sizes, k + 1, ring.num_batches)
        ctx.analyze(f, frontier_only=False, queue_capacity=2000)
        q = ctx.queue()
        for grown in (False, True):
            if grown:
                ctx.build(ring.ring, ring.sizes, min(upto + 1, 4), ring.num_batches)
            nn = ctx.stats().num_nodes
            for budget in (0, 1, len(q) // 2, len(q), 1 << 30):
                mask.fill_(7)
                torch.cuda.synchronize()
                ctx.refine(budget, mask)
                m = mask.cpu().numpy()
                assert set(np.nonzero(m[:nn])[0].tolist()) == set(q[:budget].tolist())
                assert np.all(m[:nn] <= 1) and np.all(m[nn:] == 7)
    ctx.close()


def test_read_backs_follow_every_change(c1_cloud):
    """Nodes, sums and analysis read right after each call that changes the tree."""
    from remobench_b200.lod import Context, DeviceRing, make_frame
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[:400_000])
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.2, pitch=-0.5, radius_scale=0.5)
    for graphs in (1, 0):
        ctx = Context(slot_capacity=100_000, max_points_per_node=5000, time_budget_ms=0.0, max_batches_per_build=1,
                      use_graphs=graphs)
        ctx.allocate(len(cloud), bmin, bmax)
        ring = DeviceRing(cloud, 100_000, slots=ctx.cfg.ring_slots, slot_capacity=100_000)
        ring.upload_window(0)
        assert len(ctx.nodes()) == 1
        for k in range(4):
            r = ctx.build(ring.ring, ring.sizes, k + 1, ring.num_batches)
            assert r.batches_this_call == 1 and r.batches_consumed == k + 1
            nodes, sums = ctx.nodes(), ctx.accums()
            assert len(nodes) == len(sums) == ctx.stats().num_nodes
            assert int(sums["count"].sum()) == int(nodes["num_points"][nodes["is_leaf"] == 1].sum()) == 100_000 * (k + 1)
            assert np.all(sums["last_touched_batch"][sums["count"] > 0] <= k + 1)
            assert np.any(sums["last_touched_batch"] == k + 1)
        ctx.analyze(f, frontier_only=False)
        before = len(ctx.nodes())
        assert len(ctx.analysis()) == len(ctx.features()) == before
        d = ctx.refine_deepen(8)
        assert len(ctx.nodes()) == before + 8 * d.nodes_split and d.nodes_split > 0
        assert int(ctx.accums()["count"].sum()) == len(cloud)
        ctx.reset()
        assert len(ctx.nodes()) == 1 and int(ctx.accums()["count"].sum()) == 0
        r = ctx.ingest_host(cloud, 100_000)
        assert r.batches_consumed == 4 and len(ctx.nodes()) == ctx.stats().num_nodes > 1
        assert int(ctx.accums()["count"].sum()) == len(cloud)
        ctx.close()


def test_mask_after_more_candidates_than_the_sort_holds(c1_cloud):
    """Then the queue keeps some of the candidates, and the mask marks those alone."""
    import torch
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[:400_000])
    ctx, _ = build_gpu(cloud, bmin, bmax, 100_000, max_points_per_node=30, store_capacity=6 << 30,
                       backlog_capacity=4_000_000)
    from remobench_b200.lod import make_frame
    f = make_frame(bmin, bmax, 1920, 1080, yaw=1.2, pitch=-0.5, radius_scale=0.5)
    r = ctx.analyze(f, min_points=1, frontier_only=False, queue_capacity=16_384)
    q = ctx.queue()
    assert r.overflow == 1 and len(q) == 16_384 and len(set(q.tolist())) == len(q)
    mask = torch.full((ctx.cfg.max_nodes,), 7, dtype=torch.uint8, device="cuda")
    for budget in (1, 5000, 16_384):
        torch.cuda.synchronize()
        ctx.refine(budget, mask)
        m = mask.cpu().numpy()
        nn = ctx.stats().num_nodes
        assert set(np.nonzero(m[:nn])[0].tolist()) == set(q[:budget].tolist())
        assert np.all(m[:nn] <= 1) and np.all(m[nn:] == 7)
    ctx.close()
