"""The raster's split of the samples over the warps, the cut's list and the EDL
tiles where they could go wrong: chunks of one point and of odd sizes, frames
smaller than a tile and of ragged widths, a full draw list, flat clouds of one
point and around a block's share, wide splats."""
import numpy as np
import pytest

from gpu_helpers import build_gpu, build_oracle
from oracle import binding as ob
from test_gpu_render import oracle_frame

pytestmark = pytest.mark.gpu


def _frame(bmin, bmax, w, h, **kw):
    from remobench_b200.lod import make_frame
    return make_frame(bmin, bmax, w, h, yaw=1.9, pitch=-0.5, radius_scale=0.45, **kw)


def _buffers(w, h):
    import torch
    return (torch.empty(w * h, dtype=torch.int64, device="cuda"), torch.empty(w * h, dtype=torch.int32, device="cuda"))


def _u64(t):
    return t.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("ppc,limit", [(1, 400), (7, 400), (333, 2000), (1000, 50000)])
def test_lod_frame_for_chunk_sizes(c1_cloud, ppc, limit):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::40])
    cfg = dict(points_per_chunk=ppc, max_points_per_node=limit)
    ctx, _ = build_gpu(cloud, bmin, bmax, 20_011, store_capacity=6 << 30, **cfg)
    tree = build_oracle(cloud, bmin, bmax, 20_011, persistent_capacity=6 << 30, **cfg)
    for w, h, ps in ((1, 1, 1), (63, 17, 1), (641, 359, 3), (1280, 720, 1)):
        f = _frame(bmin, bmax, w, h, budget=40.0, point_size=ps)
        fb, rgba = _buffers(w, h)
        r = ctx.render(f, fb, rgba)
        ofb, orr, _ = tree.render(oracle_frame(f))
        assert (r.draw_items, r.draw_samples) == (orr.draw_items, orr.draw_samples)
        assert np.array_equal(_u64(fb), ofb), (w, h)
        assert np.array_equal(rgba.cpu().numpy().view(np.uint32), (ofb & 0xFFFFFFFF).astype(np.uint32))
    ctx.close()
    tree.close()


def test_full_draw_list(c1_cloud):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::10])
    f = _frame(bmin, bmax, 640, 360, budget=30.0)
    full, _ = build_gpu(cloud, bmin, bmax, 100_000, max_points_per_node=2000)
    fb, _ = _buffers(640, 360)
    n = full.render(f, fb).draw_items
    whole = _u64(fb)
    for cap in (1, 5, n - 1, n):
        ctx, _ = build_gpu(cloud, bmin, bmax, 100_000, max_points_per_node=2000, drawlist_capacity=cap)
        r = ctx.render(f, fb)
        part = _u64(fb)
        assert r.draw_items == n and r.drawlist_overflow == (1 if cap < n else 0)
        assert np.all(part >= whole) and (cap < n or np.array_equal(part, whole))
        assert 0 < np.count_nonzero(part < np.uint64(0x7F80000000332211)) <= r.draw_samples
        ctx.close()
    full.close()


# 1 x 1 up to past one 16-row tile; 2048 x 2049 takes the 32-row tiles (4 Mi pixels and up)
@pytest.mark.parametrize("w,h", [(1, 1), (2, 3), (64, 16), (65, 17), (199, 101), (2048, 2049)])
def test_edl_tiles_and_colours(c1_cloud, w, h):
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::20])
    ctx, _ = build_gpu(cloud, bmin, bmax, 50_000)
    fb, rgba = _buffers(w, h)
    ctx.render(_frame(bmin, bmax, w, h), fb)
    oe = ob.edl(_u64(fb), w, h, 0.4)
    ctx.render(_frame(bmin, bmax, w, h, edl=True), fb, rgba)
    g = _u64(fb)
    assert np.array_equal(g >> np.uint64(32), oe >> np.uint64(32))
    assert np.array_equal(rgba.cpu().numpy().view(np.uint32), (g & np.uint64(0xFFFFFFFF)).astype(np.uint32))
    steps = [np.abs((g >> np.uint64(s) & np.uint64(255)).astype(int) - (oe >> np.uint64(s) & np.uint64(255)).astype(int))
             for s in (0, 8, 16, 24)]
    assert max(int(s.max()) for s in steps) <= 1  # libm against CUDA log2f and expf
    ctx.close()


@pytest.mark.parametrize("n", [1, 31, 33, 255, 513, 40_000, 300_001])
@pytest.mark.parametrize("ps", [1, 3])
def test_flat_frame(c1_cloud, n, ps):
    import torch
    from remobench_b200.lod import Context
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[:n])
    ctx = Context(pipeline=2)
    ctx.allocate(n, bmin, bmax)
    w, h = 333, 111  # small: pixels shared by many points
    f = _frame(bmin, bmax, w, h, point_size=ps)
    fb, _ = _buffers(w, h)
    ctx.render_flat(f, torch.from_numpy(cloud.view(np.float32).reshape(-1, 4)).cuda(), fb)
    assert np.array_equal(_u64(fb), ob.render_flat(cloud, oracle_frame(f)))
    ctx.close()


def test_flat_frame_of_more_than_2_32_pixels():
    """Points of one column in rows 32768 apart, 2^32 pixels in index: the nearer
    ones hide nothing of the further ones. 34 GB of framebuffer."""
    import torch
    from remobench_b200 import capi
    from remobench_b200.lod import Context
    w, h, group, far_row = 131_072, 32_769, 1024, 32_768
    f = capi.Frame()
    f.width, f.height, f.lod_pixel_budget, f.point_size = float(w), float(h), 128.0, 1
    for t in (f.transform, f.transform_frozen):
        t[0] = t[5] = t[10] = t[14] = 1.0  # clip = (x, y, z, z)
    for a in range(3):
        f.box_min[a], f.box_max[a] = -4.0, 4.0
    # 1,024 columns, each 512 points near in the first row, then 512 further in the last
    i = np.arange(group * group)
    col, far = (i // group) * 128, i % group >= group // 2
    z = np.where(far, 2.0, 1.0)
    p = np.zeros(len(i), dtype=ob.POINT_DTYPE)
    p["x"] = ((2 * col + 1) / w - 1.0) * z
    p["y"] = ((2 * np.where(far, far_row, 0) + 1) / h - 1.0) * z
    p["z"] = z
    p["color"] = np.where(far, 7, 3)
    fb = torch.empty(w * h, dtype=torch.int64, device="cuda")
    ctx = Context(pipeline=2)
    ctx.allocate(len(p), (-4, -4, -4), (4, 4, 4))
    ctx.render_flat(f, torch.from_numpy(p.view(np.float32).reshape(-1, 4)).cuda(), fb)
    at = torch.arange(group, device="cuda") * 128
    depth = {1.0: 0x3F800000, 2.0: 0x40000000}
    assert np.all(_u64(fb[at]) == (depth[1.0] << 32 | 3))
    assert np.all(_u64(fb[far_row * w + at]) == (depth[2.0] << 32 | 7))
    ctx.close()
    del fb, at
    torch.cuda.empty_cache()


@pytest.mark.parametrize("ps", [-5, 0, 2, 4, 5, 7, 8, 10, 25, 1000])
def test_splats_of_any_size(c1_cloud, ps):
    """Rows of a splat around four pixels, wider than the frame, of no size."""
    import torch
    _, cloud, bmin, bmax = c1_cloud
    cloud = np.ascontiguousarray(cloud[::4000])
    ctx, _ = build_gpu(cloud, bmin, bmax, 200, max_points_per_node=50)
    tree = build_oracle(cloud, bmin, bmax, 200, max_points_per_node=50)
    pts = torch.from_numpy(cloud.view(np.float32).reshape(-1, 4)).cuda()
    for w, h in ((1, 1), (61, 37), (320, 200)):
        f = _frame(bmin, bmax, w, h, budget=40.0, point_size=ps)
        fb, _ = _buffers(w, h)
        ctx.render(f, fb)
        assert np.array_equal(_u64(fb), tree.render(oracle_frame(f))[0])
        ctx.render_flat(f, pts, fb)
        assert np.array_equal(_u64(fb), ob.render_flat(cloud, oracle_frame(f)))
    ctx.close()
    tree.close()
