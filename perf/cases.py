"""What the speed of this framework is measured on.

A case is one pass of work that a program hands to the public entry points
(remobench_b200.lod.Context): build a progressive LOD tree from a cloud, draw
it, analyse and refine it, train the scorer that ranks the refinement. The
clouds are the seeded synthetic lidar scans the benchmark and the tests use
(remobench_b200.synth), at the benchmark's densities and at ragged sizes.

Kinds of pass, and who asks for them:

  ingest       the headless harness: reset, the whole cloud from a device ring
               in batches (Update + Accumulate), one frame, the statistics
  ingest_host  the same from pinned host memory
  stream       the viewer's loop: per frame one batch, Analysis, Refinement's
               budget, and the refined frame
  frame        one frame of the streaming run on a finished tree: Analysis,
               budget, refined render with EDL
  render       one frame of a finished tree, no refinement
  flat         one frame of every point, the quality harness's ground truth
  analyze      Analysis alone with everything it logs, ranked by the learned
               scorer, as the scorer's data collection reads it
  filter       Refinement's colour filtering and the frame that shows it
  train        optimiser steps of the scorer on one minibatch each
  gradients    the scorer's loss and gradient over a whole data set
"""
import math

import numpy as np
import torch

from remobench_b200 import capi, synth
from remobench_b200.camera import orbit_path
from remobench_b200.lod import ACCUM_DTYPE, ANALYSIS_DTYPE, Context, make_frame

PX = {"360p": (640, 360), "720p": (1280, 720), "1080p": (1920, 1080), "4k": (3840, 2160), "8k": (7680, 4320)}
SCORER_SIZES = ((64, 16), (64,), (64, 64), (64,), (2, 64), (2,))  # W1 b1 W2 b2 W3 b3


def listed():
    return [
        # one batch that fits a single leaf or two: a viewer's first frame, a preview tile
        {"name": "ingest_first_batch", "kind": "ingest", "points": 100_000, "batch": 100_000, "scene": 1,
         "limit": 50_000, "frame": "720p"},
        # configuration 1: a 2M-point tile in 256K batches
        {"name": "ingest_tile_2m", "kind": "ingest", "points": 2_097_152, "batch": 262_144, "scene": 1,
         "limit": 50_000, "frame": "720p"},
        # configuration 2's scan, 1M-point batches, 20 per build call, the last one ragged
        {"name": "ingest_scan_24m", "kind": "ingest", "points": 23_654_321, "batch": 1_000_000, "scene": 2,
         "limit": 50_000, "frame": "1080p"},
        # configuration 5's streaming: 4M-point batches from pinned host memory, 5% outliers
        {"name": "ingest_host_12m", "kind": "ingest_host", "points": 12_000_000, "batch": 4_000_000, "scene": 5,
         "limit": 50_000, "frame": "1080p"},
        # the viewer while a tile streams in: a frame after every batch
        {"name": "stream_tile_720p", "kind": "stream", "points": 2_000_003, "batch": 250_001, "scene": 1,
         "limit": 20_000, "frame": "720p"},
        # a frame of the streaming run: Analysis, 10% of the frontier refined, EDL
        {"name": "frame_refined_8k", "kind": "frame", "points": 12_000_000, "batch": 1_000_000, "scene": 2,
         "limit": 50_000, "frame": "8k"},
        # an orbiting camera on a finished tree
        {"name": "render_1080p", "kind": "render", "points": 8_000_000, "batch": 1_000_000, "scene": 2,
         "limit": 50_000, "frame": "1080p", "edl": True, "color_mode": 0, "point_size": 1},
        # the quality harness's ground truth: every point, no tree
        {"name": "flat_1080p", "kind": "flat", "points": 8_000_000, "scene": 2, "frame": "1080p", "edl": False},
        # the scorer's data collection on a finely split tree (many nodes)
        {"name": "analyze_fine_tree", "kind": "analyze", "points": 4_000_000, "batch": 500_000, "scene": 1,
         "limit": 1_000, "frame": "360p"},
        # colour filtering of a frame's queue
        {"name": "filter_colors", "kind": "filter", "points": 4_000_000, "batch": 1_000_000, "scene": 2,
         "limit": 20_000, "frame": "1080p", "budget": 64},
        # the scorer's training at its default minibatch
        {"name": "train_2048", "kind": "train", "samples": 2_048, "steps": 1},
        # the scorer's loss and gradient over the collected pairs, once per epoch
        {"name": "gradients_400k", "kind": "gradients", "samples": 400_003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("ingest", "ingest", "ingest_host", "stream", "frame", "render", "render", "flat", "analyze",
                       "filter", "train", "gradients"))
    if kind == "train":
        return {"kind": kind, "samples": _log_int(rng, 200, 16_384), "steps": rng.randint(1, 4)}
    if kind == "gradients":
        return {"kind": kind, "samples": _log_int(rng, 2_000, 400_000)}
    case = {"kind": kind, "scene": rng.choice((1, 2)), "frame": rng.choice(("360p", "720p", "1080p", "4k"))}
    if kind == "flat":
        return {**case, "points": _log_int(rng, 50_000, 8_000_000), "edl": rng.random() < 0.5}
    case["limit"] = rng.choice((20_000, 50_000))
    if kind == "ingest":
        case["points"] = _log_int(rng, 60_000, 12_000_000)
        case["batch"] = min(case["points"], _log_int(rng, 100_000, 1_000_000))
    elif kind == "ingest_host":
        case["scene"] = rng.choice((1, 2, 5))
        case["points"] = _log_int(rng, 200_000, 8_000_000)
        case["batch"] = min(case["points"], _log_int(rng, 200_000, 4_000_000))
    elif kind == "stream":
        case["points"] = _log_int(rng, 300_000, 2_000_000)
        case["batch"] = (case["points"] + 6) // rng.randint(3, 7)
    else:
        case["points"] = _log_int(rng, 300_000, 4_000_000)
        case["batch"] = min(case["points"], _log_int(rng, 200_000, 1_000_000))
    if kind == "render":
        case.update(edl=rng.random() < 0.5, color_mode=rng.choice((0, 0, 1, 2)), point_size=rng.choice((1, 1, 3)))
    if kind == "analyze":
        case["limit"] = rng.choice((1_000, 3_000, 20_000))
    if kind == "filter":
        case["budget"] = rng.choice((16, 64, 200))
    return case


# ------------------------------------------------------------------ inputs

def _cloud(case, seed):
    """The case's cloud as a POINT_DTYPE array, with its box. Scene 1 is a
    200 m tile scanned whole; 2 the first part of a 2 km scan at the
    benchmark's density; 5 the same scan with 5% uniform outliers."""
    n, gen = case["points"], 32_768  # points generated per thread and step
    over = {"seed": seed + 1, "batch_size": gen}
    if case["scene"] == 1:
        cfg = synth.config(1, num_points=n, **over)
    else:
        cfg = synth.config(2, outlier_fraction=0.05 if case["scene"] == 5 else 0.0, **over)
    pts = synth.generate(cfg, 0, n)
    return (pts, *synth.scene_box(cfg))


def _pixels(case):
    return PX[case["frame"]]


def _node_rows(case):
    """Rows that hold the tree of any seed: outputs have one shape per case."""
    return 512 + 16 * case["points"] // case["limit"]


def _fill(buffer, values):
    """The values in the first rows of a kept buffer (zeros after them: a state always has as many)."""
    buffer[:len(values)] = values
    return buffer


def _frame(case, box_min, box_max, seed, step=0, **more):
    """Frame `step` of a seeded orbit around the cloud."""
    yaw, pitch, radius = orbit_path(box_min, box_max, 16, seed=seed)[step % 16]
    f = make_frame(box_min, box_max, *_pixels(case), yaw=yaw, pitch=pitch, radius_scale=radius, **more)
    f.color_mode = case.get("color_mode", 0)
    return f


def _buffers(case):
    w, h = _pixels(case)
    return (torch.empty(w * h, dtype=torch.int64, device="cuda"),
            torch.empty(w * h, dtype=torch.int32, device="cuda"))


def _context(case, box_min, box_max, **more):
    slots = -(-case["points"] // case["batch"])
    # a split limit far below the default needs more grids than 48 B per point
    # pay for, and lists more new voxels per batch than the default holds
    fine = case["limit"] < 10_000
    more.update(store_capacity=4 << 30 if fine else 0, backlog_capacity=10_000_000 if fine else 0)
    ctx = Context(ring_slots=max(slots, 1), slot_capacity=case["batch"], max_points_per_node=case["limit"],
                  time_budget_ms=0.0, **more)
    ctx.allocate(case["points"], box_min, box_max)
    return ctx


def _ring(case, points):
    """The cloud as a device ring that holds all of it: batch b in slot b."""
    n, batch = case["points"], case["batch"]
    slots = -(-n // batch)
    ring = torch.zeros((slots, batch, 4), dtype=torch.float32, device="cuda")
    ring.view(-1, 4)[:n].copy_(torch.from_numpy(points.view(np.float32).reshape(n, 4)))
    return ring, [min(batch, n - b * batch) for b in range(slots)]


def _build(ctx, ring, sizes):
    consumed = 0
    while consumed < len(sizes):
        r = ctx.build(ring, sizes, len(sizes), len(sizes))
        if r.batches_this_call == 0:
            raise RuntimeError("the build made no progress")
        consumed = r.batches_consumed


def _scorer_params(seed):
    """Glorot-uniform weights, zero biases."""
    rng = np.random.default_rng(seed)
    parts = []
    for shape in SCORER_SIZES:
        a = math.sqrt(6.0 / sum(shape)) if len(shape) == 2 else 0.0
        parts.append(rng.uniform(-1.0, 1.0, int(np.prod(shape))) * a)
    return np.concatenate(parts).astype(np.float32)


def _scorer_data(case, seed):
    """Feature rows in the ranges Analysis logs, and targets of both outputs."""
    rng = np.random.default_rng(seed + 7)
    n = case["samples"]
    x = rng.random((n, capi.NUM_FEATURES), dtype=np.float32)
    x[:, 5:11] = rng.normal(0.0, 0.35, (n, 6)).astype(np.float32)
    t = np.empty((n, 2), dtype=np.float32)
    t[:, 0] = rng.normal(0.0, 1.0, n) * (0.2 + x[:, 15])
    t[:, 1] = rng.random(n) < 0.3 + 0.4 * x[:, 15] / 2
    return x, t


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("train", "gradients"):
        x, t = _scorer_data(case, seed)
        s["x"], s["t"] = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
        ctx = Context(slot_capacity=65_536, max_nodes=20_000)
        ctx.allocate(65_536, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0))
        ctx.mlp_set_params(_scorer_params(seed))
        s["ctx"] = ctx
        return s
    pts, lo, hi = _cloud(case, seed)
    if kind in ("ingest", "ingest_host", "stream"):
        s["sums"] = np.zeros((_node_rows(case), ACCUM_DTYPE.itemsize // 8), dtype=np.int64)
    s["fb"], s["rgba"] = _buffers(case)
    s["frame"] = _frame(case, lo, hi, seed, edl=case.get("edl", True), point_size=case.get("point_size", 1))
    if kind == "flat":
        s["points"] = torch.from_numpy(pts.view(np.float32).reshape(-1, 4)).cuda()
        s["ctx"] = Context(pipeline=capi.RB_PIPELINE_FLAT)
        s["ctx"].allocate(len(pts), lo, hi)
        return s
    if kind == "ingest_host":
        s["host"] = torch.from_numpy(pts.view(np.float32).reshape(-1, 4)).pin_memory()
        s["ctx"] = _context(case, lo, hi, max_batches_per_build=5)
        return s
    s["queue"] = np.zeros(16_384, dtype=np.int32)
    ring, sizes = _ring(case, pts)
    s["ctx"] = ctx = _context(case, lo, hi, max_batches_per_build=1 if kind == "stream" else 20)
    if kind in ("ingest", "stream"):
        s["ring"], s["sizes"] = ring, sizes
        s["mask"] = torch.zeros(ctx.cfg.max_nodes, dtype=torch.uint8, device="cuda")
        s["frames"] = [_frame(case, lo, hi, seed, step=k, edl=True) for k in range(len(sizes))]
        torch.cuda.synchronize()
        return s
    torch.cuda.synchronize()
    _build(ctx, ring, sizes)
    if kind == "frame":
        s["mask"] = torch.zeros(ctx.cfg.max_nodes, dtype=torch.uint8, device="cuda")
    elif kind == "analyze":
        ctx.mlp_set_params(_scorer_params(seed))
        rows = _node_rows(case)
        s["features"] = np.zeros((rows, capi.NUM_FEATURES), dtype=np.float32)
        s["analysis"] = {f: np.zeros((rows, *t.shape), np.float32 if t.base.kind == "f" else np.int64)
                         for f, (t, _) in ANALYSIS_DTYPE.fields.items() if f != "pad"}
    elif kind == "filter":
        ctx.analyze(s["frame"], frontier_only=False)
    return s


# ------------------------------------------------------------------ the pass

STATS = ("num_points", "num_voxels", "num_nodes", "num_inner", "num_leaves", "max_depth", "num_chunks_points",
         "num_chunks_voxels", "num_allocated_chunks", "chunk_pool_size", "persistent_offset", "dropped_points",
         "nodes_split", "spilled_points", "num_grids", "overflow_flags")


def _tree_outputs(s):
    """What the harness dumps after a build: the statistics, the exact sums of every node, the frame."""
    ctx = s["ctx"]
    st = ctx.stats()
    return {"stats": np.array([getattr(st, f) for f in STATS], dtype=np.int64),
            "sums": _fill(s["sums"], ctx.accums().view(np.int64).reshape(-1, s["sums"].shape[1])), "fb": s["fb"], "rgba": s["rgba"]}


def run(s):
    kind, ctx = s["kind"], s["ctx"]
    if kind == "ingest":
        ctx.reset()
        _build(ctx, s["ring"], s["sizes"])
        ctx.render(s["frame"], s["fb"], s["rgba"])
        return _tree_outputs(s)
    if kind == "ingest_host":
        ctx.reset()
        ctx.ingest_host(s["host"], s["case"]["batch"])
        ctx.render(s["frame"], s["fb"], s["rgba"])
        return _tree_outputs(s)
    if kind == "stream":
        ctx.reset()
        for k, frame in enumerate(s["frames"]):
            ctx.build(s["ring"], s["sizes"], k + 1, len(s["sizes"]))
            a = ctx.analyze(frame, closure_margin=2)
            ctx.refine(math.ceil(0.1 * a.eligible), s["mask"])
            ctx.render(frame, s["fb"], s["rgba"], force_large=s["mask"])
        return _tree_outputs(s)
    if kind == "frame":
        a = ctx.analyze(s["frame"], queue_capacity=16_384)
        ctx.refine(math.ceil(0.1 * a.eligible), s["mask"])
        ctx.render(s["frame"], s["fb"], s["rgba"], force_large=s["mask"])
        return {"queue": _fill(s["queue"], ctx.queue()), "fb": s["fb"], "rgba": s["rgba"]}
    if kind == "render":
        ctx.render(s["frame"], s["fb"], s["rgba"])
        return {"fb": s["fb"], "rgba": s["rgba"]}
    if kind == "flat":
        ctx.render_flat(s["frame"], s["points"], s["fb"], s["rgba"])
        return {"fb": s["fb"], "rgba": s["rgba"]}
    if kind == "analyze":
        ctx.analyze(s["frame"], closure_margin=2, queue_capacity=16_384, score_mode=capi.RB_SCORE_LEARNED)
        a = ctx.analysis()
        return {"queue": _fill(s["queue"], ctx.queue()), "features": _fill(s["features"], ctx.features()),
                **{f: _fill(v, a[f]) for f, v in s["analysis"].items()}}
    if kind == "filter":
        r = ctx.refine_colors(s["case"]["budget"])
        ctx.render(s["frame"], s["fb"], s["rgba"])
        return {"counts": np.array([r.nodes_filtered, r.voxels_filtered, r.points_visited], dtype=np.int64),
                "fb": s["fb"], "rgba": s["rgba"]}
    if kind == "train":
        for _ in range(s["case"]["steps"]):
            loss = ctx.mlp_train_step(s["x"], s["t"], 3e-3, want_loss=True)
        return {"params": ctx.mlp_params(), "loss": loss}
    grad, loss = ctx.mlp_gradients(s["x"], s["t"])
    return {"grad": grad, "loss": loss}


# ------------------------------------------------------------------ the least a pass costs

def work(case):
    """Bytes read and written once, and the scorer's multiply-adds."""
    kind = case["kind"]
    if kind in ("train", "gradients"):
        n = case["samples"] * case.get("steps", 1)
        return {"bytes": n * 4 * (capi.NUM_FEATURES + 2) + 4 * capi.MLP_NUM_PARAMS,
                "flops": 3 * 2 * (16 * 64 + 64 * 64 + 64 * 2) * n}
    w, h = _pixels(case)
    n, px = case["points"], w * h
    frame = px * (8 + 4)                     # the packed framebuffer and its colours
    drawn = 16 * min(n, 3 * px // 2)         # about 1.5 samples a pixel at the default budget
    nodes = 8 * n // case.get("limit", n)    # inner, empty and filled nodes per full leaf
    if kind == "flat":
        return {"bytes": 16 * n + frame, "flops": 0}
    if kind in ("ingest", "ingest_host"):
        return {"bytes": n * (16 + 20 + 5) + frame + drawn, "flops": 0}  # a point, its copy and index, 0.3 voxels
    if kind == "stream":
        return {"bytes": n * (16 + 20 + 5) + -(-n // case["batch"]) * (frame + drawn), "flops": 0}
    if kind == "analyze":
        return {"bytes": nodes * (184 + 64 + 64), "flops": 2 * (16 * 64 + 64 * 64 + 64 * 2) * nodes}
    if kind == "filter":
        return {"bytes": 16 * n // 4 + frame + drawn, "flops": 0}  # the points below a part of the queue
    return {"bytes": frame + drawn + (nodes * 184 if kind == "frame" else 0), "flops": 0}


# ------------------------------------------------------------------ 64-bit values

def _exact_scorer(case, seed):
    """The scorer in float64 torch: parameters after the steps, or the gradient, and the loss."""
    x, t = (torch.from_numpy(v).double() for v in _scorer_data(case, seed))
    flat = torch.from_numpy(_scorer_params(seed)).double().requires_grad_()

    def loss_of():
        parts, at = [], 0
        for shape in SCORER_SIZES:
            k = int(np.prod(shape))
            parts.append(flat[at:at + k].view(shape))
            at += k
        w1, b1, w2, b2, w3, b3 = parts
        gelu = lambda v: torch.nn.functional.gelu(v, approximate="tanh")  # noqa: E731
        y = gelu(gelu(x @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
        bce = torch.nn.functional.binary_cross_entropy_with_logits(y[:, 1], t[:, 1])
        return ((y[:, 0] - t[:, 0]) ** 2).mean() + bce

    if case["kind"] == "gradients":
        loss = loss_of()
        (grad,) = torch.autograd.grad(loss, flat)
        return {"grad": grad, "loss": float(loss.detach())}
    adam = torch.optim.Adam([flat], lr=3e-3)
    for _ in range(case["steps"]):
        adam.zero_grad()
        loss = loss_of()
        loss.backward()
        adam.step()
    return {"params": flat.detach(), "loss": float(loss.detach())}


def _spread3(v):
    """20-bit integers with two zero bits between their bits."""
    v = v.astype(np.uint64)
    for shift, mask in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F),
                        (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        v = (v | (v << np.uint64(shift))) & np.uint64(mask)
    return v


def _exact_tree(case, pts, lo, hi):
    """The octree the batches make, by counting: per node (in the order the
    splits number them) its level, and its points' range in Morton order."""
    size = np.float32(max(float(h - l) for l, h in zip(lo, hi)))
    cells = [((np.float32(2 ** 20) * (pts[a] - np.float32(lo[k]))) / size).astype(np.uint32)
             for k, a in enumerate("xyz")]
    code = (_spread3(cells[0]) << np.uint64(2)) | (_spread3(cells[1]) << np.uint64(1)) | _spread3(cells[2])
    level, prefix, leaves = [0], [0], [0]
    seen = np.empty(0, dtype=np.uint64)
    for first in range(0, len(pts), case["batch"]):
        seen = np.sort(np.concatenate([seen, code[first:first + case["batch"]]]), kind="stable")

        def count(ids):
            shift = np.array([60 - 3 * level[i] for i in ids], dtype=np.uint64)
            p = np.array([prefix[i] for i in ids], dtype=np.uint64)
            return np.searchsorted(seen, (p + np.uint64(1)) << shift) - np.searchsorted(seen, p << shift)

        todo = leaves
        while todo:
            over = [i for i, c in zip(todo, count(todo)) if c > case["limit"] and level[i] < 20]
            gone, todo = set(over), []
            for i in over:
                todo += range(len(level), len(level) + 8)
                level += [level[i] + 1] * 8
                prefix += range(8 * prefix[i], 8 * prefix[i] + 8)
            leaves = [i for i in leaves if i not in gone] + todo
    order = np.argsort(code, kind="stable")
    shift = np.array([60 - 3 * v for v in level], dtype=np.uint64)
    p = np.array(prefix, dtype=np.uint64)
    a, b = np.searchsorted(seen, p << shift), np.searchsorted(seen, (p + np.uint64(1)) << shift)
    xyz = np.stack([pts[k][order].astype(np.float64) - float(lo[i]) for i, k in enumerate("xyz")], 1) / float(size)
    return np.array(level), a, b, xyz


def _exact_analysis(case, seed):
    """Eigenvalues of every node's points, descending in units of its size squared, and what follows from them."""
    pts, lo, hi = _cloud(case, seed)
    level, a, b, xyz = _exact_tree(case, pts, lo, hi)
    cov = np.zeros((len(level), 3, 3))
    for i in np.nonzero(b - a >= 3)[0]:
        d = xyz[a[i]:b[i]] * 2.0 ** level[i]
        d = d - d.mean(0)
        cov[i] = d.T @ d / len(d)
    eig = np.maximum(np.linalg.eigvalsh(cov)[:, ::-1], 0.0)
    total = eig.sum(1)
    sv = np.divide(eig[:, 2], total, out=np.zeros_like(total), where=total > 0)
    planarity = np.divide(eig[:, 1] - eig[:, 2], eig[:, 0], out=np.zeros_like(total), where=eig[:, 0] > 0)
    out = {"eig": eig, "surface_variation": sv, "planarity": planarity}
    return {k: _fill(np.zeros((_node_rows(case), *v.shape[1:])), v) for k, v in out.items()}


def exact(case, seed):
    """The floating outputs in 64 bits: the scorer's, and Analysis's eigenvalues
    and what follows from them (framebuffers, sums and counts are whole numbers)."""
    if case["kind"] in ("train", "gradients"):
        return _exact_scorer(case, seed)
    if case["kind"] == "analyze":
        return _exact_analysis(case, seed)
    return None
