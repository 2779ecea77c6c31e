"""The frames, plans and cloud builds that this framework's users run, as timed cases.

A case is a dict of plain values.  `kind` says which path it takes:

  frame    Context.render of a LAS-derived cloud (loop_las, loop_las_prefetch,
           loop_las_hqs) from one or more camera poses, one framebuffer each,
           resolved and re-cleared as the methods' defaults do.  `order`
           "morton" is a cloud sorted as Sort_Frugal sorts it, "file" the
           points as a scanner wrote them; `files` > 1 is a mosaic of LAS
           tiles of uneven sizes, laid back to back.
  plain    Context.render of 16-byte points (early-z, dedup, early-z & reduce).
  nodes    Context.render of a Potree octree (loop_nodes).
  views    MultiView.render: many views of one cloud in one captured frame,
           every image copied to pinned host memory.
  serve    Server.replay of a burst of requests over resident clouds.
  build    cr_morton_sort_device + cr_encode_las_device of unsorted records.

Every output is whole numbers (images, framebuffer words, encoded streams).
"""
from __future__ import annotations

import ctypes as C
import math
import tempfile

import numpy as np
import torch

import compute_rasterizer_gb300 as cr
from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import potree, synth, workloads
from compute_rasterizer_gb300.multiview import MultiView
from compute_rasterizer_gb300.serve import Server

METHODS = {"loop_las": L.METHOD_LOOP_LAS, "loop_las_prefetch": L.METHOD_LOOP_LAS_PREFETCH,
           "loop_las_hqs": L.METHOD_LOOP_LAS_HQS, "early-z": L.METHOD_EARLYZ,
           "dedup": L.METHOD_DEDUP, "early-z & reduce": L.METHOD_EARLYZ_REDUCE}
RESOLUTIONS = [(256, 256), (512, 512), (641, 359), (1280, 720), (1366, 768), (1440, 1600),
               (1920, 1080), (2560, 1440), (3840, 2160)]


def _frame(points, width, height, **kw):
    c = dict(kind="frame", points=points, density=10.0, files=1, order="morton", method="loop_las",
             payload="index", literal=False, pose="zoom", poses=1, width=width, height=height)
    c.update(kw)
    return c


def listed():
    return [
        # a preview of one small scan: five batches, the frame is launches and latency
        dict(_frame(50_000, 512, 512), name="preview_50k"),
        # a mosaic of 24 LAS tiles of uneven, odd sizes (a survey block): batches
        # start at any word, the per-file records are computed on the GPU
        dict(_frame(15_000_017, 1920, 1080, files=24), name="mosaic_24_files"),
        # one scan in the order the scanner wrote it: each batch spans the whole
        # tile, so it is drawn with 20-bit coordinates
        dict(_frame(20_000_003, 1280, 720, order="file"), name="unsorted_20m"),
        # standing in the cloud on a 4K screen: few visible batches, near ones at 20 bit
        dict(_frame(40_000_000, 3840, 2160, pose="ground", density=40.0, payload="color",
                    method="loop_las_prefetch"), name="ground_4k"),
        # the flight over a 100 M point terrain: five poses, method defaults
        dict(_frame(100_000_000, 2560, 1440, pose="flight", poses=5, density=100.0),
             name="flight_100m"),
        # high-quality shading of a city-sized terrain: depth pass, colour pass, averages
        dict(_frame(300_000_000, 1920, 1080, method="loop_las_hqs"), name="hqs_300m"),
        # a billion points in one frame, the headline
        dict(_frame(1_000_000_000, 1920, 1080, payload="color"), name="frame_1b"),
        # the 16-byte path on points in no order
        dict(kind="plain", points=4_194_304, method="early-z", literal=False, width=1920,
             height=1080, name="plain_4m"),
        # a Potree octree, level-of-detail cut
        dict(kind="nodes", points=2_000_000, max_leaf=20_000, width=1920, height=1080,
             name="octree_2m"),
        # 16 headsets and 32 thumbnails over one cloud
        dict(kind="views", points=200_000_000, pairs=16, thumbs=32, payload="color",
             name="views_64"),
        # a burst of mixed requests at a frame server with three resident clouds
        dict(kind="serve", clouds=3, points=10_000_000, requests=40, name="serve_burst"),
        # making a drawable cloud of a survey's unsorted records
        dict(kind="build", points=40_000_000, name="build_40m"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame"] * 6 + ["plain", "nodes", "views", "serve", "build"])
    width, height = rng.choice(RESOLUTIONS)
    if kind == "frame":
        order = rng.choice(["morton"] * 4 + ["file"])
        c = _frame(_log(rng, 20_000, 60_000_000 if order == "file" else 500_000_000), width, height,
                   order=order, density=float(rng.choice([2, 10, 40, 100])),
                   method=rng.choice(["loop_las", "loop_las", "loop_las_prefetch", "loop_las_hqs"]),
                   payload=rng.choice(["index", "color"]), literal=rng.random() < 0.2,
                   pose=rng.choice(["zoom", "flight", "ground"]))
        c["poses"] = rng.choice([1, 1, 2, 3]) if c["pose"] == "flight" else 1
        if rng.random() < 0.3:
            c["files"] = rng.choice([2, 3, 7, 9, 17, 40])
            c["points"] = max(c["points"], 4_000 * c["files"])
        if c["method"] == "loop_las_hqs":
            c["payload"] = "index"
        return c
    if kind == "plain":
        return dict(kind=kind, points=_log(rng, 1_000, 64_000_000), literal=rng.random() < 0.2,
                    method=rng.choice(["early-z", "dedup", "early-z & reduce"]), width=width,
                    height=height)
    if kind == "nodes":
        return dict(kind=kind, points=_log(rng, 100_000, 3_000_000),
                    max_leaf=rng.choice([3_000, 10_000, 20_000, 50_000]), width=width, height=height)
    if kind == "views":
        return dict(kind=kind, points=_log(rng, 200_000, 200_000_000), pairs=rng.randint(1, 8),
                    thumbs=rng.randint(0, 16), payload=rng.choice(["index", "color"]))
    if kind == "serve":
        return dict(kind=kind, clouds=rng.randint(1, 3), points=_log(rng, 500_000, 10_000_000),
                    requests=rng.randint(8, 40))
    return dict(kind=kind, points=_log(rng, 10_000, 60_000_000))


# ---- inputs -------------------------------------------------------------------


class _Device:
    """A library-owned device buffer as an array torch can view."""

    def __init__(self, owner, address, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "version": 3,
                                         "strides": None, "data": (address, False)}


def _tensor(owner, address, count, typestr="<i4"):
    return torch.as_tensor(_Device(owner, address, count, typestr), device="cuda")


def _outputs(fb):
    """The image of a framebuffer and its words as the next frame finds them."""
    out = [_tensor(fb, fb.device_pointer(L.FB_IMAGE), fb.W * fb.H).view(fb.H, fb.W)]
    if fb.kind == L.FB_HQS:
        return out + [_tensor(fb, fb.device_pointer(L.FB_DEPTH), fb.words),
                      _tensor(fb, fb.device_pointer(L.FB_ACCUM), 2 * fb.words, "<i8")]
    return out + [_tensor(fb, fb.device_pointer(L.FB_WORDS), fb.words, "<i8")]


def _terrain(seed, extent, origin=(0.0, 0.0)):
    p = synth.synth_params(L.SYNTH_TERRAIN, extent, seed)
    p.origin[0], p.origin[1] = origin
    return p


def _records(ctx, params, n, sort):
    """LAS format-2 records on the device, Morton-sorted or as written, and their header."""
    rec = torch.empty(n * L.LAS_FORMAT2_BYTES, dtype=torch.uint8, device="cuda")
    hdr = L.LasHeader()
    ctx.check(ctx.lib.cr_synth_points_device(ctx.handle, C.byref(params), n, rec.data_ptr(),
                                             C.byref(hdr), None), "points")
    if sort:
        ctx.check(ctx.lib.cr_morton_sort_device(ctx.handle, rec.data_ptr(), n, L.LAS_FORMAT2_BYTES,
                                                C.byref(hdr), None), "sort")
    return rec, hdr


def _encode(ctx, rec, n, hdr, sparse, file_index, dst, batch_offset=0):
    v = [np.ascontiguousarray(x[:], np.float64) for x in (hdr.scale, hdr.offset, hdr.min)]
    ctx.check(ctx.lib.cr_encode_las_device(
        ctx.handle, rec.data_ptr(), n, L.LAS_FORMAT2_BYTES, 2, *(a.ctypes.data for a in v), sparse,
        file_index, dst["batches"] + 64 * batch_offset, *(dst[k] + 4 * sparse for k in
                                                          ("low", "med", "hig", "rgba")), None),
        "encode")


def _file_sizes(n, files):
    """Uneven, mostly odd shares of n points."""
    w = [1.0 + 0.8 * math.sin(2.3 * i + 0.7) for i in range(files)]
    sizes = [max(1000, int(n * x / sum(w))) | 1 for x in w]
    sizes[0] = max(1000, n - sum(sizes[1:]))
    return sizes


def _cloud(ctx, case, seed):
    """The case's cloud and its (box_min, box_max)."""
    n, files = case["points"], case["files"]
    extent = math.sqrt(n / case["density"])
    if files == 1 and case["order"] == "morton":
        cloud, hdr = synth.build_cloud_device(ctx, _terrain(seed, extent), n)
        ctx.sync()
        return cloud, np.array(hdr.min[:]), np.array(hdr.max[:])
    sizes = _file_sizes(n, files)
    side = math.ceil(math.sqrt(files))
    nbs = [int(ctx.lib.cr_num_batches(s)) for s in sizes]
    cloud = ctx.cloud(sum(sizes), sum(nbs), files)
    dst = cloud.device_pointers()
    mins, maxs, at, bat = [], [], 0, 0
    for i, s in enumerate(sizes):
        tile = extent / side
        p = _terrain(seed, tile, (tile * (i % side), tile * (i // side)))
        p.wavelength = extent / 4.0
        rec, hdr = _records(ctx, p, s, case["order"] == "morton")
        _encode(ctx, rec, s, hdr, at, i, dst, bat)
        ctx.sync()
        at, bat = at + s, bat + nbs[i]
        mins.append(hdr.min[:])
        maxs.append(hdr.max[:])
    cloud.set_files(np.array(mins))
    return cloud, np.min(mins, axis=0), np.max(maxs, axis=0)


def _poses(case, bmin, bmax, seed):
    w, h = case["width"], case["height"]
    if case["pose"] == "zoom":
        cams = [workloads.terrain_frame(bmin, bmax, w, h)]
    elif case["pose"] == "flight":
        cams = workloads.flight_path(bmin, bmax, max(2, case["poses"]), seed, w, h)[:case["poses"]]
    else:  # "ground": a few metres above the terrain, looking over it
        rng = np.random.default_rng(seed)
        target = bmin + (bmax - bmin) * np.array([rng.uniform(0.4, 0.6), rng.uniform(0.4, 0.6), 0.6])
        cams = [(synth.orbit_view(rng.uniform(-3.0, 3.0), -0.35, 25.0, target),
                 synth.perspective(60.0, w / h, 0.1, 200000.0), w, h)]
    return [cr.make_view(v, p, w, h) for v, p, w, h in cams]


def _params(case):
    p = cr.default_params(METHODS[case["method"]])
    if case.get("payload") == "color":
        p.payload = L.PAYLOAD_COLOR
    if case["literal"]:  # the shader source's own rounding, on top of the method's defaults
        p.quirks = {"loop_las": L.QUIRK_L0_X12,
                    "loop_las_prefetch": L.QUIRK_INCLUSIVE_END | L.QUIRK_DISPATCH_BY_POINTS
                    | L.QUIRK_UVEC4_BASE,
                    "loop_las_hqs": L.QUIRK_L0_X12 | L.QUIRK_INCLUSIVE_END
                    | L.QUIRK_DISPATCH_BY_POINTS}.get(case["method"], L.QUIRK_RESOLVE_TILES)
        p.quirks |= L.QUIRK_LITERAL_ARITH
    return p


def _prepare_frame(ctx, case, seed):
    cloud, bmin, bmax = _cloud(ctx, case, seed)
    hqs = case["method"] == "loop_las_hqs"
    views = _poses(case, bmin, bmax, seed)
    fbs = [ctx.framebuffer(v.width, v.height, L.FB_HQS if hqs else L.FB_U64) for v in views]
    for fb in fbs:
        fb.clear()
    return dict(ctx=ctx, cloud=cloud, views=views, fbs=fbs, params=_params(case),
                out=[t for fb in fbs for t in _outputs(fb)])


def _prepare_plain(ctx, case, seed):
    cloud = synth.uniform_cloud_device(ctx, seed, case["points"], 100.0)
    w, h = case["width"], case["height"]
    view = synth.look_at([150.0, 150.0, 150.0], [50.0, 50.0, 50.0], [0.0, 0.0, 1.0])
    fb = ctx.framebuffer(w, h)
    fb.clear(L.PLAIN_RECLEAR)
    return dict(ctx=ctx, cloud=cloud, fbs=[fb], params=_params(case), out=_outputs(fb),
                views=[cr.make_view(view, synth.perspective(60.0, w / h, 0.1, 1000.0), w, h)])


def _prepare_nodes(ctx, case, seed):
    n, w, h = case["points"], case["width"], case["height"]
    rec, hdr = _records(ctx, _terrain(seed, math.sqrt(n / 22.0)), n, True)
    host = rec.cpu().numpy()
    with tempfile.TemporaryDirectory(prefix="cr_octree_") as d:
        potree.write_octree(d, host, n, hdr.scale[:], hdr.offset[:], hdr.min[:], hdr.max[:],
                            max_leaf=case["max_leaf"], chunk_levels=2)
        octree = potree.open_octree(d)
        cloud = octree.load(ctx)
        octree.close()
    extent = np.array(hdr.max[:]) - np.array(hdr.min[:])
    view, proj, w, h = workloads.terrain_frame(np.zeros(3), extent, w, h)
    fb = ctx.framebuffer(w, h)
    fb.clear()
    return dict(ctx=ctx, cloud=cloud, views=[cr.make_view(view, proj, w, h)], fbs=[fb],
                params=cr.default_params(L.METHOD_LOOP_NODES), out=_outputs(fb))


def _pinned(words):
    return torch.empty(words, dtype=torch.int32, pin_memory=True)


def _prepare_views(ctx, case, seed):
    n = case["points"]
    boxes = max(1, n // 100_000)  # a fifth of the points on boxes standing on the terrain
    p = workloads.multiview_cloud_params(seed, math.sqrt(n / 10.0))
    p.num_boxes, p.points_per_box = boxes, 20_000
    cloud, hdr = synth.build_cloud_device(ctx, p, n)
    cams = workloads.multiview_64(np.array(hdr.min[:]), np.array(hdr.max[:]), seed)
    cams = cams[:2 * case["pairs"]] + cams[32:32 + case["thumbs"]]
    params = cr.default_params(L.METHOD_LOOP_LAS)
    if case["payload"] == "color":
        params.payload = L.PAYLOAD_COLOR
    stream = torch.cuda.Stream()
    plan = MultiView(ctx, cloud, [(w, h) for _, _, w, h in cams], params)
    plan.set_views([cr.make_view(v, q, w, h) for v, q, w, h in cams])
    plan.clear(stream=stream.cuda_stream)
    return dict(ctx=ctx, plan=plan, cloud=cloud, stream=stream,
                out=[_pinned(w * h) for _, _, w, h in cams])


def _prepare_serve(ctx, case, seed):
    clouds, boxes = [], []
    for i in range(case["clouds"]):
        n = case["points"] * (1, 2, 5)[i]
        cloud, hdr = synth.build_cloud_device(ctx, _terrain(seed + 100 + i, math.sqrt(n / 10.0)), n)
        clouds.append(cloud)
        boxes.append((np.array(hdr.min[:]), np.array(hdr.max[:])))
    server = Server(ctx, pool_bytes=2 << 30)
    for c in clouds:
        server.add_cloud(c)
    _, cams = workloads.serving_requests(boxes, case["requests"], 1e9)
    out = [_pinned(w * h) for *_, w, h in cams]
    reqs = [Server.request(c, cr.make_view(v, p, w, h), o.numpy().view(np.uint32), i)
            for i, ((c, v, p, w, h), o) in enumerate(zip(cams, out))]
    return dict(ctx=ctx, server=server, clouds=clouds, requests=reqs, out=out,
                arrival=np.zeros(len(reqs)))


def _prepare_build(ctx, case, seed):
    n = case["points"]
    rec, hdr = _records(ctx, _terrain(seed, math.sqrt(n / 10.0)), n, False)
    cloud = ctx.cloud(n, int(ctx.lib.cr_num_batches(n)), 1)
    d = cloud.device_pointers()
    return dict(ctx=ctx, n=n, records=rec, work=torch.empty_like(rec), hdr=hdr, cloud=cloud, dst=d,
                out=[_tensor(cloud, d[k], n) for k in ("low", "med", "hig", "rgba")]
                + [_tensor(cloud, d["batches"], 16 * cloud.nb)])


def prepare(case, seed):
    ctx = cr.Context(0)
    state = globals()["_prepare_" + case["kind"]](ctx, case, seed)
    state["kind"] = case["kind"]
    ctx.sync()
    return state


# ---- one pass -----------------------------------------------------------------


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind in ("frame", "plain", "nodes"):
        stream = torch.cuda.current_stream().cuda_stream
        for view, fb in zip(state["views"], state["fbs"]):
            ctx.render(state["cloud"], view, state["params"], fb, stream)
    elif kind == "views":
        plan, stream = state["plan"], state["stream"].cuda_stream
        plan.render(use_graph=True, stream=stream)
        for i, o in enumerate(state["out"]):
            ctx.check(ctx.lib.cr_mv_read(plan.handle, i, L.FB_IMAGE, o.data_ptr(), 4 * o.numel(),
                                         stream), "read")
    elif kind == "serve":
        done = state["server"].replay(state["requests"], state["arrival"])
        if not (done["status"] == L.OK).all():
            raise RuntimeError("a request failed")
    else:
        state["work"].copy_(state["records"])
        stream = torch.cuda.current_stream().cuda_stream
        ctx.check(ctx.lib.cr_morton_sort_device(ctx.handle, state["work"].data_ptr(), state["n"],
                                                L.LAS_FORMAT2_BYTES, C.byref(state["hdr"]), stream),
                  "sort")
        _encode(ctx, state["work"], state["n"], state["hdr"], 0, 0, state["dst"])
    return state["out"]


# ---- the work of one pass -------------------------------------------------------

# Share of the points in visible batches, over the poses of the kind.
VISIBLE = {"zoom": 0.96, "flight": 0.67, "ground": 0.21}
# Per drawn point: decode (6), projection (21), divide and pixel (10).
FLOPS_PER_POINT = 37


def work(case):
    kind, n = case["kind"], case["points"]
    if kind == "frame":
        drawn = n * VISIBLE[case["pose"]] * case["poses"]
        pixels = case["width"] * case["height"] * case["poses"]
        words = 1 if case["order"] == "morton" else 2
        if case["method"] == "loop_las_hqs" or case["payload"] == "color":
            words += 1
        return {"bytes": 4.0 * words * drawn + 64.0 * n / L.POINTS_PER_BATCH + 4.0 * pixels,
                "flops": FLOPS_PER_POINT * drawn}
    if kind == "plain":
        return {"bytes": 16.0 * n + 4.0 * case["width"] * case["height"], "flops": 31.0 * n}
    if kind == "nodes":
        return {"bytes": 4.0 * n + 4.0 * case["width"] * case["height"], "flops": FLOPS_PER_POINT * n}
    if kind == "views":
        pixels = 2 * case["pairs"] * 1440 * 1600 + case["thumbs"] * 512 * 512
        words = 2 if case["payload"] == "color" else 1
        share = 0.3 * (2 * case["pairs"] + case["thumbs"])  # of the cloud in a view, on average
        return {"bytes": 4.0 * words * n + 4.0 * pixels, "flops": FLOPS_PER_POINT * n * share}
    if kind == "serve":
        total = n * sum((1, 2, 5)[:case["clouds"]])
        pixels = case["requests"] * sum(w * h for w, h in workloads.SERVING_RESOLUTIONS) / 5
        return {"bytes": 8.0 * total + 4.0 * pixels,
                "flops": FLOPS_PER_POINT * 0.9 * case["requests"] * total / case["clouds"]}
    return {"bytes": (26.0 + 16.0) * n + 64.0 * n / L.POINTS_PER_BATCH, "flops": 40.0 * n}


def exact(case, seed):
    """None: the outputs are whole numbers (images, indices, encoded words), compared word for word."""
    return None
