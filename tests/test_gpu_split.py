"""The unit split of the batched and multi-view kernels (whole batches first, the
last item per CTA in parts): item counts around every switch of the rule,
against the oracle, bit for bit."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import default_params, make_view
from compute_rasterizer_gb300.multiview import MultiView
from helpers import QUIRKS, cameras, encoded, first_diff, gpu_raw, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu

BATCHES = 310


@pytest.fixture(scope="module")
def cloud_310(ctx):
    n = (BATCHES - 1) * L.POINTS_PER_BATCH + 6_001  # the last batch is partial
    cl = encoded(n=n, extent=800.0, seed=23)
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"],
                                  cl["box_min"])
    yield cl, cloud
    cloud.close()


# With one CTA per SM (152): 20 parts below 31 items, 10 below 61, 5 from there,
# whole items from 153; 153 with two CTAs per SM is again below two parts a CTA.
@pytest.mark.parametrize("block", [128, 256, 512])
@pytest.mark.parametrize("items,ctas", [(1, 1), (30, 1), (31, 1), (60, 1), (61, 1), (152, 1),
                                        (153, 1), (153, 2), (310, 1)])
def test_item_counts(ctx, cloud_310, items, ctas, block):
    cl, cloud = cloud_310
    points = min(cl["n"], items * L.POINTS_PER_BATCH)
    cloud.set_loaded(points, items)
    cam = cameras(cl)["far"]
    try:
        fb, _ = gpu_raw(ctx, cloud, cam, L.METHOD_LOOP_LAS, L.PAYLOAD_INDEX, culling=0,
                        block_threads=block, ctas_per_sm=ctas)
        fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[L.METHOD_LOOP_LAS], culling=0)
        want = O.raster_batched(fr, cl["batches"][:items], points, cl["lo"], cl["md"], cl["hi"],
                                cl["rgba"])
        got = fb.read(L.FB_WORDS)
        assert np.array_equal(got, want), first_diff(got, want)
        fb.close()
        fb, _ = gpu_raw(ctx, cloud, cam, L.METHOD_LOOP_LAS_HQS, culling=0, block_threads=block,
                        ctas_per_sm=ctas)
        fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[L.METHOD_LOOP_LAS_HQS], culling=0)
        depth, accum, _ = O.hqs(fr, cl["batches"][:items], points, cl["lo"], cl["md"], cl["hi"],
                                cl["rgba"])
        assert np.array_equal(fb.read(L.FB_DEPTH), depth)
        assert np.array_equal(fb.read(L.FB_ACCUM), accum)
        fb.close()
    finally:
        cloud.set_loaded()


# Two views per group: an item per batch and group.  The third view makes a
# second group of one view, so counts are twice the batches.
@pytest.mark.parametrize("block", [64, 128, 256])
@pytest.mark.parametrize("batches", [1, 15, 16, 30, 31, 76, 77, 310])
def test_multiview_item_counts(ctx, cloud_310, batches, block):
    cl, cloud = cloud_310
    points = min(cl["n"], batches * L.POINTS_PER_BATCH)
    cloud.set_loaded(points, batches)
    cams = [cameras(cl, 97, 61)[k] for k in ("far", "corner", "mid")]
    params = default_params(L.METHOD_LOOP_LAS, frustum_culling=0, views_per_group=2, ctas_per_sm=1,
                            block_threads=block, clear_after=0)
    try:
        mv = MultiView(ctx, cloud, [(c[2], c[3]) for c in cams], params)
        mv.set_views([make_view(*c) for c in cams])
        mv.clear()
        mv.render()
        ctx.sync()
        for i, cam in enumerate(cams):
            fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[L.METHOD_LOOP_LAS], culling=0)
            want = O.raster_batched(fr, cl["batches"][:batches], points, cl["lo"], cl["md"],
                                    cl["hi"], cl["rgba"])
            got = mv.read(i, L.FB_WORDS)
            assert np.array_equal(got, want), (i, first_diff(got, want))
            img = O.resolve_index(cam[2], cam[3], want, cl["rgba"])
            assert np.array_equal(mv.read(i, L.FB_IMAGE), img), i
        mv.close()
    finally:
        cloud.set_loaded()


# one grid for both lists up to 512 batches, two above; near the ground the cloud
# has 20- and 30-bit batches beside 10-bit ones
@pytest.mark.parametrize("batches", [511, 512, 513])
@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
def test_one_grid_or_two(ctx, batches, literal):
    n = (batches - 1) * L.POINTS_PER_BATCH + 77
    cl = encoded(n=n, extent=700.0, seed=batches)
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"],
                                  cl["box_min"])
    streams = (cl["lo"], cl["md"], cl["hi"], cl["rgba"])
    for name in ("near", "mid"):
        cam = cameras(cl, 321, 200)[name]
        for method, payload in ((L.METHOD_LOOP_LAS, L.PAYLOAD_INDEX), (L.METHOD_LOOP_LAS, L.PAYLOAD_COLOR)):
            fb, p = gpu_raw(ctx, cloud, cam, method, payload, quirks=QUIRKS[method] | literal)
            with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
                fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[method], payload)
                want = O.raster_batched(fr, cl["batches"], n, *streams)
            got = fb.read(L.FB_WORDS)
            assert np.array_equal(got, want), (name, payload, first_diff(got, want))
            per_level = list(ctx.frame_stats(cloud, p).points_per_level)
            assert per_level[1] > 0 and sum(per_level[2:]) > 0
            fb.close()
        q = QUIRKS[L.METHOD_LOOP_LAS_HQS]
        fb, _ = gpu_raw(ctx, cloud, cam, L.METHOD_LOOP_LAS_HQS, quirks=q | literal)
        with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
            fr = oracle_frame(cam, cl["box_min"][None], q)
            depth, accum, _ = O.hqs(fr, cl["batches"], n, *streams)
        assert np.array_equal(fb.read(L.FB_DEPTH), depth)
        assert np.array_equal(fb.read(L.FB_ACCUM), accum)
        fb.close()
    cloud.close()
