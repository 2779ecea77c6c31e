"""The point bodies of the batched kernels (masks or none, pairs, 10/20/30 bit)
on one handmade batch whose points share pixels and depths, so every merge of a
lane's points has ties to break: against the oracle, bit for bit."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from helpers import QUIRKS, first_diff, gpu_raw, handmade_cloud, identity_cam, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# widths at which the identity view sees the box at precision level 4, 1 and 0
LEVELS = {4: (64, 32), 1: (1024, 32), 0: (8192, 8)}
# every point strictly inside the view, or on its edges and partly outside
BOXES = {"inside": ((-0.9, -0.9, 0.1), (0.9, 0.9, 0.9)), "edge": ((-1.0, -1.0, 0.0), (1.0, 1.0, 1.0)),
         "outside": ((-1.5, -0.5, 0.0), (1.0, 1.25, 1.0))}


def tied_cloud(count, pad, box, seed):
    """Runs of 1-6 equal points in steps of a coarse grid; colors repeat, so
    lanes meet equal pixels with equal and different payloads."""
    rng = np.random.default_rng(seed)
    cells = rng.integers(0, 1024, (count, 3)) & ~np.array([63, 127, 255])
    runs = np.repeat(np.arange(count), rng.integers(1, 7, count))[:count]
    colors = rng.integers(0, 4, count) * 0x00402010 + 1
    return handmade_cloud(cells[runs], colors, *box, pad_before=pad)


# a view whose w falls from point to point: the fourth row of the projection
# mixes x, y and z into w (column-major), so merges see many depths per pixel
W_VARIES = np.array([1, 0, 0, 0.25, 0, 1, 0, 0.125, 0, 0, 1, 0.5, 0, 0, 0, 2], np.float64)


@pytest.mark.parametrize("level", LEVELS)
@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("count,pad", [(10240, 0), (10240, 1), (10239, 4), (2049, 3), (5, 2)])
def test_bodies(ctx, level, box, count, pad):
    cl = tied_cloud(count, pad, BOXES[box], 31 * level + count + pad)
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"],
                                  cl["box_min"])
    w, h = LEVELS[level]
    streams = (cl["lo"], cl["md"], cl["hi"], cl["rgba"])
    for proj in (identity_cam()[1], W_VARIES):
        cam = (identity_cam()[0], proj, w, h)
        for literal, arith in ((0, O.ARITH_CONTRACT), (L.QUIRK_LITERAL_ARITH, O.ARITH_LITERAL)):
            for method, payload in ((L.METHOD_LOOP_LAS, L.PAYLOAD_INDEX),
                                    (L.METHOD_LOOP_LAS_PREFETCH, L.PAYLOAD_COLOR)):
                fb, _ = gpu_raw(ctx, cloud, cam, method, payload, quirks=QUIRKS[method] | literal,
                                culling=0)
                with O.arith(arith):
                    fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[method], payload, culling=0)
                    want = O.raster_batched(fr, cl["batches"], cl["n"], *streams)
                got = fb.read(L.FB_WORDS)
                assert np.array_equal(got, want), (method, literal, first_diff(got, want))
                fb.close()
            q = QUIRKS[L.METHOD_LOOP_LAS_HQS]
            fb, _ = gpu_raw(ctx, cloud, cam, L.METHOD_LOOP_LAS_HQS, quirks=q | literal, culling=0)
            with O.arith(arith):
                fr = oracle_frame(cam, cl["box_min"][None], q, culling=0)
                depth, accum, _ = O.hqs(fr, cl["batches"], cl["n"], *streams)
            assert np.array_equal(fb.read(L.FB_DEPTH), depth)
            assert np.array_equal(fb.read(L.FB_ACCUM), accum)
            fb.close()
    cloud.close()
