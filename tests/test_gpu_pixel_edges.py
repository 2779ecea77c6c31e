"""Pixel coordinates where rounding decides: points whose (q * 0.5 + 0.5) * size is
just below a whole number and rounds to it.  A fused product and sum would give the
pixel before.  Every body against the oracle: masked pairs, whole batches inside the
view, 20-bit pairs and the multi-view kernel."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import default_params, make_view
from compute_rasterizer_gb300.multiview import MultiView
from helpers import QUIRKS, first_diff, gpu_raw, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu
W, H = 1917, 1079
CAM = (np.eye(4).reshape(16), np.eye(4).reshape(16), W, H)  # w = 1: x / w is x


def edge_coordinates(size):
    """x in [0, 1) whose pixel product lies below the whole number it rounds to."""
    k = np.arange(size // 2 + 1, size)
    g = (k / size).astype(np.float32)  # in [0.5, 1): 2 g - 1 and its way back are exact
    below = g.astype(np.float64) * size < k
    rounds = (g * np.float32(size)) == k.astype(np.float32)
    return (2.0 * g.astype(np.float64) - 1.0)[below & rounds].astype(np.float32)


def cloud_at_edges(per_batch, count, stretch=0.0):
    """Batches of `per_batch` points at one edge coordinate each; `stretch` widens
    the boxes in z, which raises the precision level."""
    xs, ys = edge_coordinates(W), edge_coordinates(H)
    assert len(xs) > 100 and len(ys) > 100
    assert ((xs * np.float32(0.5) + np.float32(0.5)) * np.float32(W) % 1 == 0).all()
    i = np.linspace(0, len(xs) - 1, count).astype(int)
    batches = np.zeros(count, dtype=L.BATCH_DTYPE)
    batches["min_x"] = batches["max_x"] = xs[i]
    batches["min_y"] = batches["max_y"] = ys[i % len(ys)]
    batches["max_z"] = stretch
    batches["num_points"] = per_batch
    batches["first_point"] = np.arange(count) * per_batch
    n = count * per_batch
    rng = np.random.default_rng(3)
    lo, md, hi, rgba = (rng.integers(0, 2 ** 30, n, dtype=np.uint32) for _ in range(4))
    return n, batches, lo, md, hi, rgba


# 0.9 units of z are a radius of 862 pixels: level 1
@pytest.mark.parametrize("per_batch,count,stretch", [(8, 600, 0.0), (7, 600, 0.0),
                                                     (L.POINTS_PER_BATCH, 40, 0.0), (8, 600, 0.9)])
@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
def test_frames(ctx, per_batch, count, stretch, literal):
    n, batches, *streams = cloud_at_edges(per_batch, count, stretch)
    cloud = ctx.cloud_from_arrays(batches, *streams, np.zeros(3))
    for payload in (L.PAYLOAD_INDEX, L.PAYLOAD_COLOR):
        q = QUIRKS[L.METHOD_LOOP_LAS]
        fb, p = gpu_raw(ctx, cloud, CAM, L.METHOD_LOOP_LAS, payload, quirks=q | literal)
        per_level = list(ctx.frame_stats(cloud, p).points_per_level)
        assert per_level[1 if stretch else 4] == n
        with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
            want = O.raster_batched(oracle_frame(CAM, np.zeros((1, 3)), q, payload), batches, n, *streams)
        got = fb.read(L.FB_WORDS)
        assert np.array_equal(got, want), first_diff(got, want)
        fb.close()
    cloud.close()


@pytest.mark.parametrize("per_batch,count,stretch", [(8, 600, 0.0), (L.POINTS_PER_BATCH, 40, 0.0),
                                                     (8, 600, 0.9)])
def test_plan(ctx, per_batch, count, stretch):
    n, batches, *streams = cloud_at_edges(per_batch, count, stretch)
    cloud = ctx.cloud_from_arrays(batches, *streams, np.zeros(3))
    plan = MultiView(ctx, cloud, [(W, H)] * 3, default_params(L.METHOD_LOOP_LAS, resolve=0, clear_after=0))
    plan.set_views([make_view(*CAM)] * 3)
    plan.clear()
    plan.render()
    ctx.sync()
    want = O.raster_batched(oracle_frame(CAM, np.zeros((1, 3)), QUIRKS[L.METHOD_LOOP_LAS]), batches, n,
                            *streams)
    for i in range(3):
        got = plan.read(i, L.FB_WORDS)
        assert np.array_equal(got, want), (i, first_diff(got, want))
    plan.close()
    cloud.close()
