"""A view whose transform overflows float for one column, on a cloud that is flat
there: x / w is a NaN for every point, none is drawn, and no batch may take the
body that trusts the inside proof."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import default_params, make_view, synth
from compute_rasterizer_gb300.multiview import MultiView
from helpers import QUIRKS, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu
W, H = 256, 192


def flat_cloud(n=20_480):
    """Points on the plane x = 0, in two whole batches."""
    rng = np.random.default_rng(11)
    xyz = rng.integers(0, 20_000, (n, 3)).astype("<i4")
    xyz[:, 0] = 0
    rec = np.zeros((n, 26), np.uint8)
    rec[:, :12] = xyz.view(np.uint8).reshape(n, 12)
    rec[:, 20:26] = 200
    hdr = L.LasHeader()
    hdr.num_points, hdr.point_format, hdr.bytes_per_point = n, 2, 26
    hdr.scale[:], hdr.offset[:] = [0.001] * 3, [0.0] * 3
    hdr.min[:], hdr.max[:] = [0.0, 0.0, 0.0], [20.0, 20.0, 20.0]
    return (n, *synth.encode_las(rec.reshape(-1), n, hdr, bytes_per_point=26))


def overflowing_camera():
    """Looks down at the cloud; proj * view overflows float in column 0 only."""
    view = np.eye(4).reshape(16)
    view[0] = 3.2e38
    view[13], view[14] = -10.0, -100.0
    proj = synth.perspective(60.0, W / H, 0.1, 1000.0)
    t0 = np.float64(proj[0]) * view[0]
    assert np.isfinite(np.float32(view[0])) and t0 > float(np.finfo(np.float32).max)
    return view, proj, W, H


@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
@pytest.mark.parametrize("method", [L.METHOD_LOOP_LAS, L.METHOD_LOOP_LAS_HQS])
def test_nothing_drawn(ctx, method, literal):
    n, batches, lo, md, hi, rgba = flat_cloud()
    cloud = ctx.cloud_from_arrays(batches, lo, md, hi, rgba, np.zeros(3))
    cam = overflowing_camera()
    hqs = method == L.METHOD_LOOP_LAS_HQS
    fb = ctx.framebuffer(W, H, L.FB_HQS if hqs else L.FB_U64)
    fb.clear(0xFF800000 if hqs else L.DEFAULT_CLEAR)
    p = default_params(method, quirks=QUIRKS[method] | literal, resolve=0, clear_after=0)
    ctx.render(cloud, make_view(*cam), p, fb)
    ctx.sync()
    # 10-bit batches that are not culled, so the proof was asked for
    assert sum(ctx.frame_stats(cloud, p).batches_per_level[2:]) == 2
    with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
        fr = oracle_frame(cam, np.zeros((1, 3)), QUIRKS[method])
        if hqs:
            depth, accum, _ = O.hqs(fr, batches, n, lo, md, hi, rgba)
            assert np.array_equal(fb.read(L.FB_DEPTH), depth)
            assert np.array_equal(fb.read(L.FB_ACCUM), accum)
            assert not accum.any()
        else:
            want = O.raster_batched(fr, batches, n, lo, md, hi, rgba)
            assert np.array_equal(fb.read(L.FB_WORDS), want)
            assert (want == np.uint64(L.DEFAULT_CLEAR)).all()
    fb.close()
    cloud.close()


def test_nothing_drawn_by_a_plan(ctx):
    n, batches, lo, md, hi, rgba = flat_cloud()
    cloud = ctx.cloud_from_arrays(batches, lo, md, hi, rgba, np.zeros(3))
    cam = overflowing_camera()
    plan = MultiView(ctx, cloud, [(W, H)] * 2,
                     default_params(L.METHOD_LOOP_LAS, resolve=0, clear_after=0))
    plan.set_views([make_view(*cam)] * 2)
    plan.clear()
    plan.render()
    ctx.sync()
    for i in range(2):
        assert (plan.read(i, L.FB_WORDS) == np.uint64(L.DEFAULT_CLEAR)).all()
    plan.close()
    cloud.close()
