"""cr_last_frame_stats counts the last cull that ran: with eager frames and graph
replays in any order, with and without a resolve, after a resolve that is refused,
and for a frame without batches."""
import numpy as np
import pytest
import torch

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import default_params, make_view
from compute_rasterizer_gb300.raster import CRError
from helpers import QUIRKS, cameras, encoded, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu
W, H = 161, 121


def visible_per_level(cl, cam):
    """Batches per precision level that the oracle's cull keeps."""
    fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[L.METHOD_LOOP_LAS])
    lib, counts = O.lib(), [0] * 5
    for b in cl["batches"]:
        lo = np.array([b["min_x"], b["min_y"], b["min_z"]], np.float32)
        hi = np.array([b["max_x"], b["max_y"], b["max_z"]], np.float32)
        if lib.or_intersects_frustum(fr.files[0].planes, O._p(lo), O._p(hi)):
            counts[lib.or_precision_level(fr, fr.files[0], O._p(lo), O._p(hi))] += 1
    return counts


@pytest.fixture(scope="module")
def scene():
    cl = encoded(n=210_000, extent=300.0, seed=5)
    cams = cameras(cl, W, H)
    want = {k: visible_per_level(cl, cams[k]) for k in ("far", "corner", "mid")}
    assert len({tuple(v) for v in want.values()}) == 3
    assert any(sum(v[:2]) for v in want.values())  # the back of the list too
    return cl, cams, want


@pytest.mark.parametrize("first,second", [(0, 1), (1, 0), (1, 1), (0, 0)])
def test_replay_after_an_eager_frame(ctx, scene, first, second):
    """A frame captured with resolve=`first`, one drawn with resolve=`second`, a replay."""
    cl, cams, want = scene
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"], cl["box_min"])
    fb = ctx.framebuffer(W, H)
    st = torch.cuda.Stream()

    def params(resolve):
        return default_params(L.METHOD_LOOP_LAS, resolve=resolve)

    def stats():
        st.synchronize()
        return list(ctx.frame_stats(cloud, params(0)).batches_per_level)

    def draw(cam, resolve):
        ctx.render(cloud, make_view(*cams[cam]), params(resolve), fb, st.cuda_stream)

    fb.clear(stream=st.cuda_stream)
    draw("far", 1)  # the scratch buffer is there, its counters zero
    assert stats() == want["far"]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        draw("corner", first)
    for _ in range(2):
        draw("mid", second)
        assert stats() == want["mid"]
        with torch.cuda.stream(st):
            g.replay()
        assert stats() == want["corner"]
    fb.close()
    cloud.close()


def test_eager_frames(ctx, scene):
    cl, cams, want = scene
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"], cl["box_min"])
    fb = ctx.framebuffer(W, H)
    fb.clear()
    for cam, resolve in (("far", 1), ("mid", 1), ("corner", 0), ("mid", 0), ("far", 1)):
        p = default_params(L.METHOD_LOOP_LAS, resolve=resolve)
        ctx.render(cloud, make_view(*cams[cam]), p, fb)
        assert list(ctx.frame_stats(cloud, p).batches_per_level) == want[cam], (cam, resolve)
    # nothing loaded: no cull runs, nothing is visible
    cloud.set_loaded(0, 0)
    for resolve in (1, 0):
        p = default_params(L.METHOD_LOOP_LAS, resolve=resolve)
        ctx.render(cloud, make_view(*cams["far"]), p, fb)
        assert ctx.frame_stats(cloud, p).batches_visible == 0
    fb.close()
    cloud.close()


def test_refused_resolve(ctx, scene):
    """The tiled resolve refuses the color payload after the raster is enqueued; the
    counts are that frame's, not those of the larger frame before it."""
    cl, cams, _ = scene
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"], cl["box_min"])
    fb = ctx.framebuffer(W, H)
    fb.clear()
    ctx.render(cloud, make_view(*cams["mid"]), default_params(L.METHOD_LOOP_LAS), fb)
    assert ctx.frame_stats(cloud, default_params(L.METHOD_LOOP_LAS)).batches_visible > 3
    cloud.set_loaded(3 * L.POINTS_PER_BATCH, 3)
    p = default_params(L.METHOD_LOOP_LAS, payload=L.PAYLOAD_COLOR, frustum_culling=0,
                       quirks=L.QUIRK_RESOLVE_TILES)
    with pytest.raises(CRError):
        ctx.render(cloud, make_view(*cams["far"]), p, fb)
    assert ctx.frame_stats(cloud, p).batches_visible == 3
    cloud.close()
    fb.close()
