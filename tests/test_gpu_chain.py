"""The frame's launch chain: the counters a resolve leaves for the next frame,
frames without one between, graph replays between eager frames, and the GPU's
per-file records at the small and the large parameter chunk."""
import numpy as np
import pytest
import torch

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import default_params, make_view
from helpers import QUIRKS, cameras, encoded, many_file_cameras, many_file_cloud, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def frame_words(cl, cam, method=L.METHOD_LOOP_LAS):
    fr = oracle_frame(cam, cl["box_min"][None], QUIRKS[method])
    return O.raster_batched(fr, cl["batches"], cl["n"], cl["lo"], cl["md"], cl["hi"], cl["rgba"])


def test_counters_across_frames(ctx):
    cl = encoded(n=41_000, extent=120.0, seed=5)
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"],
                                  cl["box_min"])
    cams = cameras(cl, 161, 121)
    fb = ctx.framebuffer(161, 121)
    st = torch.cuda.Stream()
    sh = st.cuda_stream
    graphs = {}

    def params(resolve):
        return default_params(L.METHOD_LOOP_LAS, resolve=resolve, clear_after=0)

    def check(cam, resolve, visible):
        want = frame_words(cl, cams[cam])
        st.synchronize()
        assert np.array_equal(fb.read(L.FB_WORDS, sh), want), (cam, resolve)
        if resolve:
            assert np.array_equal(fb.read(L.FB_IMAGE, sh), O.resolve_index(161, 121, want, cl["rgba"]))
        if visible:
            assert ctx.frame_stats(cloud, params(resolve)).batches_visible > 0

    def eager(cam, resolve):
        fb.clear(stream=sh)
        ctx.render(cloud, make_view(*cams[cam]), params(resolve), fb, sh)
        check(cam, resolve, True)

    def replay(cam, resolve):
        g = graphs[cam, resolve]
        fb.clear(stream=sh)
        with torch.cuda.stream(st):
            g.replay()
        check(cam, resolve, False)

    for cam, resolve in (("far", 1), ("near", 1), ("mid", 0), ("far", 0), ("corner", 1), ("near", 1)):
        eager(cam, resolve)
    for cam, resolve in (("far", 1), ("mid", 0)):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            ctx.render(cloud, make_view(*cams[cam]), params(resolve), fb, sh)
        graphs[cam, resolve] = g
    for step in (eager, replay, replay, eager, eager, replay):
        for cam, resolve in graphs:
            step(cam, resolve)
    eager("near", 1)
    eager("corner", 1)
    fb.close()
    cloud.close()


# 64 files is the last count of the small parameter chunk
@pytest.mark.parametrize("nfiles", [9, 63, 64, 65])
@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
def test_file_records(ctx, nfiles, literal):
    cl = many_file_cloud(nfiles, seed=nfiles, extent=900.0, base=700, spread=99)
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"],
                                  cl["box_min"])
    for name, cam in many_file_cameras(cl, 160, 90).items():
        view, proj, w, h = cam
        fb = ctx.framebuffer(w, h)
        fb.clear()
        p = default_params(L.METHOD_LOOP_LAS, quirks=QUIRKS[L.METHOD_LOOP_LAS] | literal, resolve=0,
                           clear_after=0)
        ctx.render(cloud, make_view(view, proj, w, h), p, fb)
        with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
            fr = oracle_frame(cam, cl["box_min"], QUIRKS[L.METHOD_LOOP_LAS])
            want = O.raster_batched(fr, cl["batches"], cl["n"], cl["lo"], cl["md"], cl["hi"],
                                    cl["rgba"])
        assert np.array_equal(fb.read(L.FB_WORDS), want), name
        fb.close()
    cloud.close()
