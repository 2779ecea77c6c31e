"""The plain early-z raster with and without the depth read in front of its atomics
(a rule on the points per pixel), at point counts that leave partial tiles, against
the oracle."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import default_params, make_view, synth
from helpers import first_diff
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# 1,024 points per CTA step; the read starts at 6,000,000 points and 5 per pixel
@pytest.mark.parametrize("n,w,h", [(1, 64, 48), (1023, 64, 48), (1025, 640, 360), (5_999_999, 320, 200),
                                   (6_000_000, 320, 200), (6_000_001, 1200, 1000),
                                   (6_000_001, 1200, 1001)])
@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
def test_early_z(ctx, n, w, h, literal):
    v = synth.uniform_vertices_host(n % 97, n, 100.0)
    v["color"] &= 3  # equal depths with equal and different colors
    v["x"][n // 2:] = v["x"][:n - n // 2]
    v["y"][n // 2:] = v["y"][:n - n // 2]
    v["z"][n // 2:] = v["z"][:n - n // 2]
    cloud = ctx.plain_cloud(v)
    view = synth.look_at([150.0, 150.0, 150.0], [50.0, 50.0, 50.0], [0.0, 0.0, 1.0])
    proj = synth.perspective(60.0, w / h, 0.1, 1000.0)
    fb = ctx.framebuffer(w, h)
    fb.clear(0xFFFFFFFFFFFFFFFF)
    p = default_params(L.METHOD_EARLYZ, resolve=0, clear_after=0, quirks=L.QUIRK_RESOLVE_TILES | literal)
    ctx.render(cloud, make_view(view, proj, w, h), p, fb)
    with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
        want, _, _ = O.plain(view, proj, w, h, v)
    got = fb.read(L.FB_WORDS)
    assert np.array_equal(got, want), first_diff(got, want)
    fb.close()
    cloud.close()
