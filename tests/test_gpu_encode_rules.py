"""The encoder either side of each rule that picks its kernel: few points, long
records, and record lengths that fill the ring, against the host encoder."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import synth
from compute_rasterizer_gb300._lib import ptr
from test_gpu_tiles import header, make_records, on_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bpp", [(1, 26), (2_047, 26), (2_048, 34), (2_049, 26), (2_049, 34),
                                   (2_048, 300), (2_049, 300), (30_001, 28), (30_001, 29),
                                   (30_001, 30), (30_001, 139), (30_001, 140), (30_001, 141),
                                   (152 * 10_240 + 1, 30)])
@pytest.mark.parametrize("step", [1, 1024])
def test_encoder_rules(ctx, n, bpp, step):
    rng = np.random.default_rng(n + bpp)
    # step 1,024: ranges with a large power of two, whose points lie on cell borders
    xyz = rng.integers(-2 ** 9, 2 ** 9, (n, 3)) * step + 3
    rec = make_records(xyz, bpp, n)
    hdr = header(n, bpp, xyz)
    want = synth.encode_las(rec, n, hdr, bytes_per_point=bpp)
    cloud = ctx.cloud(n, len(want[0]), 1)
    d = cloud.device_pointers()
    buf, at = on_device(rec, 0)
    v = [np.ascontiguousarray(x[:], np.float64) for x in (hdr.scale, hdr.offset, hdr.min)]
    ctx.check(ctx.lib.cr_encode_las_device(ctx.handle, at, n, bpp, 2, *(ptr(a) for a in v), 0, 0,
                                           d["batches"], d["low"], d["med"], d["hig"], d["rgba"],
                                           None), "encode")
    ctx.sync()
    assert np.array_equal(cloud.read(0).view(np.uint8), want[0].view(np.uint8))
    for which, arr in zip((L.STREAM_LOW, L.STREAM_MED, L.STREAM_HIG, L.STREAM_RGBA), want[1:]):
        assert np.array_equal(cloud.read(which), arr), which
    cloud.close()
