"""The tiled record kernels: the encoder's shapes (by batches per SM) and its byte
path, odd record lengths and unaligned records, against the host encoder; the
Morton sort's short radix keys with runs left to the run sort, runs too long for
it, and unaligned records, against the host sort."""
import ctypes as C

import numpy as np
import pytest
import torch

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300 import synth
from compute_rasterizer_gb300._lib import ptr

pytestmark = pytest.mark.gpu


def header(n, bpp, xyz, scale=0.001):
    hdr = L.LasHeader()
    hdr.num_points, hdr.point_format, hdr.bytes_per_point = n, 2, bpp
    hdr.scale[:], hdr.offset[:] = [scale] * 3, [0.0] * 3
    hdr.min[:], hdr.max[:] = list(xyz.min(0) * scale), list(xyz.max(0) * scale)
    return hdr


def make_records(xyz, bpp, seed):
    n = len(xyz)
    rec = np.random.default_rng(seed).integers(0, 256, (n, bpp), dtype=np.uint8)
    rec[:, :12] = np.ascontiguousarray(xyz, "<i4").view(np.uint8).reshape(n, 12)
    return rec.reshape(-1)


def on_device(rec, shift):
    """The records on the device, `shift` bytes past a 256-byte boundary."""
    buf = torch.zeros(rec.size + 256, dtype=torch.uint8, device="cuda")
    buf[shift:shift + rec.size] = torch.from_numpy(rec).cuda()
    return buf, buf.data_ptr() + shift


# 152 SMs: one, two and more batches per SM; 20,000 bytes: longer than a tile holds
@pytest.mark.parametrize("n,bpp,shift", [(1, 26, 0), (10_241, 26, 0), (152 * 10240, 26, 0),
                                         (152 * 10240 + 1, 26, 0), (304 * 10240 + 5, 26, 0),
                                         (30_001, 27, 0), (30_001, 67, 16), (30_001, 26, 2),
                                         (30_001, 27, 1), (2_000, 20_000, 0), (300, 30_000, 0)])
def test_encoder_shapes(ctx, n, bpp, shift):
    rng = np.random.default_rng(n + bpp)
    xyz = rng.integers(-2 ** 20, 2 ** 20, (n, 3)) + np.arange(n)[:, None] * np.array([3, 1, 0])
    rec = make_records(xyz, bpp, n)
    hdr = header(n, bpp, xyz)
    want = synth.encode_las(rec, n, hdr, bytes_per_point=bpp)
    cloud = ctx.cloud(n, len(want[0]), 1)
    d = cloud.device_pointers()
    buf, at = on_device(rec, shift)
    v = [np.ascontiguousarray(x[:], np.float64) for x in (hdr.scale, hdr.offset, hdr.min)]
    ctx.check(ctx.lib.cr_encode_las_device(ctx.handle, at, n, bpp, 2, *(ptr(a) for a in v), 0, 0,
                                           d["batches"], d["low"], d["med"], d["hig"], d["rgba"],
                                           None), "encode")
    ctx.sync()
    assert np.array_equal(cloud.read(0).view(np.uint8), want[0].view(np.uint8))
    for which, arr in zip((L.STREAM_LOW, L.STREAM_MED, L.STREAM_HIG, L.STREAM_RGBA), want[1:]):
        assert np.array_equal(cloud.read(which), arr), which
    cloud.close()


# spread: half of int32's range per axis, no equal upper bits; runs: cells of 3-40
# points that differ in the low bits only; long: one cell of 5,000 points, past the
# run sort's limit; equal: duplicates, whose order is the records' own
@pytest.mark.parametrize("case", ["spread", "runs", "long", "equal"])
@pytest.mark.parametrize("n,bpp,shift", [(2, 26, 0), (2_049, 26, 0), (200_003, 34, 0),
                                         (50_001, 26, 2), (50_001, 26, 6)])
def test_morton_sort_runs(ctx, case, n, bpp, shift):
    rng = np.random.default_rng(n)
    if case == "spread":
        xyz = rng.integers(-2 ** 30, 2 ** 30, (n, 3))
    else:
        cells = max(1, n // (20 if case == "runs" else 50))
        at = rng.integers(-2 ** 30, 2 ** 30, (cells, 3))
        xyz = at[rng.integers(0, cells, n)] + (0 if case == "equal" else rng.integers(0, 2 ** 15, (n, 3)))
        if case == "long":
            m = min(n, 5_000)
            xyz[:m] = at[0] + rng.integers(0, 2 ** 14, (m, 3))
        xyz[0], xyz[-1] = -2 ** 30, 2 ** 30 + 2 ** 15
    rec = make_records(xyz, bpp, n + 1)
    hdr = header(n, bpp, xyz)
    want = rec.copy()
    assert ctx.lib.cr_morton_sort_host(ptr(want), n, bpp, C.byref(hdr)) == L.OK
    buf, at = on_device(rec, shift)
    ctx.check(ctx.lib.cr_morton_sort_device(ctx.handle, at, n, bpp, C.byref(hdr), None), "sort")
    got = buf[shift:shift + rec.size].cpu().numpy()
    assert np.array_equal(got, want)
    assert int(buf[:shift].sum()) == 0 and int(buf[shift + rec.size:].sum()) == 0
