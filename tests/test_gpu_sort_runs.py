"""The Morton sort's run sort against the host sort: runs of equal upper key bits of
every length up to the limit, across tile borders, with ties, one at the limit (all
bits are sorted instead), and counts either side of the rule for short clouds."""
import ctypes as C

import numpy as np
import pytest
import torch

from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300._lib import ptr

pytestmark = pytest.mark.gpu
BPP = 26


def records(n, lengths, ties, seed):
    """n records in cells of 2^18 units (equal upper 40 key bits), whose point
    counts cycle through `lengths`, in random order."""
    rng = np.random.default_rng(seed)
    sizes = np.resize(lengths, n)  # more than enough
    sizes = sizes[:np.searchsorted(np.cumsum(sizes), n) + 1]
    cells = rng.choice(2 ** 24, len(sizes), replace=False)
    at = np.stack([cells >> 16, (cells >> 8) & 255, cells & 255], 1) * 2 ** 23 - 2 ** 30
    # spacing of the q cells is 1,024 units; with ties a cell has few distinct keys
    step = 2 ** 15 if ties else 2 ** 10
    xyz = np.repeat(at, sizes, 0)[:n] + rng.integers(0, 2 ** 17 // step, (n, 3)) * step
    xyz = xyz[rng.permutation(n)].astype("<i4")
    rec = rng.integers(0, 256, (n, BPP), dtype=np.uint8)
    rec[:, :12] = xyz.view(np.uint8).reshape(n, 12)
    hdr = L.LasHeader()
    hdr.num_points, hdr.point_format, hdr.bytes_per_point = n, 2, BPP
    hdr.scale[:], hdr.offset[:] = [1.0] * 3, [0.0] * 3
    hdr.min[:], hdr.max[:] = [-2.0 ** 30] * 3, [2.0 ** 30] * 3
    return rec.reshape(-1), hdr


@pytest.mark.parametrize("ties", [False, True])
@pytest.mark.parametrize("lengths", [[1], [2, 1, 3], [31, 5, 62], [63], [63, 1, 64], [5000]])
@pytest.mark.parametrize("n", [81_920, 81_921, 100_003])
def test_runs(ctx, n, lengths, ties):
    rec, hdr = records(n, lengths, ties, n + len(lengths))
    want = rec.copy()
    assert ctx.lib.cr_morton_sort_host(ptr(want), n, BPP, C.byref(hdr)) == L.OK
    got = torch.from_numpy(rec).cuda()
    ctx.check(ctx.lib.cr_morton_sort_device(ctx.handle, got.data_ptr(), n, BPP, C.byref(hdr), None),
              "sort")
    assert np.array_equal(got.cpu().numpy(), want)
