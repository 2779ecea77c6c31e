"""The sort's kept buffer: it grows, serves smaller calls, is given back by a call
with n = 0 and by an allocation that runs out of memory, and two sorts of one
context at once each have their own."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from compute_rasterizer_gb300 import Context, default_params, synth
from compute_rasterizer_gb300 import _lib as L
from compute_rasterizer_gb300._lib import ptr
from compute_rasterizer_gb300.multiview import MultiView
from compute_rasterizer_gb300.raster import CRError

pytestmark = pytest.mark.gpu
BPP = L.LAS_FORMAT2_BYTES


def cloud_records(n, seed):
    rec, hdr = synth.las_records_host(synth.synth_params(L.SYNTH_TERRAIN, 300.0, seed), n)
    want = rec.copy()
    lib = L.load()
    assert lib.cr_morton_sort_host(ptr(want), n, BPP, C.byref(hdr)) == L.OK
    return rec, hdr, want


def sort(ctx, rec, hdr, stream=None):
    got = torch.from_numpy(rec).cuda()
    torch.cuda.synchronize()
    ctx.check(ctx.lib.cr_morton_sort_device(ctx.handle, got.data_ptr(), len(rec) // BPP, BPP,
                                            C.byref(hdr), stream), "sort")
    return got.cpu().numpy()


def free_bytes():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_grow_and_shrink():
    ctx = Context(0)
    for n in (20_000, 1_500_000, 3, 80_000, 2_000_000):
        rec, hdr, want = cloud_records(n, n)
        assert np.array_equal(sort(ctx, rec, hdr), want), n
    ctx.close()


@pytest.mark.parametrize("how", ["empty call", "out of memory"])
def test_given_back(how):
    ctx = Context(0)
    n = 4_000_000
    rec, hdr, want = cloud_records(n, 9)
    assert np.array_equal(sort(ctx, rec, hdr), want)
    kept = free_bytes()
    if how == "empty call":
        ctx.check(ctx.lib.cr_morton_sort_device(ctx.handle, None, 0, BPP, C.byref(hdr), None), "sort")
    else:
        # item lists of 2^20 batches and 65,536 views are 1 TB: the allocation fails at once
        cloud = ctx.cloud(10, 1 << 20, 1)
        with pytest.raises(CRError) as e:
            MultiView(ctx, cloud, [(16, 16)] * 65_536, default_params(L.METHOD_LOOP_LAS))
        assert e.value.status == L.OUT_OF_MEMORY
        cloud.close()
    assert free_bytes() - kept >= n * (8 + 8 + 4 + 4 + BPP)
    assert np.array_equal(sort(ctx, rec, hdr), want)
    ctx.close()


def test_two_at_once(ctx):
    jobs = [cloud_records(n, n) for n in (300_000, 400_001)]
    streams = [torch.cuda.Stream() for _ in jobs]
    out = [[], []]

    def work(i):
        rec, hdr, _ = jobs[i]
        out[i] = [sort(ctx, rec, hdr, streams[i].cuda_stream) for _ in range(4)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (_, _, want), got in zip(jobs, out):
        assert len(got) == 4 and all(np.array_equal(g, want) for g in got)
