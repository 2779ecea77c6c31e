"""HQS frames either side of the batch count up to which the color pass draws both
lists in one grid, against the oracle; one file and many."""
import numpy as np
import pytest

from compute_rasterizer_gb300 import _lib as L
from helpers import QUIRKS, cameras, encoded, gpu_raw, many_file_cameras, many_file_cloud, oracle_frame
from oracle import oracle as O

pytestmark = pytest.mark.gpu
Q = QUIRKS[L.METHOD_LOOP_LAS_HQS]


def check(ctx, cl, cam, box_min, literal):
    cloud = ctx.cloud_from_arrays(cl["batches"], cl["lo"], cl["md"], cl["hi"], cl["rgba"], cl["box_min"])
    fb, p = gpu_raw(ctx, cloud, cam, L.METHOD_LOOP_LAS_HQS, quirks=Q | literal)
    per_level = list(ctx.frame_stats(cloud, p).points_per_level)
    with O.arith(O.ARITH_LITERAL if literal else O.ARITH_CONTRACT):
        fr = oracle_frame(cam, box_min, Q)
        depth, accum, _ = O.hqs(fr, cl["batches"], cl["n"], cl["lo"], cl["md"], cl["hi"], cl["rgba"])
    assert np.array_equal(fb.read(L.FB_DEPTH), depth)
    assert np.array_equal(fb.read(L.FB_ACCUM), accum)
    fb.close()
    cloud.close()
    return per_level


@pytest.mark.parametrize("batches", [223, 224, 225])
@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
def test_one_grid_or_two(ctx, batches, literal):
    cl = encoded(n=(batches - 1) * L.POINTS_PER_BATCH + 77, extent=450.0, seed=batches)
    for name in ("near", "mid"):
        per_level = check(ctx, cl, cameras(cl, 321, 200)[name], cl["box_min"][None], literal)
        assert per_level[1] > 0 and sum(per_level[2:]) > 0


@pytest.mark.parametrize("nfiles", [20, 230])
@pytest.mark.parametrize("literal", [0, L.QUIRK_LITERAL_ARITH])
def test_many_files(ctx, nfiles, literal):
    cl = many_file_cloud(nfiles, seed=nfiles, extent=900.0, base=700, spread=99)
    for cam in many_file_cameras(cl, 160, 90).values():
        check(ctx, cl, cam, cl["box_min"], literal)
