"""The kernels' own edges against the oracle: the block shapes, vectors and
launch sizes at which a kernel takes another branch or a partial tile.
Everything compared is a whole number, so the tolerance is none."""
import numpy as np
import pytest

import oracle
import rivet_h26x_codecs_b200.capi as capi
from _common import assert_results_equal, random_picture, shifted

H264, HEVC = capi.RME_CODEC_H264, capi.RME_CODEC_HEVC


@pytest.mark.gpu
@pytest.mark.parametrize("bd,cross", [(8, 0), (12, 1)])
def test_weighted_refine_part_edges(ms, bd, cross):
    """Blocks of one tile, of a part and a remainder, of many parts; starts
    on every fraction, out of the picture, and where the ring's vectors wrap
    in 16 bits."""
    rng = np.random.default_rng(bd)
    w, h = 208, 144
    ref = random_picture(rng, w, h, bd)
    src = shifted(ref, 2, -1, rng, 2.0)
    ms.upload(2200, src, HEVC, bd, as_ref=False)
    ms.upload(2201, ref, HEVC, bd, as_ref=True)
    p = oracle.params(HEVC, 30, predictor_mode=capi.RME_PRED_GIVEN, hevc_quarter_cross=cross)
    shapes = [(4, 4), (8, 4), (12, 20), (16, 16), (20, 36), (64, 64), (4, 64), (48, 16)]
    starts = [(0, 0), (1, 3), (-2, 5), (400, -300), (-900, 7), (32767, 0), (3, -32768), (32766, -32767), (-32767, 32766)]
    jobs = np.zeros(len(shapes) * len(starts), capi.JOB_DTYPE)
    for i, j in enumerate(jobs):
        bw, bh = shapes[i % len(shapes)]
        j["w"], j["h"], j["nseeds"] = bw, bh, 1
        j["x"], j["y"] = rng.integers(0, (w - bw) // 4 + 1) * 4, rng.integers(0, (h - bh) // 4 + 1) * 4
        j["seeds"][0] = starts[i // len(shapes)]
        j["mvp"] = rng.integers(-60, 61, (2, 2))
    got = ms.hevc_weighted_refine(2200, [2201], p, jobs, 8, 70, 5)
    assert_results_equal(got, oracle.hevc_weighted_refine(bd, src, [ref], p, jobs, 8, 70, 5), "weighted parts")
    ms.release(2200)
    ms.release(2201)

