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


@pytest.mark.gpu
@pytest.mark.parametrize("codec,bd", [(HEVC, 8), (HEVC, 12), (H264, 8), (H264, 12)])
@pytest.mark.parametrize("w,h", [(16, 16), (16, 210), (403, 16), (83, 75)])
def test_lowres_rows_of_every_shape(ms, codec, bd, w, h):
    """One block, one column, one row of blocks, ragged sides; still, even
    and torn motion (the first pass's rings known or not), several pairs."""
    rng = np.random.default_rng(w * h + bd)
    pics = [random_picture(rng, w, h, bd, smooth=2)]
    pics.append(shifted(pics[0], 4, -2))
    torn = shifted(pics[0], -7, 5, rng, 2.0)
    torn[: h // 2] = shifted(pics[0], 12, 9)[: h // 2]
    pics.append(torn)
    for i, pic in enumerate(pics):
        ms.upload(2400 + i, pic, codec, bd, as_ref=False)
        ms.lowres_build(2400 + i)
    pairs = [(1, 0), (2, 0), (0, 0), (2, 1), (0, 2)]
    got = ms.lowres_search_batch([(2400 + a, 2400 + b) for a, b in pairs])
    for (a, b), g in zip(pairs, got):
        for x, y, name in zip(g, oracle.lowres_search(pics[a], pics[b], bd, codec), ("cost", "mv", "nsad")):
            np.testing.assert_array_equal(x, y, f"{name} of {a} against {b}")
    for i in range(3):
        ms.release(2400 + i)
