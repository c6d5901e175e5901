"""The STANDALONE kernels' published vectors outlive their launch in a launch
slot's buffer, which later launches of either codec, shape and place reuse: a
word an earlier launch left must never pass for the present one's. Everything
is compared with the oracle, and whole numbers, so the tolerance is none."""
import numpy as np
import pytest

import oracle
import rivet_h26x_codecs_b200.capi as capi
import rivet_h26x_codecs_b200.host as host
from _common import assert_results_equal, random_jobs, random_picture, shifted

H264, HEVC = capi.RME_CODEC_H264, capi.RME_CODEC_HEVC
SLOTS = 4  # the launch slots a context takes in turn


def _pictures(ms, rng, base, codec, bd, w, h, nref):
    """A source (id `base`) and its references, moved apart so that blocks'
    vectors differ from one another and from zero."""
    refs = [random_picture(rng, w, h, bd)]
    for k in range(1, nref):
        refs.append(shifted(refs[0], 5 * k, -3 * k, rng, 2.0))
    src = shifted(refs[-1], -7, 6, rng, 2.0)
    src[: h // 2] = shifted(refs[0], 11, 3, rng, 1.0)[: h // 2]
    for i, pic in enumerate([src] + refs):
        ms.upload(base + i, pic, codec, bd)
    return src, refs, [base + 1 + i for i in range(nref)]


@pytest.mark.gpu
@pytest.mark.parametrize("nref,ref", [(1, 0), (3, 0), (3, 1), (3, 2)])
def test_an_hevc_launch_takes_no_h264_word_for_its_own(nref, ref):
    """H.264 frames at each slot's first epoch, GIVEN calls, which publish
    nothing, up to the epoch 4 + `ref`, then HEVC frames over the places the
    H.264 ones wrote."""
    rng = np.random.default_rng(10 * nref + ref)
    with host.MotionSearch(0) as ms:
        hsrc, hrefs, hids = _pictures(ms, rng, 10, H264, 8, 512, 256, nref)  # 512 macroblocks
        src, refs, ids = _pictures(ms, rng, 20, HEVC, 8, 128, 96, 2)         # 508 searches
        hp, p = oracle.params(H264, 28), oracle.params(HEVC, 32)
        gp = oracle.params(HEVC, 32, predictor_mode=capi.RME_PRED_GIVEN)
        jobs = random_jobs(rng, HEVC, 128, 96, 2, 6)
        want = oracle.frame_search(H264, 8, hsrc, hrefs, hp)
        for _ in range(SLOTS):
            assert_results_equal(ms.search(10, hids, hp), want, "H.264")
        for _ in range((2 + ref) * SLOTS):
            ms.search(20, ids, gp, jobs)
        want = oracle.frame_search(HEVC, 8, src, refs, p)
        for k in range(SLOTS):
            assert_results_equal(ms.search(20, ids, p), want, f"HEVC, slot {k}")


@pytest.mark.gpu
def test_frames_of_both_codecs_change_places_from_call_to_call():
    """Twenty batches of H.264 and HEVC frames in orders of their own."""
    rng = np.random.default_rng(4)
    with host.MotionSearch(0) as ms:
        frames, params, want = [], [], []
        for k, (codec, w, h, nref) in enumerate([(H264, 320, 160, 3), (HEVC, 96, 64, 2), (H264, 96, 64, 2),
                                                 (HEVC, 128, 96, 1), (HEVC, 64, 64, 4)]):
            src, refs, ids = _pictures(ms, rng, 100 + 10 * k, codec, 8, w, h, nref)
            frames.append((100 + 10 * k, ids))
            params.append(oracle.params(codec, 30))
            want.append(oracle.frame_search(codec, 8, src, refs, params[-1]))
        for call in range(20):
            order = rng.permutation(len(frames))[: rng.integers(1, len(frames) + 1)]
            got = ms.search_batch([frames[i] for i in order], [params[i] for i in order])
            for i, g in zip(order, got):
                assert_results_equal(g, want[i], f"call {call}, frame {i} of {list(order)}")


@pytest.mark.gpu
def test_a_buffer_that_grows_where_it_stood_holds_no_earlier_words():
    """Two hundred contexts whose launches grow by small steps, the four
    slots' buffers at different calls: a larger buffer may begin where the old
    one did and end over another slot's old words."""
    rng = np.random.default_rng(2)
    ref = random_picture(rng, 64, 64, 8)
    src = shifted(ref, -7, 6, rng, 2.0)
    src[:32] = shifted(ref, 11, 3, rng, 1.0)[:32]
    p = oracle.params(HEVC, 32)
    want = oracle.frame_search(HEVC, 8, src, [ref], p)
    for context in range(200):
        with host.MotionSearch(0) as ms:
            ms.upload(0, src, HEVC, 8)
            ms.upload(1, ref, HEVC, 8)
            n = 1
            while (n := int(n * rng.uniform(1.2, 2.0)) + 1) < 100:
                for _ in range(rng.integers(1, 7)):
                    for got in ms.search_batch([(0, [1])] * int(n if rng.random() < 0.7 else rng.integers(1, n + 1)), p):
                        assert_results_equal(got, want, f"context {context}, {n} frames")
