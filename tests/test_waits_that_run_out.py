"""The STANDALONE launches' waits for other rows' vectors, given so few polls
that they run out all over a launch, at different steps of different warps:
the launch ends all the same, and soon, and says so, or was not short of polls
and is right; the context goes on as if nothing had been. Nothing here faults
or hangs the GPU: a wait that gives up ends its row, its CTA and the launch."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle
import rivet_h26x_codecs_b200.capi as capi
import rivet_h26x_codecs_b200.host as host
from _common import assert_results_equal, random_picture, shifted

H264, HEVC = capi.RME_CODEC_H264, capi.RME_CODEC_HEVC
POLLS = 1 << 22  # the default


def _frame(ms, rng, base, codec, bd, w, h, nref):
    refs = [random_picture(rng, w, h, bd)]
    for k in range(1, nref):
        refs.append(shifted(refs[0], 5 * k, -3 * k, rng, 2.0))
    src = shifted(refs[-1], -7, 6, rng, 2.0)
    for i, pic in enumerate([src] + refs):
        ms.upload(base + i, pic, codec, bd)
    return src, refs, [base + 1 + i for i in range(nref)]


def _limit(ms, polls):
    assert capi.lib().rme_probe_wait_polls(ms.ctx, polls) == capi.RME_OK


def test_the_limit_of_polls_is_checked():
    lib = capi.lib()
    assert lib.rme_probe_wait_polls(None, 100) == capi.RME_EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("codec,bd,nref,kw", [
    (HEVC, 8, 2, {}), (HEVC, 10, 1, dict(hevc_search_rings=1)), (HEVC, 8, 3, dict(hevc_amp=5)),
    (HEVC, 10, 2, dict(hevc_pu_mask=0b0101)), (H264, 8, 1, {}), (H264, 10, 4, dict(h264_dia=1)),
    (H264, 8, 3, dict(h264_umh=1, h264_range=24)), (H264, 8, 2, dict(h264_refine_ratio=1.0))])
def test_a_launch_short_of_polls_ends_and_the_next_is_right(codec, bd, nref, kw):
    rng = np.random.default_rng(bd + nref)
    with host.MotionSearch(0) as ms:
        assert capi.lib().rme_probe_wait_polls(ms.ctx, 0) == capi.RME_EINVAL
        assert capi.lib().rme_probe_wait_polls(ms.ctx, POLLS + 1) == capi.RME_EINVAL
        src, refs, ids = _frame(ms, rng, 10, codec, bd, 416, 240, nref)
        p = oracle.params(codec, 30, **kw)
        want = oracle.frame_search(codec, bd, src, refs, p)
        ran_out = 0
        for polls in (1, 2, 5, 15, 40, 64, 100, 200, 400, 1000) * 3:
            _limit(ms, polls)
            t0 = time.time()
            try:
                got = ms.search(10, ids, p)
            except RuntimeError as e:
                assert "device status 1" in str(e), e
                ran_out += 1
            else:
                assert_results_equal(got, want, f"{polls} polls")
            assert time.time() - t0 < 5.0
        assert ran_out > 0  # a row's first block is waited for longer than one poll
        _limit(ms, POLLS)
        for _ in range(4):
            assert_results_equal(ms.search(10, ids, p), want, "with every poll again")


@pytest.mark.gpu
def test_a_batch_of_both_codecs_short_of_polls_ends():
    rng = np.random.default_rng(8)
    with host.MotionSearch(0) as ms:
        frames, params, want = [], [], []
        for k, (codec, bd, w, h, nref) in enumerate([(H264, 8, 320, 160, 3), (HEVC, 8, 416, 240, 2), (HEVC, 10, 256, 160, 1),
                                                     (H264, 10, 176, 144, 1)]):
            src, refs, ids = _frame(ms, rng, 100 + 10 * k, codec, bd, w, h, nref)
            frames.append((100 + 10 * k, ids))
            params.append(oracle.params(codec, 30))
            want.append(oracle.frame_search(codec, bd, src, refs, params[-1]))
        for polls in (1, 20, 60) * 4:
            _limit(ms, polls)
            with pytest.raises(RuntimeError, match="device status 1"):
                ms.search_batch(frames, params)
        _limit(ms, POLLS)
        for _ in range(4):
            for g, w_ in zip(ms.search_batch(frames, params), want):
                assert_results_equal(g, w_, "with every poll again")


@pytest.mark.gpu
def test_a_failed_launchs_buffer_is_not_written_by_a_later_one():
    """Pageable results of launches that failed, then launches on the same
    slots that keep theirs on the device."""
    import torch
    rng = np.random.default_rng(3)
    with host.MotionSearch(0) as ms:
        src, refs, ids = _frame(ms, rng, 10, HEVC, 8, 416, 240, 1)
        p = oracle.params(HEVC, 30)
        want = oracle.frame_search(HEVC, 8, src, refs, p)
        n = ms.batch_result_count([(10, ids)], p)
        old = [np.zeros(n, capi.RESULT_DTYPE) for _ in range(4)]  # one for each launch slot
        _limit(ms, 1)
        for o in old:
            with pytest.raises(RuntimeError, match="device status 1"):
                ms.search_batch([(10, ids)], p, out=o)
            o.view(np.uint8)[:] = 0x5a
        _limit(ms, POLLS)
        out = torch.zeros(n * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
        for k in range(8):
            ms.search_batch([(10, ids)], p, out=out)
            assert all((o.view(np.uint8) == 0x5a).all() for o in old), f"call {k}"
        assert_results_equal(out.cpu().numpy().view(capi.RESULT_DTYPE), want, "on the device")


@pytest.mark.gpu
@pytest.mark.parametrize("bd", [8, 10])
def test_a_resident_search_short_of_polls_reports_it_and_ends(bd):
    """The engine's rows: the frames complete with an error, soon, and another
    server on the same device is right."""
    rng = np.random.default_rng(bd)
    pics = [random_picture(rng, 416, 240, bd)]
    while len(pics) < 8:
        pics.append(shifted(pics[-1], 3, -2, rng, 2.0))
    p = oracle.params(HEVC, 30)
    for polls in (1, 40, POLLS):
        with host.MotionSearch(0) as ms:
            _limit(ms, polls)
            srv = host.Server(ms, hbm_budget_bytes=4 << 30, max_frames_per_launch=8, resident=True)
            got, t0 = {}, time.time()
            try:
                assert srv.open_stream(1, HEVC, bd, 416, 240, p, 1) == 0
                ids = {srv.submit(1, pic): k for k, pic in enumerate(pics)}
                while len(got) < len(ids):
                    for c in srv.poll():
                        got[ids[c["id"]]] = c
                    assert time.time() - t0 < 20, f"{len(got)} frames"
                    time.sleep(0.001)
            finally:
                srv.stop()
            failed = {c["status"] for c in got.values()} - {0}
            assert failed <= {capi.RME_EDEVICE}
            if polls == 1:
                assert failed
            if polls == POLLS:
                assert not failed
            for k in (1, 7):
                if got[k]["status"] == 0 and not failed:
                    assert_results_equal(got[k]["results"], oracle.frame_search(HEVC, bd, pics[k], [pics[k - 1]], p), f"{k}")
