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


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,bd,nref,kw", [
    (16, 16, 8, 1, {}), (16, 80, 10, 2, {}), (176, 16, 8, 4, dict(h264_umh=1)), (33, 47, 8, 3, {}),
    (208, 144, 12, 4, dict(h264_umh=1, h264_range=37)), (208, 144, 8, 2, dict(h264_dia=1, h264_qpel_diamond=1)),
    (208, 144, 8, 3, dict(h264_range=0, h264_refine_ratio=0.0)), (208, 144, 8, 2, dict(h264_range=1, h264_umh=1)),
    (112, 96, 10, 3, dict(h264_hpel_iters=0, h264_qpel_iters=0)), (112, 96, 8, 3, dict(h264_vertical_range=3)),
    (112, 96, 8, 2, dict(h264_pad=8, h264_hpel_iters=5, h264_qpel_iters=1))])
def test_h264_rows_of_every_shape(ms, w, h, bd, nref, kw):
    """One macroblock, one row, one column, ragged sides, every pattern and
    the settings' ends, one to four references."""
    rng = np.random.default_rng(w + h + nref)
    refs = [random_picture(rng, w, h, bd)]
    for k in range(1, nref):
        refs.append(shifted(refs[0], 3 * k, -2 * k, rng, 2.0))
    src = shifted(refs[-1], -5, 6, rng, 2.0)
    src[: h // 2] = shifted(refs[0], 9, 2, rng, 1.0)[: h // 2]
    for i, pic in enumerate(refs + [src]):
        ms.upload(2500 + i, pic, H264, bd, as_ref=i < nref)
    p = oracle.params(H264, 29, **kw)
    got = ms.search(2500 + nref, [2500 + i for i in range(nref)], p)
    assert_results_equal(got, oracle.frame_search(H264, bd, src, refs, p), "H.264 rows")
    for i in range(nref + 1):
        ms.release(2500 + i)


@pytest.mark.gpu
@pytest.mark.parametrize("bd,kw", [
    (8, dict(h264_range=40)), (10, dict(h264_range=40, h264_dia=1)), (8, dict(h264_range=24, h264_hpel_iters=13)),
    (10, dict(h264_range=24, h264_hpel_iters=14, h264_qpel_iters=1)), (8, dict(h264_umh=1, h264_range=25)),
    (10, dict(h264_umh=1, h264_range=25)), (8, dict(h264_umh=1, h264_range=26)), (10, dict(h264_umh=1, h264_range=3))])
def test_h264_walks_beyond_the_staged_window(ms, bd, kw):
    """Long walks over smooth pictures, which leave the samples staged around
    their start; refinements too long to be staged; the UMH ranges on both
    sides of the largest staged one."""
    w, h = 144, 112
    rng = np.random.default_rng(bd + kw["h264_range"])
    yy, xx = np.mgrid[0:h + 64, 0:w + 64]
    full = (1 << bd) - 1
    wave = np.sin(xx / 23.0) + np.sin(yy / 19.0) + np.sin((xx + 2 * yy) / 41.0)
    big = np.clip((wave / 6 + 0.5) * full + rng.normal(0, 1.0, wave.shape), 0, full)
    big = big.astype(np.uint8 if bd == 8 else np.uint16)
    ref = np.ascontiguousarray(big[32:32 + h, 32:32 + w])
    src = np.ascontiguousarray(big[32 - 13:32 - 13 + h, 32 + 19:32 + 19 + w])
    ms.upload(2560, ref, H264, bd)
    ms.upload(2561, src, H264, bd, as_ref=False)
    p = oracle.params(H264, 30, **kw)
    got = ms.search(2561, [2560], p)
    assert_results_equal(got, oracle.frame_search(H264, bd, src, [ref], p), "long walks")
    ms.release(2560)
    ms.release(2561)


@pytest.mark.gpu
def test_h264_rows_of_uneven_frames_together(ms):
    """Frames of different sizes, settings and reference counts in one
    launch, beside a GIVEN-free HEVC frame: as each by itself."""
    rng = np.random.default_rng(77)
    frames, params, want = [], [], []
    for k, (codec, w, h, nref) in enumerate([(H264, 96, 64, 1), (H264, 160, 48, 3), (HEVC, 128, 96, 2), (H264, 16, 96, 2)]):
        refs = [random_picture(rng, w, h, 8) for _ in range(nref)]
        src = shifted(refs[0], 2, 1, rng, 2.0)
        base = 2600 + 10 * k
        for i, pic in enumerate(refs + [src]):
            ms.upload(base + i, pic, codec, 8)
        frames.append((base + nref, [base + i for i in range(nref)]))
        params.append(oracle.params(codec, 28, h264_umh=k & 1))
        want.append(oracle.frame_search(codec, 8, src, refs, params[-1]))
    for _ in range(4):  # the first calls, the capture, its replays
        for g, w_ in zip(ms.search_batch(frames, params), want):
            assert_results_equal(g, w_, "mixed rows")
    for s, r in frames:
        for i in [s] + r:
            ms.release(i)


@pytest.mark.gpu
def test_a_launch_of_more_than_128_dataflow_frames(ms):
    """A task kept by the warp that made it ready is named by frame and task
    in 32 bits: frames 128 and up set the top one."""
    rng = np.random.default_rng(5)
    ref = random_picture(rng, 64, 32, 8)
    src = shifted(ref, 1, -2, rng, 2.0)
    ms.upload(2700, ref, HEVC, 8)
    ms.upload(2701, src, HEVC, 8)
    p = oracle.params(HEVC, 32, hevc_amp=1)
    want = oracle.frame_search(HEVC, 8, src, [ref], p)
    for got in ms.search_batch([(2701, [2700])] * 200, p):
        assert_results_equal(got, want, "frame of 200")
    ms.release(2700)
    ms.release(2701)


@pytest.mark.gpu
@pytest.mark.parametrize("codec,bd", [(HEVC, 8), (HEVC, 12), (H264, 8), (H264, 12)])
@pytest.mark.parametrize("kw", [{}, dict(hevc_amp=15, hevc_lambda_scale=1024.0)])
def test_distortion_and_rate_at_their_ends(ms, codec, bd, kw):
    """Samples at the depth's ends only, in stripes, squares and noise, so
    that Hadamard sums reach their largest magnitudes; the largest rates."""
    rng = np.random.default_rng(bd + len(kw))
    w, h, top = 144, 80, (1 << bd) - 1
    yy, xx = np.mgrid[0:h, 0:w]
    fields = [xx % 2, yy % 2, (xx + yy) % 2, rng.integers(0, 2, (h, w)), np.zeros((h, w)), (xx // 2 + yy // 2) % 2]
    pics = [(np.asarray(f) * top).astype(np.uint8 if bd == 8 else np.uint16) for f in fields]
    for i, pic in enumerate(pics):
        ms.upload(2800 + i, pic, codec, bd)
    p = oracle.params(codec, 63 if kw else 12, **kw)
    for a, b in [(0, 1), (2, 4), (3, 2), (5, 3), (1, 5)]:
        got = ms.search(2800 + a, [2800 + b], p)
        assert_results_equal(got, oracle.frame_search(codec, bd, pics[a], [pics[b]], p), f"fields {a} against {b}")
    for i in range(len(pics)):
        ms.release(2800 + i)


@pytest.mark.gpu
@pytest.mark.parametrize("bd,kw", [(8, {}), (10, dict(hevc_search_rings=2, hevc_quarter_cross=1)),
                                   (12, dict(hevc_search_range=1)), (8, dict(hevc_search_range=0, hevc_pad=8))])
def test_given_jobs_of_every_shape(ms, bd, kw):
    """Every block shape, no seed to ten, seeds far outside, blocks at the
    picture's edges."""
    rng = np.random.default_rng(bd + len(kw))
    w, h = 150, 102
    ref = random_picture(rng, w, h, bd)
    src = shifted(ref, -4, 3, rng, 2.0)
    ms.upload(2900, src, HEVC, bd)
    ms.upload(2901, ref, HEVC, bd)
    jobs = np.zeros(512, capi.JOB_DTYPE)
    for i, j in enumerate(jobs):
        bw, bh = 4 * (i % 16) + 4, 4 * (i // 16 % 16) + 4
        j["w"], j["h"] = bw, bh
        j["x"] = rng.choice([0, w - bw, rng.integers(0, w - bw + 1)])
        j["y"] = rng.choice([0, h - bh, rng.integers(0, h - bh + 1)])
        j["nseeds"] = i % 11
        spread = 40 if i % 3 else 2000
        j["mvp"] = rng.integers(-spread, spread + 1, (2, 2))
        j["seeds"] = rng.integers(-spread, spread + 1, (capi.RME_MAX_SEEDS, 2))
    p = oracle.params(HEVC, 31, predictor_mode=capi.RME_PRED_GIVEN, **kw)
    got = ms.search(2900, [2901], p, jobs)
    assert_results_equal(got, oracle.frame_search(HEVC, bd, src, [ref], p, jobs), "GIVEN shapes")
    ms.release(2900)
    ms.release(2901)


@pytest.mark.gpu
@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("kw", [{}, dict(hevc_search_rings=3, hevc_quarter_cross=1), dict(hevc_search_range=2)])
def test_given_jobs_of_half_a_warp(ms, bd, kw):
    """Blocks of at most sixteen words (8 bits: a warp's halves score
    candidates of their own) and just above: one seed to ten, several alike,
    walks through the picture and along its edges."""
    rng = np.random.default_rng(bd + 17 * len(kw))
    w, h = 134, 98
    ref = random_picture(rng, w, h, bd, smooth=6)
    src = shifted(ref, 6, -5, rng, 2.0)
    ms.upload(2920, src, HEVC, bd)
    ms.upload(2921, ref, HEVC, bd)
    shapes = [(4, 4), (8, 4), (4, 8), (8, 8), (16, 4), (4, 16), (12, 4), (4, 12), (12, 8), (4, 20), (20, 4)]
    jobs = np.zeros(660, capi.JOB_DTYPE)
    for i, j in enumerate(jobs):
        bw, bh = shapes[i % len(shapes)]
        j["w"], j["h"] = bw, bh
        j["x"] = rng.choice([0, w - bw, rng.integers(0, w - bw + 1)])
        j["y"] = rng.choice([0, h - bh, rng.integers(0, h - bh + 1)])
        j["nseeds"] = i // len(shapes) % 11
        spread = 30 if i % 5 else 900
        j["mvp"] = rng.integers(-spread, spread + 1, (2, 2))
        j["seeds"] = rng.integers(-spread, spread + 1, (capi.RME_MAX_SEEDS, 2))
        j["seeds"][2] = j["seeds"][0]
    p = oracle.params(HEVC, 27, predictor_mode=capi.RME_PRED_GIVEN, **kw)
    want = oracle.frame_search(HEVC, bd, src, [ref], p, jobs)
    small = jobs["w"] * jobs["h"] <= 64
    for pick, name in ((slice(None), "with larger ones"), (small, "small ones only"),
                       (np.nonzero(small)[0][:1], "one"), (np.nonzero(jobs["w"] * jobs["h"] == 64)[0][:41], "16 words")):
        assert_results_equal(ms.search(2920, [2921], p, jobs[pick]), want[pick], name)
    bi = np.zeros(300, capi.BI_JOB_DTYPE)  # refine_bi's search, from target blocks of their own
    for i, j in enumerate(bi):
        j["w"], j["h"] = shapes[i % 8]
        j["x"], j["y"] = rng.integers(0, w - j["w"] + 1), rng.integers(0, h - j["h"] + 1)
        j["ref"], j["list"] = (0, 1), i & 1
        j["mv"] = rng.integers(-60, 61, (2, 2))
        j["mvp"] = j["mv"] + rng.integers(-6, 7, (2, 2))
    got = ms.bi_refine(2920, [2921, 2920], p, bi)
    assert_results_equal(got, oracle.hevc_bi(bd, src, [ref, src], p, bi, refine=True), "refine_bi of small blocks")
    ms.release(2920)
    ms.release(2921)


@pytest.mark.gpu
def test_amp_frames_of_both_depths_with_given_frames(ms):
    """AMP units of several frames of two depths in one launch, frames
    without units and H.264 frames among them: each as by itself."""
    rng = np.random.default_rng(91)
    frames, params, want = [], [], []
    shapes = [(HEVC, 10, 130, 70, 2, 5), (HEVC, 8, 64, 64, 1, 0), (HEVC, 8, 96, 48, 2, 15), (H264, 8, 64, 48, 1, 0),
              (HEVC, 10, 72, 136, 1, 8), (HEVC, 8, 16, 16, 3, 2)]
    for k, (codec, bd, w, h, nref, amp) in enumerate(shapes):
        refs = [random_picture(rng, w, h, bd) for _ in range(nref)]
        src = shifted(refs[0], -2, 3, rng, 2.0)
        base = 3000 + 10 * k
        for i, pic in enumerate(refs + [src]):
            ms.upload(base + i, pic, codec, bd)
        frames.append((base + nref, [base + i for i in range(nref)]))
        params.append(oracle.params(codec, 30, hevc_amp=amp))
        want.append(oracle.frame_search(codec, bd, src, refs, params[-1]))
    for _ in range(4):  # the first calls, the capture, its replays
        for g, w_ in zip(ms.search_batch(frames, params), want):
            assert_results_equal(g, w_, "AMP among others")
    for s, r in frames:
        for i in [s] + r:
            ms.release(i)


@pytest.mark.gpu
@pytest.mark.parametrize("bd,extra", [(8, 0), (8, 1), (8, 2), (8, 3), (10, 1), (10, 2)])
def test_no_alloc_search_on_rows_at_any_offset(ms, bd, extra):
    """A caller's planes whose rows lie whole words apart, and not."""
    import ctypes as C
    import torch
    rng = np.random.default_rng(bd + extra)
    w, h, pad = 96, 72, 80
    ref = random_picture(rng, w, h, bd)
    src = shifted(ref, 3, -2, rng, 2.0)
    for i, pic in enumerate((src, ref)):
        ms.upload(3100 + i, pic, HEVC, bd)
    p = oracle.params(HEVC, 30, predictor_mode=capi.RME_PRED_GIVEN)
    from _common import random_jobs
    jobs = random_jobs(rng, HEVC, w, h, 1, 120, spread=200)
    want = oracle.frame_search(HEVC, bd, src, [ref], p, jobs)
    sets, keep = [], []
    for i in range(2):
        planes = np.stack([ms.plane(3100 + i, k) for k in range(16)])
        wide = np.zeros(planes.shape[:2] + (planes.shape[2] + extra,), planes.dtype)
        wide[:, :, :planes.shape[2]] = planes
        buf = torch.zeros(wide.nbytes + 16, dtype=torch.uint8, device="cuda")
        buf[:wide.nbytes].copy_(torch.from_numpy(wide.view(np.uint8).ravel()))
        keep.append(buf)
        sets.append(capi.PlaneSet(buf.data_ptr(), wide.shape[1] * wide.shape[2], wide.shape[2], pad))
    d_jobs = torch.from_numpy(jobs.view(np.uint8).copy()).cuda()
    d_out = torch.zeros(len(jobs) * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    d = capi.PictureDesc(HEVC, bd, w, h, w)
    refs = (capi.PlaneSet * 1)(sets[1])
    rc = capi.lib().rme_search_given_noalloc(C.byref(d), C.byref(p), C.byref(sets[0]), refs, 1,
                                             C.c_void_p(d_jobs.data_ptr()), len(jobs), C.c_void_p(d_out.data_ptr()), None)
    assert rc == capi.RME_OK, rc
    assert_results_equal(d_out.cpu().numpy().view(capi.RESULT_DTYPE), want, f"rows {extra} samples further apart")
    ms.release(3100)
    ms.release(3101)


@pytest.mark.gpu
@pytest.mark.parametrize("bd", [8, 9, 10, 12])
@pytest.mark.parametrize("w,h", [(16, 16), (17, 31), (97, 45), (130, 70)])
def test_phase_planes_at_tile_edges(ms, bd, w, h):
    """Every phase over pictures whose padded planes end inside a tile, a
    lane's columns and a strip's rows; noise and rails."""
    rng = np.random.default_rng(w + bd)
    top = (1 << bd) - 1
    pic = np.where(rng.random((h, w)) < 0.5, rng.integers(0, 2, (h, w)) * top, rng.integers(0, top + 1, (h, w)))
    pic = pic.astype(np.uint8 if bd == 8 else np.uint16)
    ms.upload(3200, pic, HEVC, bd)
    base, _ = oracle.hevc_planes(pic, bd)
    want, ext = oracle.hevc_planes(pic, bd, force_quarter=True)
    np.testing.assert_array_equal(ms.plane(3200, 0), base[0])
    sl = (slice(80 - ext, 80 + h + ext), slice(80 - ext, 80 + w + ext))
    for k in range(1, 16):
        np.testing.assert_array_equal(ms.plane(3200, k)[sl], want[k][sl], err_msg=f"phase {k}")
    # The whole padded plane is the interpolation of the replicated picture.
    taps = np.array([[0, 0, 0, 64, 0, 0, 0, 0], [-1, 4, -10, 58, 17, -5, 1, 0], [-1, 4, -11, 40, 40, -11, 4, -1],
                     [0, 1, -5, 17, 58, -10, 4, -1]], np.int64)
    full = np.pad(pic.astype(np.int64), 80 + 4, mode="edge")
    rows, cols = h + 160, w + 160
    for fy in range(4):
        for fx in range(4):
            if not fx and not fy:
                continue
            if fx:
                t = sum(taps[fx][k] * full[:, k + 1:k + 1 + cols] for k in range(8)) >> (min(bd, 12) - 8)
            else:
                t = full[:, 4:4 + cols]
            if fy:
                t = sum(taps[fy][k] * t[k + 1:k + 1 + rows] for k in range(8)) >> (6 if fx else min(bd, 12) - 8)
            else:
                t = t[4:4 + rows]
            sh = 14 - bd
            np.testing.assert_array_equal(ms.plane(3200, fy * 4 + fx), np.clip((t + (1 << (sh - 1))) >> sh, 0, top),
                                          err_msg=f"padded phase {fx}, {fy}")
    ms.release(3200)


@pytest.mark.gpu
@pytest.mark.parametrize("codec,bd,w,h,extra,as_ref", [
    (HEVC, 8, 16, 16, 0, True), (HEVC, 8, 33, 17, 0, True), (HEVC, 8, 850, 21, 5, True), (HEVC, 10, 131, 40, 0, True),
    (HEVC, 10, 130, 16, 2, False), (HEVC, 8, 47, 19, 0, False), (H264, 8, 31, 47, 0, True), (H264, 10, 99, 33, 0, True),
    (H264, 8, 99, 33, 7, True), (H264, 8, 17, 16, 0, False)])
def test_padded_plane_of_packed_and_of_strided_rows(ms, codec, bd, w, h, extra, as_ref):
    """Plane 0 is the picture, its border replicated, whichever way the rows
    came: chunks across the sides, odd addresses, in place or from a packed
    picture."""
    import ctypes as C
    rng = np.random.default_rng(w * h + extra)
    rows = rng.integers(0, 1 << bd, (h, w + extra)).astype(np.uint8 if bd == 8 else np.uint16)
    d = capi.PictureDesc(codec, bd, w, h, w + extra)
    ms.upload(3300, np.zeros((h, w), rows.dtype), codec, bd, as_ref=as_ref)  # registers the picture's shape
    assert capi.lib().rme_picture_upload(ms.ctx, 3300, C.byref(d), capi.ptr(rows), int(as_ref), None) == capi.RME_OK
    pad = 32 if codec == H264 else 80
    cw, ch = ((w + 15) // 16 * 16, (h + 15) // 16 * 16) if codec == H264 else (w, h)
    want = np.pad(rows[:, :w], ((pad, pad + ch - h), (pad, pad + cw - w)), mode="edge")
    np.testing.assert_array_equal(ms.plane(3300, 0), want)
    ms.release(3300)


@pytest.mark.gpu
@pytest.mark.parametrize("bd", [8, 10])
@pytest.mark.parametrize("vr", [-1, 0, 1])
@pytest.mark.parametrize("kw", [{}, dict(h264_dia=1, h264_pad=8), dict(h264_umh=1, h264_range=24, h264_hpel_iters=5),
                                dict(h264_umh=1, h264_range=512), dict(h264_range=40, h264_hpel_iters=64)])
def test_h264_windows_of_no_row_and_of_few(ms, bd, vr, kw):
    """A vertical range of -1 leaves the window empty: every start is clamped
    to the row above, nothing else is scored; 0 and 1 leave one row, three."""
    rng = np.random.default_rng(bd + vr)
    w, h, nref = 80, 64, 3
    refs = [random_picture(rng, w, h, bd)]
    for k in range(1, nref):
        refs.append(shifted(refs[0], 3 * k, -2 * k, rng, 2.0))
    src = shifted(refs[-1], -5, 6, rng, 2.0)
    for i, pic in enumerate(refs + [src]):
        ms.upload(3400 + i, pic, H264, bd, as_ref=i < nref)
    p = oracle.params(H264, 28, h264_vertical_range=vr, **kw)
    got = ms.search(3400 + nref, [3400 + i for i in range(nref)], p)
    want = oracle.frame_search(H264, bd, src, refs, p)
    assert_results_equal(got, want, f"vertical range {vr}")
    if vr < 0:
        assert set(want["mvy"]) == {-4} and set(want["n_sad"]) <= set(range(nref, 9 * nref + 1))
    for i in range(nref + 1):
        ms.release(3400 + i)
