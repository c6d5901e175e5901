"""The resident engine in a process of its own, where no kernel has run yet:
the kernels that work beside the running search (uploads of every format, the
publishing of both forms) are on the device before it starts. One that had to
be brought there while the search runs would wait for it to leave, which it
does only once that kernel has run."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

SCRIPT = """
import sys, time
sys.path[:0] = [{root!r}, {root!r} + "/oracle", {root!r} + "/tests"]
import numpy as np
import oracle
import rivet_h26x_codecs_b200.capi as capi
import rivet_h26x_codecs_b200.host as host
from _common import assert_results_equal, random_picture, shifted
HEVC, H264 = capi.RME_CODEC_HEVC, capi.RME_CODEC_H264
rng = np.random.default_rng(1)
streams = {streams}  # (codec, depth, width, height, frames), the first searched while the others begin
pics = []
for codec, bd, w, h, n in streams:
    p = [random_picture(rng, w, h, bd)]
    while len(p) < min(n, 3):
        p.append(shifted(p[-1], 3, -2, rng, 2.0))
    pics.append([p[k % len(p)] for k in range(n)])
with host.MotionSearch(0) as ms:
    srv = host.Server(ms, hbm_budget_bytes=8 << 30, max_frames_per_launch=8, resident=True)
    try:
        for i, (codec, bd, w, h, n) in enumerate(streams):
            assert srv.open_stream(i, codec, bd, w, h, capi.default_params(codec, 30), 1) == 0
        ids = {{}}
        for i, ps in enumerate(pics):
            for k, pic in enumerate(ps):
                ids[srv.submit(i, pic)] = (i, k)
        got, t0 = {{}}, time.time()
        while len(got) < len(ids):
            for c in srv.poll():
                assert c["status"] == 0, c
                got[ids[c["id"]]] = c["results"]
            assert time.time() - t0 < 30, f"{{len(got)}} of {{len(ids)}} frames"
            time.sleep(0.001)
    finally:
        srv.stop()
for i, (codec, bd, w, h, n) in enumerate(streams):
    want = oracle.frame_search(codec, bd, pics[i][1], [pics[i][0]], capi.default_params(codec, 30))
    assert_results_equal(got[(i, 1)], want, f"stream {{i}}")
print("served", len(got))
"""
HEVC8, HEVC10, H8, H10 = (1, 8, 128, 64, 4), (1, 10, 96, 64, 3), (0, 8, 96, 64, 3), (0, 10, 64, 64, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("streams", [((1, 8, 640, 352, 40), H8, HEVC10, H10), ((0, 8, 320, 192, 40), HEVC8, H10, HEVC10)],
                         ids=["HEVC first", "H.264 first"])
def test_formats_that_begin_while_the_engine_runs(streams):
    run = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT), streams=list(streams))],
                         capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-2000:]
    assert "served" in run.stdout


BESIDE = """
import sys, time
sys.path[:0] = [{root!r}, {root!r} + "/oracle", {root!r} + "/tests"]
import numpy as np
import torch
import oracle
import rivet_h26x_codecs_b200.capi as capi
import rivet_h26x_codecs_b200.host as host
from _common import assert_results_equal, random_picture, shifted
HEVC, H264 = capi.RME_CODEC_HEVC, capi.RME_CODEC_H264
a = torch.rand(1024, 1024, device="cuda")
def work():  # kernels whose blocks do not fit beside the resident search, on the default stream
    a.copy_(torch.rand(1024, 1024, device="cuda") @ a).clamp_(0, 1)
work()
torch.cuda.synchronize()
rng = np.random.default_rng(1)
sizes = [(HEVC, 8, 320, 192), (HEVC, 10, 192, 128), (H264, 8, 160, 96)]
pics = []
for codec, bd, w, h in sizes:
    p = [random_picture(rng, w, h, bd)]
    while len(p) < 6:
        p.append(shifted(p[-1], 3, -2, rng, 2.0))
    pics.append(p)
with host.MotionSearch(0) as ms:
    srv = host.Server(ms, hbm_budget_bytes=8 << 30, max_frames_per_launch=8, resident={resident})
    try:
        for i, (codec, bd, w, h) in enumerate(sizes):
            assert srv.open_stream(i, codec, bd, w, h, capi.default_params(codec, 24 + 5 * i), 3) == 0
        ids = {{}}
        for t in range(6):  # a stream's second to fourth picture has a reference more each
            for i in range(len(sizes)):
                ids[srv.submit(i, pics[i][t])] = (i, t)
                work()
        got, t0 = {{}}, time.time()
        while len(got) < len(ids):
            for c in srv.poll():
                assert c["status"] == 0, c
                got[ids[c["id"]]] = c["results"]
            assert time.time() - t0 < 30, f"{{len(got)}} of {{len(ids)}} frames"
            time.sleep(0.001)
        torch.cuda.synchronize()
    finally:
        srv.stop()
for i, (codec, bd, w, h) in enumerate(sizes):
    for t in range(1, 6):
        refs = [pics[i][t - 1 - r] for r in range(min(3, t))]
        want = oracle.frame_search(codec, bd, pics[i][t], refs, capi.default_params(codec, 24 + 5 * i))
        assert_results_equal(got[(i, t)], want, f"stream {{i}} frame {{t}}")
print("served", len(got))
"""


@pytest.mark.gpu
@pytest.mark.parametrize("resident", [False, True])
def test_a_program_with_work_of_its_own_on_the_default_stream(resident):
    """Frame shapes, references and quantisers that come while the program's
    kernels wait on the default stream for the resident search to leave: the
    serving thread waits for nothing there."""
    run = subprocess.run([sys.executable, "-c", BESIDE.format(root=str(ROOT), resident=resident)],
                         capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout[-2000:] + run.stderr[-2000:]
    assert "served 18" in run.stdout
