"""The resident engine with more than 128 frames in flight: a task that a warp
or a CTA runs next by itself is named by its frame's slot and its number in 32
bits, whose top bit is set from slot 128 on. The slots in use are read from the
server's trace, in a process of its own."""
import os
import re
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
codec, w, h, n = {codec}, 448, 256, 192
rng = np.random.default_rng(4)
pics = [random_picture(rng, w, h, 8)]
while len(pics) < 4:
    pics.append(shifted(pics[-1], 3, -2, rng, 2.0))
p = oracle.params(codec, 30, hevc_amp=15)
with host.MotionSearch(0) as ms:
    srv = host.Server(ms, hbm_budget_bytes=16 << 30, max_frames_per_launch=8, max_streams=n, resident=True)
    try:
        for i in range(n):
            assert srv.open_stream(i, codec, 8, w, h, p, 1) == 0
        ids = {{}}
        for t, pic in enumerate(pics):
            for i in range(n):
                ids[srv.submit(i, pic)] = t
        got, t0 = [], time.time()
        while len(got) < len(ids):
            for c in srv.poll():
                assert c["status"] == 0, c
                got.append((ids[c["id"]], c["results"]))
            assert time.time() - t0 < 60, f"{{len(got)}} of {{len(ids)}} frames"
            time.sleep(0.001)
    finally:
        srv.stop()
want = [None] + [oracle.frame_search(codec, 8, pics[t], [pics[t - 1]], p) for t in range(1, 4)]
for t, res in got:
    if t:
        assert_results_equal(res, want[t], f"frame {{t}}")
print("served", len(got))
"""


@pytest.mark.gpu
@pytest.mark.parametrize("codec", [1, 0], ids=["HEVC with AMP units", "H.264"])
def test_tasks_of_frames_in_the_upper_slots(codec):
    run = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT), codec=codec)], capture_output=True,
                         text=True, timeout=180, env=dict(os.environ, RME_SERVE_TRACE="1"))
    assert run.returncode == 0 and "served 768" in run.stdout, run.stdout[-2000:] + run.stderr[-2000:]
    slots = {int(s) for s in re.findall(r"slot (\d+):", run.stderr)}
    if max(slots) < 128:  # every result was right all the same
        pytest.skip(f"{len(slots)} slots in use: the host submitted too slowly to reach the upper ones")
