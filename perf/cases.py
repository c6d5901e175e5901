"""The workloads this library is measured on: what an encoder asks of the
motion search, through the package's public entry points (MotionSearch and
Server), from pinned host pictures to results.

Kinds
  frame      one picture of a stream: uploaded, then searched against its
             resident references (the plain per-frame path)
  batch      many pictures of streams of one or several formats: uploaded,
             then searched in one launch, results left on the device
  given      a mode decision's own calls: a list of blocks of any shape with
             their predictors and seeds
  lookahead  the half-resolution pass over a few new pictures
  bframe     the pair searches of a B picture (HEVC also its chroma)
  weighted   a weighted reference: the fit's sums, the weighted plane, the
             search on it and the sub-sample refinement (HEVC)
  serve      the serving loop: streams submit pictures, the caller polls

Pictures are a sum of eight sinusoids with noise; each next picture moves
every 64x64 region (H.264: 16x16) of the last one by a vector of its own,
with camera noise on top.
"""
import math
import time

import numpy as np
import torch

import rivet_h26x_codecs_b200 as rme
import rivet_h26x_codecs_b200.capi as capi

H264, HEVC = capi.RME_CODEC_H264, capi.RME_CODEC_HEVC
CODEC = {"h264": H264, "hevc": HEVC}


def listed():
    return [
        # The smallest call: a CIF P picture, one reference, the medium tier.
        dict(name="h264_cif", kind="frame", codec="h264", width=352, height=288, depth=8, refs=1, range=16, qp=28),
        # A small picture whose sides are no multiple of any block size.
        dict(name="hevc_ragged", kind="frame", codec="hevc", width=850, height=478, depth=8, refs=2, range=64, qp=32),
        # The ordinary picture of the serving workload: 1080p, two references.
        dict(name="hevc_1080p", kind="frame", codec="hevc", width=1920, height=1080, depth=8, refs=2, range=64,
             qp=32),
        # The largest: 2160p at 10 bits, four references, AMP shapes.
        dict(name="hevc_2160p10_amp", kind="frame", codec="hevc", width=3840, height=2160, depth=10, refs=4,
             range=128, qp=32, amp=5),
        # A slow H.264 tier: the UMH pattern over three references.
        dict(name="h264_1080p_umh", kind="frame", codec="h264", width=1920, height=1080, depth=8, refs=3, range=24,
             qp=26, umh=1),
        # A transcoder's step over one format: twelve 1080p pictures.
        dict(name="batch_hevc_1080p", kind="batch", streams="12x1920x1080:hevc:8", refs=2, qp=32),
        # A step of streams of uneven shape.
        dict(name="batch_mix", kind="batch", refs=2, qp=30,
             streams="4x640x360:h264:8 6x1280x720:hevc:8 4x1920x1080:hevc:10 2x3840x2160:hevc:8"),
        # An encoder's calls over a picture, 10 bits, every partition shape.
        dict(name="given_hevc10", kind="given", codec="hevc", width=1920, height=1080, depth=10, refs=2, range=48,
             qp=30, jobs=6000),
        # Four new pictures of a lookahead, each against its two predecessors.
        dict(name="lookahead_1080p", kind="lookahead", codec="hevc", width=1920, height=1080, depth=8, pictures=4),
        # Every 16x16 unit of a B picture.
        dict(name="bframe_1080p", kind="bframe", codec="hevc", width=1920, height=1080, depth=8, qp=32),
        # A fade: one explicitly weighted 1080p reference.
        dict(name="weighted_1080p", kind="weighted", codec="hevc", width=1920, height=1080, depth=8, qp=32),
        # Four 720p streams served together, three pictures each in flight.
        dict(name="serve_720p", kind="serve", codec="hevc", width=1280, height=720, depth=8, refs=2, range=64, qp=32,
             streams=4, pictures=3),
    ]


def draw(rng):
    def log_int(lo, hi):
        return min(hi, int(lo * math.exp(rng.random() * math.log((hi + 1) / lo))))

    def size(lo, hi, step):
        w = log_int(lo, hi)
        h = max(96, min(2160, int(w * rng.choice((9 / 16, 9 / 16, 3 / 4, 0.41)))))
        return w // step * step, h // step * step

    kind = rng.choice(("frame", "frame", "frame", "batch", "given", "lookahead", "bframe", "weighted", "serve"))
    codec = rng.choice(("hevc", "hevc", "h264"))
    depth = rng.choice((8, 8, 10))
    qp = rng.randrange(20, 41)
    if kind == "frame":
        umh = int(codec == "h264" and rng.random() < 0.5)
        w, h = size(176, 1920 if codec == "h264" else 3840, 1)
        c = dict(codec=codec, width=w, height=h, depth=depth, refs=rng.randrange(1, 5), qp=qp)
        if codec == "h264":
            return dict(c, kind=kind, range=rng.choice((16, 24, 32)), umh=umh)
        return dict(c, kind=kind, range=rng.choice((32, 64, 128)), rings=rng.choice((0, 0, 1)),
                    cross=rng.choice((0, 0, 1)), amp=rng.choice((0, 0, 0, 5, 15)) if c["refs"] < 4 else 0)
    if kind == "batch":
        groups = []
        for _ in range(rng.randrange(1, 4)):
            w, h = size(320, 1920, 2)
            groups.append("%dx%dx%d:%s:%d" % (rng.randrange(1, 7), w, h, rng.choice(("hevc", "hevc", "h264")),
                                              rng.choice((8, 8, 10))))
        return dict(kind=kind, streams=" ".join(groups), refs=rng.randrange(1, 4), qp=qp)
    if kind == "given":
        w, h = size(320, 3840, 2)
        return dict(kind=kind, codec=codec, width=w, height=h, depth=depth, refs=rng.randrange(1, 5),
                    range=rng.choice((16, 24)) if codec == "h264" else rng.choice((32, 64)), qp=qp,
                    jobs=log_int(40, 20000))
    if kind == "lookahead":
        w, h = size(176, 2560, 1)
        return dict(kind=kind, codec=codec, width=w, height=h, depth=depth, pictures=rng.randrange(1, 9))
    if kind == "bframe":
        w, h = size(176, 2560, 16)
        return dict(kind=kind, codec=codec, width=w, height=h, depth=depth, qp=qp)
    if kind == "weighted":
        w, h = size(176, 2560, 2)
        return dict(kind=kind, codec="hevc", width=w, height=h, depth=depth, qp=qp)
    w, h = size(320, 1920, 2)
    return dict(kind=kind, codec=codec, width=w, height=h, depth=depth, refs=rng.randrange(1, 3),
                range=16 if codec == "h264" else 64, qp=qp, streams=rng.randrange(1, 6), pictures=rng.randrange(1, 4))


# ---- inputs -------------------------------------------------------------------

def pictures(seed, codec, width, height, depth, count):
    """`count` pictures of a moving sequence, as pinned host arrays."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = dict(device="cuda", dtype=torch.float32)
    block, reach, sigma = (16, 12.0, 2.0) if codec == H264 else (64, 40.0, 2.0)
    scale, top = float(1 << (depth - 8)), float((1 << depth) - 1)
    xx, yy = torch.arange(width, **dev)[None, :], torch.arange(height, **dev)[:, None]
    u = torch.rand(8, 4, generator=g, **dev).cpu().tolist()
    pic = torch.full((height, width), 128.0, **dev)
    for period, amp, theta, phase in u:
        t = math.pi * theta
        pic += (4 + 36 * amp) * torch.cos(2 * math.pi * ((xx * math.cos(t) + yy * math.sin(t)) / (4 + 60 * period)
                                                         + phase))
    pic += torch.randint(-6, 7, (height, width), generator=g, device="cuda")
    pic = ((pic - pic.mean() + 128).round().clamp_(0, 255) * scale).clamp_(0, top)
    got = []
    rows = torch.arange(height, device="cuda")[:, None] // block
    cols = torch.arange(width, device="cuda")[None, :] // block
    for k in range(count):
        if k:
            mv = ((torch.rand(-(-height // block), -(-width // block), 2, generator=g, **dev) * 2 - 1) * reach * 4)
            mv = (mv.round() / 4)[rows, cols]
            sx, sy = xx + mv[..., 0], yy + mv[..., 1]
            x0, y0 = sx.floor(), sy.floor()
            fx, fy = sx - x0, sy - y0

            def at(x, y):
                return pic[y.clamp(0, height - 1).long(), x.clamp(0, width - 1).long()]

            pic = ((at(x0, y0) * (1 - fx) + at(x0 + 1, y0) * fx) * (1 - fy)
                   + (at(x0, y0 + 1) * (1 - fx) + at(x0 + 1, y0 + 1) * fx) * fy)
            pic += (torch.randn(height, width, generator=g, **dev) * sigma * scale).round()
            pic = pic.round().clamp_(0, top)
        host = torch.empty(height, width, dtype=torch.uint8 if depth == 8 else torch.int16, pin_memory=True)
        host.copy_(pic.to(host.dtype))
        got.append(host.numpy() if depth == 8 else host.numpy().view(np.uint16))
    return got


def results(n):
    """A pinned result buffer, reused from call to call as an encoder's motion field is."""
    return torch.empty(max(n, 1) * capi.RESULT_DTYPE.itemsize, dtype=torch.uint8,
                       pin_memory=True).numpy().view(capi.RESULT_DTYPE)


def rows_of(res):
    """Results as eight 32-bit numbers each."""
    return res.view(np.int32).reshape(-1, capi.RESULT_DTYPE.itemsize // 4)


def params(codec, c, given=False):
    p = rme.default_params(codec, c["qp"])
    if given:
        p.predictor_mode = capi.RME_PRED_GIVEN
    if codec == H264:
        p.h264_range = c.get("range", 16)
        p.h264_umh = c.get("umh", 0)
    else:
        p.hevc_search_range = c.get("range", 64)
        p.hevc_search_rings = c.get("rings", 0)
        p.hevc_quarter_cross = c.get("cross", 0)
        p.hevc_amp = c.get("amp", 0)
    return p


_contexts = {}


def context(case):
    """The context of a kind of work: a process keeps it, and its launch
    shapes have settled after its first calls."""
    key = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    new = key not in _contexts
    if new:
        _contexts[key] = [rme.MotionSearch(0), 0]
    return _contexts[key], new


class State:
    """Resident pictures of one sequence; given back with the state."""

    def __init__(self, held):
        self.held, self.ms, self.ids = held, held[0], []

    def new_id(self):
        self.held[1] += 1
        self.ids.append(self.held[1])
        return self.held[1]

    def upload(self, pic, codec, depth, as_ref=True):
        i = self.new_id()
        self.ms.upload(i, pic, codec, depth, as_ref=as_ref)
        return i

    def __del__(self):
        for i in self.ids:
            try:
                self.ms.release(i)
            except Exception:
                pass


def streams_of(case):
    got = []
    for part in case["streams"].split():
        size, codec, depth = part.split(":")
        n, w, h = (int(v) for v in size.split("x"))
        got.append((n, w, h, CODEC[codec], int(depth)))
    return got


def encoder_jobs(rng, codec, w, h, nref, n):
    """`n` blocks of the partition shapes, with predictors and seeds around a motion of their own."""
    shapes = np.array([(16, 16), (16, 8), (8, 16), (8, 8)] if codec == H264 else
                      [(8, 8), (16, 16), (32, 32), (64, 64), (16, 8), (8, 16), (32, 16), (16, 32), (64, 32), (16, 12),
                       (32, 24), (64, 48)])
    j = np.zeros(n, capi.JOB_DTYPE)
    s = shapes[rng.integers(len(shapes), size=n)]
    j["w"], j["h"] = s[:, 0], s[:, 1]
    j["x"] = rng.integers(0, 1 << 30, n) % ((w - s[:, 0]) // 4 + 1) * 4
    j["y"] = rng.integers(0, 1 << 30, n) % ((h - s[:, 1]) // 4 + 1) * 4
    j["ref"] = rng.integers(nref, size=n)
    j["nseeds"] = rng.integers(2, 7, n)
    true = rng.integers(-120, 121, (n, 1, 2))
    j["mvp"] = true + rng.integers(-12, 13, (n, 2, 2))
    j["seeds"] = true + rng.integers(-24, 25, (n, capi.RME_MAX_SEEDS, 2))
    j["seeds"][:, 0] = 0
    return j


# ---- prepare --------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "serve":
        return Served(case, seed)
    held, new = context(case)
    s = globals()["prepare_" + case["kind"]](State(held), case, seed)
    s.case = case
    if new:
        for _ in range(18):  # a fresh context tries its launch shapes on its first calls
            run(s)
    return s


def prepare_frame(s, c, seed):
    s.codec, s.depth = CODEC[c["codec"]], c["depth"]
    pics = pictures(seed, s.codec, c["width"], c["height"], c["depth"], c["refs"] + 1)
    s.refs = [s.upload(p, s.codec, s.depth) for p in pics[:-1]][::-1]
    s.pic, s.src = pics[-1], s.new_id()
    s.params = params(s.codec, c)
    s.ms.upload(s.src, s.pic, s.codec, s.depth)
    s.out = results(s.ms.result_count(s.src, s.refs, s.params))
    return s


def run_frame(s):
    s.ms.upload(s.src, s.pic, s.codec, s.depth)
    return rows_of(s.ms.search(s.src, s.refs, s.params, out=s.out))


def prepare_batch(s, c, seed):
    s.new, s.frames, s.params = [], [], []
    at = 0
    for n, w, h, codec, depth in streams_of(c):
        p = params(codec, dict(qp=c["qp"], range=(16 if w < 1280 else 32) if codec == H264 else
                               32 if w < 1280 else 64 if w < 2560 else 128))
        # One sequence feeds the group's streams, each stream a step further on.
        pics = pictures(seed + at, codec, w, h, depth, c["refs"] + n)
        at += 1
        ids = [s.upload(q, codec, depth) for q in pics]
        for k in range(n):
            t = c["refs"] + k
            s.new.append((ids[t], pics[t], codec, depth))
            s.frames.append((ids[t], [ids[t - 1 - r] for r in range(c["refs"])]))
            s.params.append(p)
    total = s.ms.batch_result_count(s.frames, s.params)
    s.out = torch.zeros(total, capi.RESULT_DTYPE.itemsize // 4, dtype=torch.int32, device="cuda")
    return s


def run_batch(s):
    for i, pic, codec, depth in s.new:
        s.ms.upload(i, pic, codec, depth)
    s.ms.search_batch(s.frames, s.params, out=s.out)
    return s.out


def prepare_given(s, c, seed):
    codec = CODEC[c["codec"]]
    pics = pictures(seed, codec, c["width"], c["height"], c["depth"], c["refs"] + 1)
    ids = [s.upload(p, codec, c["depth"]) for p in pics]
    s.src, s.refs = ids[-1], ids[:-1][::-1]
    s.params = params(codec, c, given=True)
    s.jobs = encoder_jobs(np.random.default_rng(seed), codec, c["width"], c["height"], c["refs"], c["jobs"])
    s.out = results(c["jobs"])
    return s


def run_given(s):
    return rows_of(s.ms.search(s.src, s.refs, s.params, jobs=s.jobs, out=s.out))


def prepare_lookahead(s, c, seed):
    s.codec, s.depth = CODEC[c["codec"]], c["depth"]
    pics = pictures(seed, s.codec, c["width"], c["height"], c["depth"], c["pictures"] + 2)
    ids = []
    for p in pics:
        ids.append(s.upload(p, s.codec, s.depth, as_ref=False))
        s.ms.lowres_build(ids[-1])
    s.all, s.new = ids, list(zip(ids[2:], pics[2:]))
    s.pairs = [(ids[t], ids[t - d]) for t in range(2, len(ids)) for d in (1, 2)]
    return s


def run_lookahead(s):
    got = []
    for i, p in s.new:
        s.ms.upload(i, p, s.codec, s.depth, as_ref=False)
        s.ms.lowres_build(i)
    found = s.ms.lowres_search_batch(s.pairs)
    for k in range(len(s.new)):
        (a, m0, _), (b, m1, _) = found[2 * k], found[2 * k + 1]
        i = s.all[k + 2]
        got.append((s.ms.lowres_intra(i), a, m0, b, m1,
                    s.ms.lowres_bi_cost(i, s.all[k + 1], m0, s.all[k], m1)))
    return [np.concatenate([g[j].reshape(-1).view(np.int32) if g[j].dtype != np.int16 else g[j].reshape(-1)
                            for g in got]) for j in range(6)]


def prepare_bframe(s, c, seed):
    codec, w, h = CODEC[c["codec"]], c["width"], c["height"]
    rng = np.random.default_rng(seed)
    pics = pictures(seed, codec, w, h, c["depth"], 3)
    ids = [s.upload(p, codec, c["depth"]) for p in pics]
    s.codec, s.src, s.refs = codec, ids[1], [ids[0], ids[2]]
    s.params = params(codec, c, given=True)
    xs, ys = np.meshgrid(np.arange(0, w - 15, 16), np.arange(0, h - 15, 16))
    n = xs.size
    s.jobs = np.zeros(n, capi.H264_BI_JOB_DTYPE if codec == H264 else capi.BI_JOB_DTYPE)
    s.jobs["x"], s.jobs["y"], s.jobs["w"], s.jobs["h"] = xs.ravel(), ys.ravel(), 16, 16
    s.jobs["ref"] = (0, 1)
    s.jobs["mv"] = rng.integers(-48, 49, size=(n, 2, 2))
    s.jobs["mvp"] = s.jobs["mv"] + rng.integers(-6, 7, size=(n, 2, 2))
    if codec == H264:
        # Vectors the joint refinement may take stay in the padded picture.
        s.jobs["limit"] = 0xFFFFFFFF
    else:
        s.jobs["list"] = rng.integers(2, size=n)
        s.blocks = np.stack([xs.ravel(), ys.ravel(), np.full(n, 16), np.full(n, 16)], 1).astype(np.int32)
        for i, p in zip(ids, pics):
            s.ms.upload_chroma(i, p[::2, ::2][:h // 2, :w // 2], p[1::2, 1::2][:h // 2, :w // 2])
    return s


def run_bframe(s):
    if s.codec == H264:
        mv, cost = s.ms.h264_bi_refine(s.src, s.refs, s.params, s.jobs)
        return mv, cost.view(np.int32)
    satd = s.ms.bi_satd(s.src, s.refs, s.params, s.jobs)
    ref = s.ms.bi_refine(s.src, s.refs, s.params, s.jobs)
    mvs = np.stack([ref["mvx"], ref["mvy"]], 1)
    chroma = s.ms.chroma_predict(s.refs[0], s.blocks, mvs)
    return satd.view(np.int32), rows_of(ref), chroma if chroma.dtype == np.uint8 else chroma.view(np.int16)


def prepare_weighted(s, c, seed):
    w, h = c["width"], c["height"]
    pics = pictures(seed, HEVC, w, h, c["depth"], 2)
    ids = [s.upload(p, HEVC, c["depth"]) for p in pics]
    s.ref, s.src, s.dst = ids[0], ids[1], s.new_id()
    s.params = params(HEVC, c, given=True)
    xs, ys = np.meshgrid(np.arange(0, w - 15, 16), np.arange(0, h - 15, 16))
    rng = np.random.default_rng(seed)
    s.jobs = np.zeros(xs.size, capi.JOB_DTYPE)
    s.jobs["x"], s.jobs["y"], s.jobs["w"], s.jobs["h"] = xs.ravel(), ys.ravel(), 16, 16
    s.jobs["nseeds"] = 3
    s.jobs["seeds"] = rng.integers(-120, 121, s.jobs["seeds"].shape)
    s.jobs["seeds"][:, 0] = 0
    s.jobs["mvp"] = s.jobs["seeds"][:, 1:3]
    return s


def run_weighted(s):
    moments = s.ms.wp_moments(s.src, s.ref)
    sad = s.ms.weighted_sad(s.src, s.ref, 72, 6, -9)
    s.ms.picture_weighted(s.ref, s.dst, 6, 72, -9)
    whole = s.ms.search(s.src, [s.dst], s.params, jobs=s.jobs)
    jobs = s.jobs.copy()
    jobs["seeds"][:, 0, 0], jobs["seeds"][:, 0, 1] = whole["int_mvx"], whole["int_mvy"]
    fine = s.ms.hevc_weighted_refine(s.src, [s.ref], s.params, jobs, 6, 72, -9)
    return moments.view(np.int64), sad, rows_of(whole), rows_of(fine)


class Served:
    """A server with its streams open and each stream's references resident."""

    def __init__(self, c, seed):
        self.case = c
        codec = CODEC[c["codec"]]
        self.ms = rme.MotionSearch(0)
        self.srv = rme.Server(self.ms, hbm_budget_bytes=40 << 30, max_frames_per_launch=4)
        p = params(codec, c)
        self.pics, self.out = [], []
        for k in range(c["streams"]):
            self.pics.append(pictures(seed + k, codec, c["width"], c["height"], c["depth"],
                                      max(c["pictures"], c["refs"])))
            if self.srv.open_stream(k, codec, c["depth"], c["width"], c["height"], p, c["refs"]) != 0:
                raise RuntimeError("the stream was refused")
            # The pictures the stream ends on come first: every pass then
            # starts from the same references.
            for pic in self.pics[k][-c["refs"]:]:
                self.srv.submit(k, pic)
            self.out.append([results(self.srv.result_count(k)) for _ in range(c["pictures"])])
        self.wait(c["streams"] * c["refs"])
        for _ in range(4):  # fill the streams' rings of resident pictures
            serve(self)

    def wait(self, n):
        got = {}
        while len(got) < n:
            for d in self.srv.poll():
                if d["status"] != 0:
                    raise RuntimeError("request failed: %r" % d["status"])
                got[d["id"]] = d["results"]
            if len(got) < n:
                time.sleep(0.00005)
        return got

    def __del__(self):
        try:
            self.srv.stop()
            self.ms.close()
        except Exception:
            pass


def serve(s):
    ids = []
    n = s.case["pictures"]
    for t in range(n):
        for k, pics in enumerate(s.pics):
            ids.append(s.srv.submit(k, pics[len(pics) - n + t], out=s.out[k][t]))
    got = s.wait(len(ids))
    return [rows_of(got[i]) for i in ids]


def run(state):
    if state.case["kind"] == "serve":
        return serve(state)
    return globals()["run_" + state.case["kind"]](state)


# ---- the work a pass cannot do without -------------------------------------------

def _search_work(codec, w, h, depth, refs, amp=0, levels=4):
    """Bytes: the picture in, it and the references read, the results out. Operations: per sample, evaluated size and
    reference at least five SAD candidates (2 each) and seventeen SATD candidates (7 each; H.264's two rings as many)."""
    bps = 1 if depth == 8 else 2
    if codec == H264:
        blocks, per = -(-w // 16) * -(-h // 16), 1
        results = blocks
    else:
        sizes = (8, 16, 32, 64)[:levels]
        units = sum((w // n) * (h // n) for n in sizes)
        units += sum((w // n) * (h // n) * 2 * bin(amp).count("1") for n in sizes if n >= 16)
        per = levels + 3 * bin(amp).count("1")
        results = units * refs
    return {"bytes": w * h * bps * (refs + 2) + results * 32, "flops": w * h * per * refs * 129}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        got = {"bytes": 0, "flops": 0}
        for n, w, h, codec, depth in streams_of(case):
            one = _search_work(codec, w, h, depth, case["refs"])
            got = {k: got[k] + n * one[k] for k in got}
        return got
    codec, w, h, depth = CODEC[case["codec"]], case["width"], case["height"], case["depth"]
    px = w * h * (1 if depth == 8 else 2)
    if kind == "frame":
        return _search_work(codec, w, h, depth, case["refs"], case.get("amp", 0))
    if kind == "serve":
        one = _search_work(codec, w, h, depth, case["refs"])
        return {k: v * case["streams"] * case["pictures"] for k, v in one.items()}
    if kind == "given":
        area = 144 if codec == H264 else 1000  # the shapes' mean
        return {"bytes": case["jobs"] * (area * 2 * (1 if depth == 8 else 2) + 100), "flops": case["jobs"] * area * 129}
    if kind == "lookahead":
        n = case["pictures"]
        return {"bytes": n * (px + px // 4 * 5 + (w // 16) * (h // 16) * 28),
                "flops": n * (w * h // 4) * (3 * 7 + 2 * (10 * 2 + 7) + 8)}
    if kind == "bframe":
        n = (w // 16) * (h // 16)
        return {"bytes": 3 * px + px // 2 + n * 88, "flops": w * h * (129 + 20)}
    n = (w // 16) * (h // 16)
    return {"bytes": 4 * px + n * 264, "flops": w * h * (10 + 2 * 129)}


def exact(case, seed):
    """Every output is a whole number."""
    return None
