// The H.264 STANDALONE search in its row form: a CTA owns a row of
// macroblocks and searches it left to right, four warps per reference.
//
// What a macroblock's search computes is p_mb's search section
// (h264_analyse.rs:1884-1975), as h264_task does it with one warp: the
// neighbours' vectors as candidates, Search::int_search and Search::refine
// (h264_hpel.rs:789-1021) per reference, the reference of least cost. Its
// candidates, order, tie-breaks and counts are the same.
//
// Macroblocks form a wavefront (A, B, C and D neighbours), so a picture is a
// chain of mbw + 2 mbh macroblocks and bound by one macroblock's latency.
// Against one warp per macroblock (the dataflow form):
//   - a reference has four warps, eight lanes per candidate: up to sixteen
//     candidates of a step at once, two rows (SAD) or two 4x4 tiles (SATD) a
//     lane, one named barrier a step (a refinement step but the first has at
//     most eight: sixteen lanes and a tile a lane);
//   - the walk and the refinement read the four planes around the seeds' best
//     point from shared memory, staged once a macroblock while it is needed;
//     from the planes a step's candidates, on lines of their own, are up to 32
//     passes through L1 a load: staging took the search of four 10-bit 720p
//     references from 3.10 to 2.41 ms, the UMH points' samples that of 1080p
//     from 3.92 to 2.61 ms;
//   - references are searched side by side, each by its own four warps; the
//     refine_ratio gate, the only tie between them, needs the whole-sample
//     costs alone, one CTA barrier;
//   - a hexagon step also scores the square around the same centre, which is
//     the walk's last step when the hexagon has settled;
//   - the UMH points are scored without a decision between them: no two of
//     them coincide and none is the start, so the one point the reference
//     leaves out, the best so far, is never among them, and the outcome is
//     the least cost, first reached;
//   - a step is its instructions' latency more than its work: counts stay in
//     the lanes, a lane's part of a sum goes to shared memory instead of three
//     shuffles, offsets that do not change are kept (CIF 0.43 -> 0.36 ms);
//   - a neighbour's result is one published word (tag, reference, vector),
//     loaded a macroblock ahead, and the next source block is staged behind
//     the search.
// Measured on one B200, the search kernel alone, the dataflow form first:
// CIF, one reference, medium tier 1.60 -> 0.36 ms; 1080p, three references,
// UMH +-24 28.3 -> 2.2 ms; 64 720p pictures of two references in one launch
// 14.5 -> 5.9 ms.
#include <algorithm>

#include "rme_search_impl.cuh"

namespace rme {
namespace {

constexpr int kRefThreads = 128;  // threads per reference
constexpr int kSlots16 = 16;      // candidates a step scores at once

// Small tables as hex digits (the lowest first), so that lanes with entries of
// their own do not queue at the constant cache: the hexagon's and the square's
// offsets + 2, the UMH hexagon's + 2, the refinement ring's + 1.
__device__ __forceinline__ int digit(unsigned long long t, int k) { return (int)((t >> (4 * k)) & 15u); }
__device__ __forceinline__ int digit(uint32_t t, int k) { return (int)((t >> (4 * k)) & 15u); }
__device__ __forceinline__ int hex_x(int k) { return digit(0x134310u, k) - 2; }
__device__ __forceinline__ int hex_y(int k) { return digit(0x442002u, k) - 2; }
__device__ __forceinline__ int square_x(int k) { return digit(0x32131321u, k) - 2; }
__device__ __forceinline__ int square_y(int k) { return digit(0x33322111u, k) - 2; }
__device__ __forceinline__ int hex12_x(int k) { return digit(0x404031314400ull, k) - 2; }
__device__ __forceinline__ int hex12_y(int k) { return digit(0x4400441313ull, k) - 2; }
__device__ __forceinline__ int ring_x(int k) { return digit(0x20201201u, k) - 1; }
__device__ __forceinline__ int ring_y(int k) { return digit(0x22002110u, k) - 1; }
// The quarter-sample table (8.4.2.2.1): per position (fy * 4 + fx) a digit
// plane * 4 + dy * 2 + dx of the first view and of the second; positions
// 0, 2, 8 and 10 have one view.
constexpr unsigned long long kView1 = 0x9c88cc8844404400ull, kView2 = 0x666290c09c881040ull;
constexpr uint32_t kTwoViews = 0xfafau;

// A reference's staged samples: its four planes kWinM samples around the seeds'
// best point, in rows of an odd number of 16-byte chunks (eight rows on eight
// different banks); the planes a chunk apart more, so that candidates of
// different planes fall on different banks.
constexpr int kWinM = 8, kWinRows = 16 + 2 * kWinM;
template <class S>
struct Win {
  static constexpr int CH = sizeof(S) == 1 ? 3 : 5;  // chunks that hold kWinRows samples from any byte on
  static constexpr int PITCH = CH * 4, PLANE = kWinRows * PITCH + 4, WORDS = 4 * PLANE;
  static_assert((kWinRows * (int)sizeof(S) + 15 + 4) / 16 <= CH && CH % 2 == 1, "row width");
};

// The UMH points' offsets: the cross, then the twelve-point hexagons.
__device__ __forceinline__ int umh_points(int range) { return 4 * (range / 2) + 12 * (range / 4); }
__device__ __forceinline__ void umh_point(int i, int range, int& x, int& y) {
  const int ncross = 4 * (range / 2);
  if (i < ncross) {
    const int r = 2 * (i / 4 + 1), k = i & 3;
    x = k == 0 ? -r : k == 1 ? r : 0;
    y = k == 2 ? -r : k == 3 ? r : 0;
  } else {
    const int j = i - ncross, r = 2 * (j / 12 + 1), k = j % 12;
    x = hex12_x(k) * r;
    y = hex12_y(k) * r;
  }
}
// The UMH points' samples staged in the same memory, where they fit (ranges to
// 25): rows of an odd number of chunks that hold the points from any byte on
// and one word more.
template <class S>
struct UmhWindow {
  int reach, rows, chunks;
  bool fit;
  __device__ __forceinline__ explicit UmhWindow(int range)
      : reach(max(2 * (range / 2), 4 * (range / 4))),
        rows(16 + 2 * reach),
        chunks(((rows * (int)sizeof(S) + 31) / 16) | 1),
        fit(range < 26 && rows * chunks * 4 <= Win<S>::WORDS) {}
};

struct RefResult {
  uint32_t cost, satd, icost;
  int mx, my, imx, imy;
};

template <class S>
struct RowSmem {
  alignas(16) uint32_t win[RME_MAX_REFS][Win<S>::WORDS];
  uint32_t src[2][16 * 16 * sizeof(S) / 4];
  alignas(16) uint32_t part[RME_MAX_REFS][2][kRefThreads];  // a step's partial sums, two steps in turn
  uint32_t umh[128];                  // UMH: where each point's samples start in the window
  uint32_t best[RME_MAX_REFS][4][2];  // UMH: each warp's least cost and its point
  uint32_t icost[2][RME_MAX_REFS];    // whole-sample costs, reference cost included
  RefResult fin[2][RME_MAX_REFS];
  uint32_t nsad[2], nsatd[2];
  volatile uint32_t lost;             // a wait gave up
  uint32_t entry;
};

// A macroblock's published word: the launch's tag in bits 34..63, the
// reference in 32..33, the vector in the low half.
__device__ __forceinline__ bool row_word_ok(unsigned long long w, uint32_t tag) {
  return ((uint32_t)(w >> 32) & ~3u) == tag;
}
// Waits for a word already loaded once: at most L.wait_polls polls, then the
// status word's timeout bit; fewer once the launch has failed elsewhere. Returns
// the word, of another tag where it gave up.
__device__ __noinline__ unsigned long long poll_row_word(const LaunchDesc& L, const unsigned long long* p, uint32_t tag,
                                                         unsigned long long w) {
  uint32_t ns = 32;
  for (uint32_t it = 0; !row_word_ok(w, tag); ++it) {
    const bool out = it >= L.wait_polls;
    if (out || ((it & 63u) == 63u && ld_relaxed32(L.status) != 0u)) {
      if (out) atomicOr(L.status, kStatusWaitTimeout);
      break;
    }
    if (it >= 16) {
      __nanosleep(ns);
      if (ns < 256) ns <<= 1;
    }
    w = ld_relaxed64(p);
  }
  return w;
}
// Sets `lost` where the wait gives up. Every thread waits by itself and says so in
// its part of the search's first sums, which all of a reference's warps read:
// they then drop what they took from words that may differ (they could take
// different numbers of steps between their barriers), for the rest of the row.
// 8 bits: at the macroblock's end the CTA leaves. Deeper: the row goes on, its
// later waits giving up after 64 polls (the check costs four references of
// 720p 1.6 %; without it CIF's schedule loses 2 %).
constexpr uint32_t kLost = 1u << 27;  // above any sum of eight parts
__device__ __forceinline__ void wait_row_word(const LaunchDesc& L, const unsigned long long* p, uint32_t tag,
                                              unsigned long long& w, uint32_t& lost) {
  if (row_word_ok(w, tag)) return;
  w = poll_row_word(L, p, tag, w);
  if (!row_word_ok(w, tag)) lost = kLost;
}

// One reference's search of a macroblock, by the 128 threads of its group.
template <class S>
struct RefSearch {
  static constexpr int WR = 16 * (int)sizeof(S) / 4;  // words of a source row
  RowSmem<S>& sm;
  const uint32_t* src;
  const DevPlanes R;  // copies: the barriers between steps would have them read again
  const uint16_t* tab;
  const int range, umh, dia, qpel_diamond;
  H264Blk B;
  const S* org;
  int g, warp, lane, sub, slot;  // group; warp in it; this lane's part of candidate `slot`
  int height;         // the plane's coded height
  uint32_t* win;      // this reference's window
  int wx = 0, wy = 0, wofs = 0;  // its centre; the centre's first byte in a row
  int buf = 0;
  uint32_t nsad = 0, nsatd = 0;  // candidates scored: this lane's eighths, sixteenths
  uint32_t s0[WR], s1[WR];       // source rows sub and sub + 8

  __device__ __forceinline__ void sync() { asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(kRefThreads) : "memory"); }

  // This lane's part of a candidate's SAD: rows sub and sub + 8.
  __device__ __forceinline__ uint32_t sad(int fx, int fy) {
    const S* rp = org + (ptrdiff_t)(fy + sub) * R.stride + fx;
    uint32_t a[WR], b[WR];
    ldrow<WR>(rp, a);
    ldrow<WR>(rp + (ptrdiff_t)8 * R.stride, b);
    return sad2(a, b);
  }
  // Copies rows of 16-byte chunks around whole-sample offset (x, y) into the
  // window, unwaited. What lies outside the padded plane is clamped to it: no
  // candidate reads it.
  __device__ __forceinline__ void copy_chunk(uint32_t* dst, int plane, int row, int chunk) {
    const int stride = R.stride * (int)sizeof(S);
    row = min(max(row, -kH264Pad), height + kH264Pad - 1);
    chunk = min(max(chunk, 0), stride / 16 - 1);
    const char* p = reinterpret_cast<const char*>(plane_at<S>(R, plane, -kH264Pad, row)) + chunk * 16;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(p)
                 : "memory");
  }
  // The four planes around (x, y): plane 0 as one copy group, the others the next.
  __device__ __forceinline__ void stage(int x, int y) {
    typedef Win<S> W;
    wx = x;
    wy = y;
    const int byte = (B.x + x - kWinM + kH264Pad) * (int)sizeof(S), c0 = byte >> 4;
    wofs = (byte & 15) + kWinM * (int)sizeof(S);
    const int t = warp * 32 + lane, row0 = B.y + y - kWinM;
    constexpr int N1 = kWinRows * W::CH;
    for (int i = t; i < N1; i += kRefThreads)
      copy_chunk(win + (i / W::CH) * W::PITCH + (i % W::CH) * 4, 0, row0 + i / W::CH, c0 + i % W::CH);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = t; i < 3 * N1; i += kRefThreads) {
      const int q = i / W::CH, pl = 1 + q / kWinRows, row = q % kWinRows;
      copy_chunk(win + pl * W::PLANE + row * W::PITCH + (i % W::CH) * 4, pl, row0 + row, c0 + i % W::CH);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // Whether points lo .. hi samples from (x, y) lie in the window.
  __device__ __forceinline__ bool in_window(int x, int y, int lo, int hi) {
    return min(x - wx, y - wy) >= lo - kWinM && max(x - wx, y - wy) <= kWinM - hi;
  }
  // N words of the window from byte `byte` of the row at `w`.
  template <int N>
  __device__ __forceinline__ void win_words(const uint32_t* w, int byte, uint32_t (&out)[N]) {
    const uint32_t* p = w + (byte >> 2);
    const uint32_t sh = (uint32_t)(byte & 3) * 8u;
    uint32_t v[N + 1];
#pragma unroll
    for (int k = 0; k <= N; ++k) v[k] = p[k];
#pragma unroll
    for (int k = 0; k < N; ++k) out[k] = __funnelshift_r(v[k], v[k + 1], sh);
  }
  // Two chains: one sum after the other is the longest of a step.
  __device__ __forceinline__ uint32_t sad2(const uint32_t (&a)[WR], const uint32_t (&b)[WR]) {
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int k = 0; k < WR; ++k) {
      lo = vsad(s0[k], a[k], lo, S());
      hi = vsad(s1[k], b[k], hi, S());
    }
    return lo + hi;
  }
  // As sad, a point of the window.
  __device__ __forceinline__ uint32_t win_sad(int fx, int fy) {
    const uint32_t* w = win + (fy - wy + kWinM + sub) * Win<S>::PITCH;
    const int byte = wofs + (fx - wx) * (int)sizeof(S);
    uint32_t a[WR], b[WR];
    win_words<WR>(w, byte, a);
    win_words<WR>(w + 8 * Win<S>::PITCH, byte, b);
    return sad2(a, b);
  }
  // NT 4x4 tiles of the window side by side (tile row ty, from tile column tx
  // on): SATD against one view or the average of two. The lower tiles' rows
  // are taken in the order 2 3 0 1, for the banks' sake: a Hadamard sum of
  // magnitudes is the same when row numbers are XORed with a constant.
  template <int NT>
  __device__ __forceinline__ uint32_t win_satd(int mx, int my, int ty, int tx) {
    constexpr int WPT = (int)sizeof(S), WPS = NT * WPT;
    const int pos = (my & 3) * 4 + (mx & 3), a = digit(kView1, pos), b = digit(kView2, pos), flip = ty & 2;
    const int row = (my >> 2) - wy + kWinM + ty * 4, byte = wofs + ((mx >> 2) - wx + tx * 4) * (int)sizeof(S);
    uint32_t pw[4][WPS];
    const uint32_t* w = win + (a >> 2) * Win<S>::PLANE + (row + ((a >> 1) & 1)) * Win<S>::PITCH;
#pragma unroll
    for (int r = 0; r < 4; ++r) win_words<WPS>(w + (r ^ flip) * Win<S>::PITCH, byte + (a & 1) * (int)sizeof(S), pw[r]);
    if ((kTwoViews >> pos) & 1u) {
      w = win + (b >> 2) * Win<S>::PLANE + (row + ((b >> 1) & 1)) * Win<S>::PITCH;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        uint32_t q[WPS];
        win_words<WPS>(w + (r ^ flip) * Win<S>::PITCH, byte + (b & 1) * (int)sizeof(S), q);
#pragma unroll
        for (int k = 0; k < WPS; ++k) pw[r][k] = vavg(pw[r][k], q[k], S());
      }
    }
    uint32_t v = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      uint32_t sw[4][WPT], qw[4][WPT];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int k = 0; k < WPT; ++k) {
          sw[r][k] = src[(ty * 4 + (r ^ flip)) * WR + (tx + t) * WPT + k];
          qw[r][k] = pw[r][t * WPT + k];
        }
      v += satd4x4<WPT>(sw, qw);
    }
    return v;
  }
  // A step's candidates, LANES threads each: every thread gives its part of
  // its candidate's cost (kNone where there is no candidate, whose cost is
  // then above any other's), and lane l gets cost << 4 | slot of slot l (mod
  // the number of slots). A cost is below 2^23 at every depth (twelve bits:
  // sixteen tiles' SATD of at most 262080 and two 16-bit rates).
  static constexpr uint32_t kNone = 1u << 23;
  template <int LANES>
  __device__ __forceinline__ uint32_t share(uint32_t part) {
    uint32_t lost;
    return share<LANES>(part, lost);
  }
  template <int LANES>
  __device__ __forceinline__ uint32_t share(uint32_t part, uint32_t& lost) {  // lost: of lane l's slot
    uint32_t* c = sm.part[g][buf];
    buf ^= 1;
    c[warp * 32 + lane] = part;
    sync();
    const int k = lane & (kRefThreads / LANES - 1);
    uint32_t v = 0;
#pragma unroll
    for (int i = 0; i < LANES / 4; ++i) {
      // Each slot from another chunk on: eight lanes' loads on all banks.
      const uint4 q = reinterpret_cast<const uint4*>(c + k * LANES)[(i + k * LANES / 32) & (LANES / 4 - 1)];
      v += (q.x + q.y) + (q.z + q.w);
    }
    lost = v >> 27;
    return v << 4 | (uint32_t)k;
  }
  __device__ __forceinline__ uint32_t rate(int qx, int qy) {
    const int dx = min(max(qx - B.px, -kMvSpan), kMvSpan), dy = min(max(qy - B.py, -kMvSpan), kMvSpan);
    return (uint32_t)__ldg(&tab[dx + kMvSpan]) + (uint32_t)__ldg(&tab[dy + kMvSpan]);
  }

  // This lane's part of the cost of the point (ox, oy), at most two samples
  // each way, from (x, y).
  __device__ __forceinline__ uint32_t score(int x, int y, int ox, int oy, bool ok) {
    const uint32_t rt = rate((x + ox) * 4, (y + oy) * 4);
    uint32_t v = 0;
    if ((uint32_t)(x - wx + kWinM - 2) <= 2u * kWinM - 4 && (uint32_t)(y - wy + kWinM - 2) <= 2u * kWinM - 4)
      v = win_sad(x + ox, y + oy);  // without a branch on ok: a point outside the box is in the window all the same
    else if (ok)
      v = sad(x + ox, y + oy);
    return ok ? v + (sub == 0 ? rt : 0u) : kNone;
  }

  // Search::int_search: lane k + 1 of every warp holds candidate k of ncand.
  __device__ __forceinline__ void whole(int ncand, int cand_x, int cand_y, uint32_t mark, int& imx, int& imy,
                                        uint32_t& icost) {
    const int pxr = min(max((B.px + 2) >> 2, B.lx), B.hx), pyr = min(max((B.py + 2) >> 2, B.ly), B.hy);
    const int qx = lane == 0 ? pxr : min(max((cand_x + 2) >> 2, B.lx), B.hx);
    const int qy = lane == 0 ? pyr : min(max((cand_y + 2) >> 2, B.ly), B.hy);
    // A candidate on the predictor's point or an earlier candidate's is
    // skipped (`tried`).
    bool skip = lane > 0 && qx == pxr && qy == pyr;
#pragma unroll
    for (int j = 1; j <= 8; ++j) {
      const int ox = __shfl_sync(kFull, qx, j), oy = __shfl_sync(kFull, qy, j);
      skip |= j < lane && ox == qx && oy == qy;
    }
    const uint32_t keep = __ballot_sync(kFull, lane <= ncand && !skip);
    int bx, by;
    uint32_t bcost;
    {
      const bool ok = (keep >> slot) & 1u;
      const int fx = __shfl_sync(kFull, qx, slot), fy = __shfl_sync(kFull, qy, slot);
      const uint32_t rt = rate(fx * 4, fy * 4);
      uint32_t lost;
      const uint32_t c = share<8>(mark + (ok ? sad(fx, fy) + (sub == 0 ? rt : 0u) : kNone), lost);
      const uint32_t m = __reduce_min_sync(kFull, c);
      nsad += ok;
      bcost = m >> 4;
      bx = __shfl_sync(kFull, qx, m & 15);
      by = __shfl_sync(kFull, qy, m & 15);
      if (__builtin_expect(__any_sync(kFull, lost != 0u), 0)) {
        sm.lost = 1u;
        B.px = B.py = bx = 0;
        by = min(max(0, B.ly), B.hy);
      }
    }
    const int x0 = max(bx - range, B.lx), x1 = min(bx + range, B.hx), y0 = max(by - range, B.ly),
              y1 = min(by + range, B.hy);
    // The box's columns (the start's among them) and rows: none where a
    // vertical range of -1 leaves the window empty.
    const uint32_t xn = (uint32_t)(x1 - x0 + 1), yn = (uint32_t)max(y1 - y0 + 1, 0);
    auto inside = [&](int x, int y) { return (uint32_t)(x - x0) < xn && (uint32_t)(y - y0) < yn; };
    if (umh) {
      const int cx = bx, cy = by, total = umh_points(range);
      uint32_t mc = kInf, mi = 0xffffffffu;  // this lane's least cost, its first point
      const UmhWindow<S> U(range);
      if (U.fit) {
        // The points' samples staged: a warp's four candidates lie on 32 lines
        // of the plane, each a pass of its own through L1.
        const int byte0 = (B.x + cx - U.reach + kH264Pad) * (int)sizeof(S), lr = lane / U.chunks,
                  lc = lane - lr * U.chunks, per = 32 / U.chunks;
        for (int r = warp * per + lr; lr < per && r < U.rows; r += 4 * per)
          copy_chunk(win + (r * U.chunks + lc) * 4, 0, B.y + cy - U.reach + r, (byte0 >> 4) + lc);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        sync();
        // Eight points for each lane (those past the last and those outside the
        // box count for nothing below); then the sums are turned, so that each
        // lane has one point's: slot's of pass `sub`.
        const uint32_t* w0 = win + sub * U.chunks * 4;
        uint32_t acc[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int at = (int)sm.umh[u * kSlots16 + slot] + (byte0 & 15);
          uint32_t a[WR], b[WR];
          win_words<WR>(w0, at, a);
          win_words<WR>(w0 + 8 * U.chunks * 4, at, b);
          acc[u] = sad2(a, b);
        }
#pragma unroll
        for (int h = 4; h > 0; h >>= 1)
#pragma unroll
          for (int u = 0; u < h; ++u) {
            const bool up = sub & h;
            const uint32_t give = up ? acc[u] : acc[u + h], keep = up ? acc[u + h] : acc[u];
            acc[u] = keep + __shfl_xor_sync(kFull, give, h);
          }
        const int i = sub * kSlots16 + slot;
        int x, y;
        umh_point(i, range, x, y);
        x += cx;
        y += cy;
        const bool ok = i < total && inside(x, y);
        nsad += ok ? 8 : 0;
        const uint32_t rt = rate(x * 4, y * 4);
        if (ok) {
          mc = acc[0] + rt;
          mi = (uint32_t)i;
        }
      } else {
#pragma unroll 2
        for (int i0 = 0; i0 < total; i0 += kSlots16) {
          const int i = i0 + slot;
          int x, y;
          umh_point(i, range, x, y);
          x += cx;
          y += cy;
          const bool ok = i < total && inside(x, y);
          uint32_t v = ok ? sad(x, y) : 0u;
          v += __shfl_xor_sync(kFull, v, 4);
          v += __shfl_xor_sync(kFull, v, 2);
          v += __shfl_xor_sync(kFull, v, 1);
          nsad += ok;
          const uint32_t c = v + rate(x * 4, y * 4);
          if (ok && c < mc) {
            mc = c;
            mi = (uint32_t)i;
          }
        }
      }
      uint32_t m = __reduce_min_sync(kFull, mc);
      uint32_t at = __reduce_min_sync(kFull, mc == m ? mi : 0xffffffffu);
      if (lane == 0) {
        sm.best[g][warp][0] = m;
        sm.best[g][warp][1] = at;
      }
      sync();
      const uint32_t wm = lane < 4 ? sm.best[g][lane][0] : kInf, wi = lane < 4 ? sm.best[g][lane][1] : 0xffffffffu;
      m = __reduce_min_sync(kFull, wm);
      at = __reduce_min_sync(kFull, wm == m ? wi : 0xffffffffu);
      if (m < bcost) {
        bcost = m;
        umh_point((int)at, range, bx, by);
        bx += cx;
        by += cy;
      }
    }
    // The steps' samples staged around the best point so far.
    stage(bx, by);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    sync();
    // A step's points around the best: offset of slot k.
    if (dia) {
      for (int it = 0; it < range; ++it) {
        auto off = [](int k, int& ox, int& oy) {
          ox = k == 0 ? -1 : k == 1 ? 1 : 0;
          oy = k == 2 ? -1 : k == 3 ? 1 : 0;
        };
        int ox, oy;
        off(slot, ox, oy);
        const bool ok = slot < 4 && inside(bx + ox, by + oy);
        const uint32_t m = __reduce_min_sync(kFull, share<8>(score(bx, by, ox, oy, ok)));
        nsad += ok;
        if (!(m >> 4 < bcost)) break;
        bcost = m >> 4;
        off(m & 15, ox, oy);
        bx += ox;
        by += oy;
      }
    } else {
      // Slots 0..5 the hexagon (after a step in direction d only d - 1, d,
      // d + 1 are new, in that order), 6..13 the square.
      auto turn = [](int d, int k) {  // direction d + k - 1 of the six
        const int e = d + k - 1;
        return e < 0 ? 5 : e > 5 ? 0 : e;
      };
      int ox = slot < 6 ? hex_x(slot) : slot < 14 ? square_x(slot - 6) : 0;
      int oy = slot < 6 ? hex_y(slot) : slot < 14 ? square_y(slot - 6) : 0;
      int dir = -1, nhex = 6;
      for (int it = 0;; ++it) {
        const bool ok = (slot < 6 ? slot < nhex : slot < 14) && inside(bx + ox, by + oy);
        const uint32_t c = share<8>(score(bx, by, ox, oy, ok));
        uint32_t m = __reduce_min_sync(kFull, (lane & 15) < 6 ? c : kInf);
        nsad += ok && slot < 6;
        if (!(m >> 4 < bcost)) {  // the hexagon has settled: the square is the last step
          nsad += ok && slot >= 6;
          m = __reduce_min_sync(kFull, (lane & 15) < 6 ? kInf : c);
          if (m >> 4 < bcost) {
            bcost = m >> 4;
            bx += square_x((int)(m & 15) - 6);
            by += square_y((int)(m & 15) - 6);
          }
          break;
        }
        bcost = m >> 4;
        dir = dir < 0 ? (int)(m & 15) : turn(dir, m & 15);
        bx += hex_x(dir);
        by += hex_y(dir);
        if (slot < 6) {
          const int e = turn(dir, min(slot, 2));
          ox = hex_x(e);
          oy = hex_y(e);
        }
        nhex = it + 1 < range ? 3 : 0;
      }
    }
    imx = bx * 4;
    imy = by * 4;
    icost = bcost;
  }

  // Search::refine from (smx, smy), as h264_refine: the start with the first
  // ring in one step.
  __device__ __forceinline__ void refine(int smx, int smy, int hpel, int qpel, int& omx, int& omy, uint32_t& osatd,
                                         uint32_t& ocost) {
    // The window in quarter samples (no row of an empty one).
    const int qlx = B.lx * 4, qly = B.ly * 4;
    const uint32_t qnx = (uint32_t)((B.hx - B.lx) * 4 + 1), qny = (uint32_t)max((B.hy - B.ly) * 4 + 1, 0);
    int bmx = smx, bmy = smy;
    uint32_t bc = kInf;
    bool first = true;
    // This lane's ring point in the first step (the start is slot 0) and in one
    // of sixteen lanes a candidate.
    const int rx0 = ring_x((slot - 1) & 7), ry0 = ring_y((slot - 1) & 7);
    const int rx1 = ring_x(warp * 2 + (lane >> 4)), ry1 = ring_y(warp * 2 + (lane >> 4));
    // No step leaves the start by more than `far` samples. A walk that went
    // too far for the window has it staged anew.
    const int far = (2 * hpel + qpel + 3) / 4;
    bool staged = in_window(smx >> 2, smy >> 2, far, far + 1);
    // (A vector that wraps at 16 bits lies elsewhere: its samples are read from the plane.)
    const bool near = max(abs(smx), abs(smy)) + 4 * far < 32768;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    sync();
    staged = staged && near;
    if (!staged && near && far + 1 <= kWinM) {
      stage(smx >> 2, smy >> 2);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      sync();
      staged = true;
    }
    for (int s = 0; s < 2; ++s) {
      const int step = s == 0 ? 2 : 1, iters = s == 0 ? hpel : qpel;
      const int pts = (step == 1 && qpel_diamond) ? 4 : 8;
      int prevx = 1 << 20, prevy = 1 << 20;  // none yet
      for (int it = 0; it < iters || first; ++it) {
        const int cmx = bmx, cmy = bmy;
        const bool ring = it < iters;
        const int base = first ? 1 : 0, n = base + (ring ? pts : 0);
        auto vec = [&](int c, int& mx, int& my) {  // slot c's vector
          mx = cmx;
          my = cmy;
          if (c >= base) {
            mx = (int)(int16_t)(cmx + ring_x((c - base) & 7) * step);
            my = (int)(int16_t)(cmy + ring_y((c - base) & 7) * step);
          }
        };
        // At most eight candidates, all but the first step's nine: sixteen
        // threads each, a tile a thread.
        const bool wide = staged && !first;
        const int sl = wide ? warp * 2 + (lane >> 4) : slot, part = wide ? lane & 15 : sub;
        int mx, my;
        if (wide) {
          mx = (int)(int16_t)(cmx + rx1 * step);
          my = (int)(int16_t)(cmy + ry1 * step);
        } else if (first && slot > 0) {
          mx = (int)(int16_t)(cmx + rx0 * step);
          my = (int)(int16_t)(cmy + ry0 * step);
        } else {
          vec(sl, mx, my);
        }
        bool ok = sl < n;
        if (sl >= base)
          ok = ok && (uint32_t)(mx - qlx) < qnx && (uint32_t)(my - qly) < qny &&
               !((uint32_t)(mx - prevx + step) <= 2u * step && (uint32_t)(my - prevy + step) <= 2u * step);
        const uint32_t rt = rate(mx, my);
        uint32_t v = kNone;
        if (ok) {
          if (wide) {
            v = win_satd<1>(mx, my, part >> 2, part & 3);
          } else if (staged) {
            v = win_satd<2>(mx, my, part >> 1, (part & 1) * 2);
          } else {
            const int xi = B.x + (mx >> 2), yi = B.y + (my >> 2);
            const int pos = (my & 3) * 4 + (mx & 3), a = digit(kView1, pos), b = digit(kView2, pos);
            const S* p1 = plane_at<S>(R, a >> 2, xi + (a & 1), yi + ((a >> 1) & 1));
            const S* p2 =
                (kTwoViews >> pos) & 1u ? plane_at<S>(R, b >> 2, xi + (b & 1), yi + ((b >> 1) & 1)) : nullptr;
            v = satd_strips<S, 2>(src, WR, 4, 4, p1, p2, R.stride, 8, sub);
          }
          v += part == 0 ? rt : 0u;
        }
        const uint32_t m = __reduce_min_sync(kFull, wide ? share<16>(v) : share<8>(v));
        nsatd += ok ? (wide ? 1 : 2) : 0;
        if (m >> 4 < bc) {
          bc = m >> 4;
          vec(m & 15, bmx, bmy);
        }
        first = false;
        if (!ring) break;
        if (bmx == cmx && bmy == cmy) break;
        prevx = cmx;
        prevy = cmy;
      }
    }
    omx = bmx;
    omy = bmy;
    osatd = bc - rate(bmx, bmy);
    ocost = bc;
  }
};

// False, for the whole CTA, where a wait gave up: the launch has failed.
template <class S>
__device__ bool h264_row(const LaunchDesc& L, const FrameDesc& F, int my, RowSmem<S>& sm, int tid,
                         unsigned long long (&cnt)[3]) {
  constexpr int WR = RefSearch<S>::WR, NSRC = 16 * WR;
  const int lane = tid & 31, g = tid >> 7, warp = (tid >> 5) & 3;
  const int mbw = F.width / 16, nref = F.nref;
  const uint32_t tag = F.tag;
  const unsigned long long* up = F.mvf + (ptrdiff_t)(my - 1) * mbw;
  auto load_src = [&](int mx) -> uint32_t {  // word tid of the macroblock's rows (16-byte aligned rows)
    const S* o = plane_at<S>(F.src, 0, mx * 16, my * 16 + tid / WR);
    return RME_LD32(reinterpret_cast<const uint32_t*>(o) + tid % WR);
  };
  if (tid < NSRC) sm.src[0][tid] = load_src(0);
  if (F.umh && tid < 128) {
    const UmhWindow<S> U(F.range);
    int x = 0, y = 0;
    if (tid < umh_points(F.range)) umh_point(tid, F.range, x, y);
    sm.umh[tid] = (uint32_t)((y + U.reach) * U.chunks * 16 + (x + U.reach) * (int)sizeof(S));
  }
  if (tid < 2) sm.nsad[tid] = sm.nsatd[tid] = 0u;
  unsigned long long wd = 0, wb = 0, wc = 0;  // the D, B and C macroblocks' words
  uint32_t lost = 0;                          // a wait of this thread gave up
  if (my > 0) {
    wb = ld_relaxed64(up);
    if (mbw > 1) wc = ld_relaxed64(up + 1);
    wait_row_word(L, up, tag, wb, lost);
    __syncwarp();
  }
  Nb A{false, -1, 0, 0};
  // What does not change along the row, read once (the frame's description is
  // in global memory, and the steps' barriers would have it read again).
  const int gr = min(g, nref - 1), width = F.width, height = F.height, pad = F.pad, vr = F.vr;
  const int hpel = F.hpel_iters, qpel = F.qpel_iters;
  const float ratio = F.refine_ratio;
  const uint32_t ref_cost = F.ref_cost[gr];
  RefSearch<S> q{sm, sm.src[0], F.ref[gr], F.tab, F.range, F.umh, F.dia, F.qpel_diamond};
  q.g = g;
  q.warp = warp;
  q.lane = lane;
  q.sub = lane & 7;
  q.slot = warp * 4 + (lane >> 3);
  q.height = height;
  q.win = sm.win[gr];
  q.B.w = q.B.h = 16;
  q.B.y = my * 16;
  q.B.ly = max(4 - pad - q.B.y, -vr);  // search_bounds (h264_hpel.rs:476-488)
  q.B.hy = min(height + pad - 20 - q.B.y, vr);
  // A macroblock's result, written a macroblock later, when the counts have
  // met: only its vector is waited for.
  int ended = 0;  // its reference
  auto write = [&](int mx) {
    const RefResult& w = sm.fin[mx & 1][ended];
    write_result(&F.out[my * mbw + mx], w.mx, w.my, ended, w.cost, w.satd, w.imx, w.imy, w.icost, sm.nsad[mx & 1],
                 sm.nsatd[mx & 1], 0);
    cnt[0] += 1;
    cnt[1] += sm.nsad[mx & 1];
    cnt[2] += sm.nsatd[mx & 1];
    sm.nsad[mx & 1] = sm.nsatd[mx & 1] = 0u;
  };
  __syncthreads();
  for (int mx = 0; mx < mbw; ++mx) {
    const int par = mx & 1;
    const bool has_c = my > 0 && mx + 1 < mbw;
    if (has_c) wait_row_word(L, up + mx + 1, tag, wc, lost);
    __syncwarp();
    // The next macroblock's C word and source, on their way during the search.
    unsigned long long wn = 0;
    if (my > 0 && mx + 2 < mbw) wn = ld_relaxed64(up + mx + 2);
    uint32_t nsrc = 0;
    if (tid < NSRC && mx + 1 < mbw) nsrc = load_src(mx + 1);
    auto nb = [](bool avail, unsigned long long w) {
      Nb m{false, -1, 0, 0};
      if (avail) {
        m.avail = true;
        m.ref = (int)((w >> 32) & 3u);
        m.x = mvx_of((uint32_t)w);
        m.y = mvy_of((uint32_t)w);
      }
      return m;
    };
    const Nb Bn = nb(my > 0, wb), C = nb(has_c, wc), D = nb(my > 0 && mx > 0, wd);
    const Nb Cc = C.avail ? C : D;
    if (g < nref) {
      // p_skip_mv, then cands = [skip_mv, 0, distinct A, B, C] and a further
      // reference's own predictor: lane k + 1 holds candidate k.
      int skx = 0, sky = 0;
      if (A.avail && Bn.avail && !(A.ref == 0 && A.x == 0 && A.y == 0) && !(Bn.ref == 0 && Bn.x == 0 && Bn.y == 0))
        median_mvp(A, Bn, Cc, 0, skx, sky);
      auto same = [](const Nb& p, const Nb& q) { return p.x == q.x && p.y == q.y; };
      const bool va = A.avail, vb = Bn.avail && !(va && same(A, Bn)),
                 vc = C.avail && !(va && same(A, C)) && !(vb && same(Bn, C));
      const int ia = 2, ib = ia + va, ic = ib + vb, nc = ic + vc, k = lane - 1;
      int prx, pry;
      median_mvp(A, Bn, Cc, g, prx, pry);
      int cx = 0, cy = 0;
      if (k == 0) {
        cx = skx;
        cy = sky;
      } else if (va && k == ia) {
        cx = A.x;
        cy = A.y;
      } else if (vb && k == ib) {
        cx = Bn.x;
        cy = Bn.y;
      } else if (vc && k == ic) {
        cx = C.x;
        cy = C.y;
      } else if (g > 0 && k == nc) {
        cx = prx;
        cy = pry;
      }
      q.src = sm.src[par];
#pragma unroll
      for (int i = 0; i < WR; ++i) {
        q.s0[i] = q.src[q.sub * WR + i];
        q.s1[i] = q.src[(q.sub + 8) * WR + i];
      }
      q.nsad = q.nsatd = 0;
      H264Blk& B = q.B;
      B.x = mx * 16;
      B.px = prx;
      B.py = pry;
      B.lx = 4 - pad - B.x;
      B.hx = width + pad - 20 - B.x;
      q.org = plane_at<S>(q.R, 0, B.x, B.y);
      RefResult r;
      uint32_t ic0;
      q.whole(nc + (g > 0), cx, cy, lost, r.imx, r.imy, ic0);
      r.icost = ic0 + ref_cost;
      bool gate = false;
      if (nref > 1) {
        // refine_ratio: a further reference whose whole-sample cost is that
        // factor of the best before it is only scored.
        if ((tid & (kRefThreads - 1)) == 0) sm.icost[par][g] = r.icost;
        asm volatile("bar.sync 8, %0;" ::"r"(nref * kRefThreads) : "memory");
        uint32_t before = kInf;
        for (int p = 0; p < g; ++p) before = min(before, sm.icost[par][p]);
        gate = g > 0 && ratio > 0.0f && __uint2float_rn(r.icost) >= __fmul_rn(ratio, __uint2float_rn(before));
      }
      q.refine(r.imx, r.imy, gate ? 0 : hpel, gate ? 0 : qpel, r.mx, r.my, r.satd, r.cost);
      r.cost += ref_cost;
      if ((tid & (kRefThreads - 1)) == 0) sm.fin[par][g] = r;
    }
    if (tid < NSRC) sm.src[par ^ 1][tid] = nsrc;
    __syncthreads();
    // The reference of least cost, the first reaching it (all threads).
    int best = 0;
    uint32_t c16 = sm.fin[par][0].cost;
    for (int r = 1; r < nref; ++r) {
      const uint32_t c = sm.fin[par][r].cost;
      if (c < c16) {
        c16 = c;
        best = r;
      }
    }
    const RefResult& w = sm.fin[par][best];
    A = Nb{true, best, (int)(int16_t)w.mx, (int)(int16_t)w.my};
    if (tid == 0) {
      st_relaxed64(F.mvf + my * mbw + mx, mv_word(tag | (uint32_t)best, w.mx, w.my));
      if (mx > 0) write(mx - 1);
      ended = best;
    }
    if (sizeof(S) == 1 && sm.lost) return false;
    if (g < nref) {
      // Both counts in one sum (a lane has a few hundred of each at most).
      const uint32_t n = __reduce_add_sync(kFull, q.nsad | q.nsatd << 16);
      if (lane == 0) {
        atomicAdd(&sm.nsad[par], (n & 0xffffu) / 8);
        atomicAdd(&sm.nsatd[par], (n >> 16) / 16);
      }
    }
    wd = wb;
    wb = wc;
    wc = wn;
  }
  __syncthreads();
  if (tid == 0) write(mbw - 1);
  return true;
}

// Rows are taken in the order the host pushed them (every frame's row 0,
// then every row 1, ...), each after the row it reads, so a row's upper row
// is always owned by a running CTA.
template <class S>
__global__ void __launch_bounds__(RME_MAX_REFS * kRefThreads) h264_row_kernel(LaunchDesc L) {
  __shared__ RowSmem<S> sm;
  const int tid = threadIdx.x;
  const uint32_t epoch = __ldg(L.epoch);
  unsigned long long cnt[3] = {0, 0, 0};
  if (tid == 0) sm.lost = 0u;
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      const unsigned long long idx = atomicAdd(L.head, 1ull);
      sm.entry = idx >= (unsigned long long)L.total ? kPopDone : pop_slot(L, idx, epoch);
    }
    __syncthreads();
    const uint32_t e = sm.entry;
    if (e == kPopDone) break;
    if (e == 0xffffffffu) continue;  // the wait ran out (status set)
    const FrameDesc& F = L.frames[e >> 24];
    const int row = (int)(e & 0xffffffu);
    if (F.codec != RME_CODEC_H264 || F.mode != RME_PRED_STANDALONE || (sizeof(S) == 1) != (F.bd == 8) ||
        F.mvf == nullptr || row >= F.height / 16 || F.nref * kRefThreads > (int)blockDim.x) {
      if (tid == 0) atomicOr(L.status, kStatusBadTask);
      continue;
    }
    if (!h264_row<S>(L, F, row, sm, tid, cnt)) break;
  }
  if (tid == 0) {
    atomicAdd(&L.counters[0], cnt[0]);
    atomicAdd(&L.counters[1], cnt[1]);
    atomicAdd(&L.counters[2], cnt[2]);
    atomicAdd(&L.counters[3], cnt[1] * 256ull);
    atomicAdd(&L.counters[4], cnt[2] * 256ull);
  }
}

}  // namespace

int h264_row_blocks_per_sm(int bytes_per_sample, int nref) {
  int n = 0;
  const cudaError_t e =
      bytes_per_sample == 1
          ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, h264_row_kernel<uint8_t>, nref * kRefThreads, 0)
          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, h264_row_kernel<uint16_t>, nref * kRefThreads, 0);
  return e == cudaSuccess && n > 0 ? n : 1;
}

cudaError_t launch_h264_rows(const LaunchDesc& L, int bytes_per_sample, int nref, int grid, cudaStream_t s) {
  if (bytes_per_sample == 1)
    h264_row_kernel<uint8_t><<<grid, nref * kRefThreads, 0, s>>>(L);
  else
    h264_row_kernel<uint16_t><<<grid, nref * kRefThreads, 0, s>>>(L);
  return cudaGetLastError();
}

}  // namespace rme
