// HEVC searches that wait for no other search of their launch: GIVEN jobs
// (any block, the caller's predictors and seeds) and the AMP units of
// STANDALONE frames, which start from their CU's finished 2Nx2N result.
//
// What a search computes is search_full and refine_subpel
// (h265_me.rs:3749-3922): candidates, order, tie-breaks and counts as
// hevc_task has them. Blocks are any multiple of 4 up to 64x64, so a lane
// takes one word column of a run of rows, and every candidate of a step is
// scored on its words at once.
//   - Seeds: one after another, a word and its neighbour per row.
//   - Diamond: the twelve points of two rounds; five rows of three (16 bits:
//     four) words give all twelve, and each row is read once: the L1's
//     wavefronts, not the arithmetic, bound the kernel (60 % of their peak
//     when every word read its five rows).
//   - SATD: a lane per 4x4 tile; a block of fewer than 32 tiles has several
//     candidates side by side.
// Blocks of kFlatBigTiles 4x4 tiles and more are searched by a CTA's four warps
// together, smaller ones by a warp each: jobs come largest first, and a
// 64x64 block is then a quarter as long for the launch to wait for. (It also
// keeps a lane's words at sixteen, which sad_add's halves hold.) Bound by
// issue and by cache reads.
// Against a warp per task of the dataflow kernel (blocks but the square ones
// went a word at a time; AMP units waited in its queue): the 680,160 AMP units
// of a 2160p 10-bit frame, four references, 7.0 ms, with the frame's 2Nx2N
// rows 17.5 ms for 45; 6,000 mixed 10-bit GIVEN jobs 0.76 -> 0.27 ms (a warp
// each: 0.60), 600 of 8 bits 0.06 (0.21), 20,000 of 8 bits 0.48. Lists of one
// shape, 8 and 10 bits: 8,040 16x16 jobs 109 -> 91 and 189 -> 115 us, 480 64x64
// 241 -> 63 and 517 -> 102; 20,000 8x8 106 -> 104 and 178 -> 140 (of 8 bits
// 125 while their 16 words left half of a warp idle: HALVES). Five or six CTAs an SM (spills) gain at most
// 2 % and lose up to 7.
#include <algorithm>

#include "rme_search_impl.cuh"

namespace rme {
namespace {

constexpr int kFlatWarps = 4, kFlatBlocks = 4;  // warps a CTA, CTAs an SM

// Points two rounds of the small diamond reach: the first round's four, then
// (2,0), (-2,0), (1,1), (1,-1), (-1,1), (-1,-1), (0,2), (0,-2), an order in
// which the second round's new points come in the reference's order whichever
// way the first moved. Offsets + 2 as hex digits, point 0 the lowest.
__device__ __forceinline__ int point_x(int q) { return (int)((0x221133042213ull >> (4 * q)) & 15u) - 2; }
__device__ __forceinline__ int point_y(int q) { return (int)((0x041313221322ull >> (4 * q)) & 15u) - 2; }
// The second round's new points after the first moved in direction j.
__device__ __forceinline__ uint32_t second_points(int j) {
  return j == 0 ? 0x0d0u : j == 1 ? 0x320u : j == 2 ? 0x540u : 0xa80u;
}

template <class S>
struct FlatBlock {
  const S* src;  // the block's first source sample
  int src_stride, x, y, w, h, r, ns;
  int p0x, p0y, p1x, p1y;
  int sx, sy;    // lane i: seed i
  float lam;
};

// The search of one block. Counts its candidates into nsad and nsatd.
// WORDS: the reference's rows lie whole 32-bit words apart; otherwise (a
// caller's own planes) the diamond is scored a point at a time. SRC: every
// row of the source block begins on a word (a GIVEN block may lie at any
// sample); otherwise its reads find their words by themselves.
// W: the warps that share the search (1, or all of the CTA's, which then
// exchange their sums through `part`).
// HALVES: blocks of 8-bit samples, at most sixteen words of them (8x8 and
// smaller): a half of a warp holds the block, a word a lane, and its halves
// score candidates of their own.
template <class S, bool WORDS, bool SRC, int W, bool HALVES>
__device__ void flat_search(const FrameDesc& F, const FlatBlock<S>& K, rme_result* out, uint32_t (*part)[W][32],
                            uint32_t& nsad, uint32_t& nsatd) {
  const int lane = threadIdx.x & 31, warp = W == 1 ? 0 : (int)(threadIdx.x >> 5), tid = warp * 32 + lane;
  int buf = 0;
  // Lane k's sum over this warp to lane k's sum over the search's warps.
  auto total = [&](uint32_t mine) -> uint32_t {
    if constexpr (W == 1) {
      return mine;
    } else {
      part[buf][warp][lane] = mine;
      __syncthreads();
      uint32_t v = 0;
#pragma unroll
      for (int i = 0; i < W; ++i) v += part[buf][i][lane];
      buf ^= 1;
      return v;
    }
  };
  constexpr int B = (int)sizeof(S), SPW = 4 / B, WPT = 4 / SPW, NW = B == 1 ? 3 : 4;
  const DevPlanes R = F.ref[K.r];
  const int x = K.x, y = K.y, w = K.w, h = K.h, stride = R.stride, wr = w / SPW;
  const int padm = F.pad - 4;
  const int lox = -padm - x, hix = F.width + padm - w - x, loy = -padm - y, hiy = F.height + padm - h - y;
  const int range = F.search_range;
  const S* const org = plane_at<S>(R, 0, x, y);
  auto rate = [&](int mx, int my) { return hevc_rate(K.lam, mx, my, K.p0x, K.p0y, K.p1x, K.p1y); };
  // This lane's words: word wd of `rows` rows from row0 (none for the lanes
  // left over). Rows follow one another, so the diamond reads each once.
  constexpr int STEP = 32 * W;
  static_assert(!HALVES || (B == 1 && W == 1), "a lone warp's 8-bit block");
  const int place = HALVES ? lane & 15 : tid;
  const int segs = HALVES ? h : min(STEP / wr, h), each = HALVES ? 1 : (h + segs - 1) / segs;
  const int seg = place / wr, wd = place - seg * wr, row0 = seg * each, rows = seg < segs ? min(each, h - row0) : 0;
  auto source = [&](const S* q) -> uint32_t {
    return SRC ? RME_LD32(reinterpret_cast<const uint32_t*>(q)) : ldw(q);
  };
  // A CTA's lanes have at most sixteen words of a block; a lone warp's may
  // have more (a caller's own job list is not sorted by size).
  auto add = [](uint32_t a, uint32_t b, uint32_t acc) { return W > 1 ? sad_add(a, b, acc, S()) : vsad(a, b, acc, S()); };
  auto sum_of = [](uint32_t acc) { return W > 1 ? sad_sum(acc, S()) : acc; };
  // One candidate's SAD over this warp.
  auto sad1 = [&](int fx, int fy) -> uint32_t {
    uint32_t acc = 0;
    const S* rp = org + (ptrdiff_t)(fy + row0) * stride + fx + wd * SPW;
    const S* sp = K.src + (ptrdiff_t)row0 * K.src_stride + wd * SPW;
#pragma unroll 4
    for (int k = 0; k < rows; ++k) acc = add(source(sp + (ptrdiff_t)k * K.src_stride), ldw(rp + (ptrdiff_t)k * stride), acc);
    return __reduce_add_sync(kFull, sum_of(acc));
  };
  // HALVES: this lane's word of the block; the two halves' sums (at most
  // 64 * 255 each) in one word, the upper half's above; the candidates of
  // mask `m`, two at a time: lane k has candidate k's point and gets its SAD.
  uint32_t own = 0;
  if constexpr (HALVES) own = rows > 0 ? source(K.src + (ptrdiff_t)row0 * K.src_stride + wd * SPW) : 0u;
  auto both = [&](uint32_t acc) -> uint32_t { return __reduce_add_sync(kFull, acc << (lane & 16)); };
  auto pairs = [&](uint32_t m, int px, int py) -> uint32_t {
    uint32_t mine = 0;
    while (m != 0u) {
      const int a = __ffs(m) - 1;
      m &= m - 1u;
      const int b = m != 0u ? __ffs(m) - 1 : a, k = lane & 16 ? b : a;
      m &= m - 1u;
      const int fx = __shfl_sync(kFull, px, k), fy = __shfl_sync(kFull, py, k);
      const uint32_t v = both(rows > 0 ? add(own, ldw(org + (ptrdiff_t)(fy + row0) * stride + fx + wd * SPW), 0u) : 0u);
      if (lane == a) mine = v & 0xffffu;
      if (lane == b) mine = v >> 16;
    }
    return mine;
  };

  // Seeds: >> 2, clamp_pos, deduplicated (`tried`), scored in order.
  const int qx = min(max(K.sx >> 2, lox), hix), qy = min(max(K.sy >> 2, loy), hiy);
  bool dup = false;
  for (int j = 0; j + 1 < K.ns; ++j) {
    const int jx = __shfl_sync(kFull, qx, j), jy = __shfl_sync(kFull, qy, j);
    dup |= j < lane && jx == qx && jy == qy;
  }
  const uint32_t kept = __ballot_sync(kFull, lane < K.ns && !dup);
  nsad = __popc(kept);
  nsatd = 9;
  uint32_t c = 0;
  if constexpr (HALVES) {
    c = pairs(kept, qx, qy);
  } else {
    for (uint32_t m = kept; m != 0u; m &= m - 1u) {
      const int s = __ffs(m) - 1;
      const uint32_t v = sad1(__shfl_sync(kFull, qx, s), __shfl_sync(kFull, qy, s));
      if (lane == s) c = v;
    }
  }
  c = total(c);
  Pick p = warp_min((kept >> lane) & 1u ? c + rate(qx * 4, qy * 4) : kInf);
  uint32_t bcost = p.cost;
  int fbx = 0, fby = 0;
  if (kept != 0u) {
    fbx = __shfl_sync(kFull, qx, p.lane);
    fby = __shfl_sync(kFull, qy, p.lane);
  }
  const int ox = fbx, oy = fby;
  auto allowed = [&](int fx, int fy) {
    return abs(fx - ox) <= range && abs(fy - oy) <= range && fx >= lox && fx <= hix && fy >= loy && fy <= hiy;
  };
  for (int it = 0, rings = 0;;) {
    while (it < 2 * range) {
      // Lane q < 12: point q. Points that may not be scored may lie outside
      // the plane: the rows and words read are kept inside the block's reach
      // by scoring such steps a point at a time.
      const int fx = fbx + point_x(min(lane, 11)), fy = fby + point_y(min(lane, 11));
      const bool ok = lane < 12 && allowed(fx, fy);
      const uint32_t there = __ballot_sync(kFull, ok);
      uint32_t mine = 0;
      if (HALVES && WORDS && fbx - 2 >= lox && fbx + 2 <= hix && fby - 2 >= loy && fby + 2 <= hiy) {
        // The lower half takes the points of even numbers, the upper half
        // those of odd numbers, which mirror them: three rows and six points
        // a lane instead of five and twelve.
        const int d = lane & 16 ? -1 : 1;
        const uintptr_t a0 = reinterpret_cast<uintptr_t>(org + (ptrdiff_t)fby * stride + fbx - 2);
        const uint32_t off = (uint32_t)(a0 & 3);
        const int rs = stride / 4;
        uint32_t acc[6] = {};
        if (rows > 0) {
          const uint32_t* const wp = reinterpret_cast<const uint32_t*>(a0 & ~uintptr_t(3)) + (ptrdiff_t)row0 * rs + wd;
          uint32_t v[3][3];  // rows 0, d, 2d
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) v[i][j] = RME_LD32(wp + (ptrdiff_t)(i * d) * rs + j);
          auto at = [&](int dx, const uint32_t (&q)[3]) {
            const uint32_t o = off + (uint32_t)(dx + 2);
            return __funnelshift_r(o >> 2 ? q[1] : q[0], o >> 2 ? q[2] : q[1], (o & 3u) * 8u);
          };
          acc[0] = add(own, at(d, v[0]), 0u);
          acc[1] = add(own, at(0, v[1]), 0u);
          acc[2] = add(own, at(2 * d, v[0]), 0u);
          acc[3] = add(own, at(1, v[1]), 0u);
          acc[4] = add(own, at(-1, v[1]), 0u);
          acc[5] = add(own, at(0, v[2]), 0u);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          const uint32_t v = both(acc[i]);
          if (lane >> 1 == i) mine = lane & 1 ? v >> 16 : v & 0xffffu;
        }
      } else if (HALVES) {
        mine = pairs(there, fx, fy);
      } else if (WORDS && fbx - 2 >= lox && fbx + 2 <= hix && fby - 2 >= loy && fby + 2 <= hiy) {
        uint32_t acc[12];
#pragma unroll
        for (int q = 0; q < 12; ++q) acc[q] = 0u;
        // dx = -2's first sample in the aligned words of a row.
        const S* const rp = org + (ptrdiff_t)fby * stride + fbx - 2;
        const uintptr_t a0 = reinterpret_cast<uintptr_t>(rp);
        const uint32_t off = (uint32_t)(a0 & 3);
        const uint32_t* const q0 = reinterpret_cast<const uint32_t*>(a0 & ~uintptr_t(3));
        const int rs = stride * B / 4;  // rows are whole words apart
        const uint32_t* wp = q0 + (ptrdiff_t)(row0 - 2) * rs + wd;
        const S* sp = K.src + (ptrdiff_t)row0 * K.src_stride + wd * SPW;
        if (rows > 0) {
          uint32_t v[5][NW];
#pragma unroll
          for (int i = 0; i < 4; ++i, wp += rs)
#pragma unroll
            for (int j = 0; j < NW; ++j) v[i][j] = RME_LD32(wp + j);
          auto at = [&](int dx, int dy) {  // the word of samples at (dx, dy)
            const uint32_t o = off + (uint32_t)((dx + 2) * B), sh = (o & 3u) * 8u;
            const int j = (int)(o >> 2);
            const uint32_t lo = B == 1 ? (j ? v[dy + 2][1] : v[dy + 2][0])
                                       : (j == 0 ? v[dy + 2][0] : j == 1 ? v[dy + 2][1] : v[dy + 2][2]);
            const uint32_t hi = B == 1 ? (j ? v[dy + 2][2] : v[dy + 2][1])
                                       : (j == 0 ? v[dy + 2][1] : j == 1 ? v[dy + 2][2] : v[dy + 2][NW - 1]);
            return __funnelshift_r(lo, hi, sh);
          };
#pragma unroll 2
          for (int k = 0; k < rows; ++k, wp += rs, sp += K.src_stride) {
#pragma unroll
            for (int j = 0; j < NW; ++j) v[4][j] = RME_LD32(wp + j);
            const uint32_t s = source(sp);
            acc[0] = add(s, at(1, 0), acc[0]);
            acc[1] = add(s, at(-1, 0), acc[1]);
            acc[2] = add(s, at(0, 1), acc[2]);
            acc[3] = add(s, at(0, -1), acc[3]);
            acc[4] = add(s, at(2, 0), acc[4]);
            acc[5] = add(s, at(-2, 0), acc[5]);
            acc[6] = add(s, at(1, 1), acc[6]);
            acc[7] = add(s, at(1, -1), acc[7]);
            acc[8] = add(s, at(-1, 1), acc[8]);
            acc[9] = add(s, at(-1, -1), acc[9]);
            acc[10] = add(s, at(0, 2), acc[10]);
            acc[11] = add(s, at(0, -2), acc[11]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < NW; ++j) v[i][j] = v[i + 1][j];
          }
        }
#pragma unroll
        for (int q = 0; q < 12; ++q) {
          const uint32_t v = __reduce_add_sync(kFull, sum_of(acc[q]));
          if (lane == q) mine = v;
        }
      } else {
        for (uint32_t m = there; m != 0u; m &= m - 1u) {
          const int q = __ffs(m) - 1;
          const uint32_t v = sad1(fbx + point_x(q), fby + point_y(q));
          if (lane == q) mine = v;
        }
      }
      mine = total(mine);
      c = ok ? mine + rate(fx * 4, fy * 4) : kInf;
      nsad += __popc(there & 0xfu);
      p = warp_min(lane < 4 ? c : kInf);
      if (!(p.cost < bcost)) break;
      const bool unscored = bcost == kInf;  // no seeds: the next round scores the centre itself
      bcost = p.cost;
      const int q1 = p.lane, bx1 = fbx + point_x(q1), by1 = fby + point_y(q1);
      const uint32_t second = second_points(q1);
      if (++it >= 2 * range) {
        fbx = bx1;
        fby = by1;
        break;
      }
      if (unscored) {
        fbx = bx1;
        fby = by1;
        continue;
      }
      nsad += 1u + __popc(there & second);  // the fourth point is the old best
      p = warp_min((second >> lane) & 1u ? c : kInf);
      if (!(p.cost < bcost)) {
        fbx = bx1;
        fby = by1;
        break;
      }
      bcost = p.cost;
      fbx += point_x(p.lane);
      fby += point_y(p.lane);
      ++it;
    }
    if (rings >= F.search_rings) break;
    ++rings;
    // The 24 ring points at 4, 8, 16 around the settled point, in order; a
    // move restarts the diamond.
    const int k = min(lane, 23), rr = k < 8 ? 4 : k < 16 ? 8 : 16, k8 = k & 7;
    const int fx = fbx + ((k8 == 0 || k8 == 4 || k8 == 6) ? rr : (k8 == 1 || k8 == 5 || k8 == 7) ? -rr : 0);
    const int fy = fby + ((k8 == 2 || k8 == 4 || k8 == 5) ? rr : (k8 == 3 || k8 == 6 || k8 == 7) ? -rr : 0);
    const bool ok = lane < 24 && allowed(fx, fy);
    const uint32_t there = __ballot_sync(kFull, ok);
    uint32_t mine = 0;
    if constexpr (HALVES) {
      mine = pairs(there, fx, fy);
    } else {
      for (uint32_t m = there; m != 0u; m &= m - 1u) {
        const int s = __ffs(m) - 1;
        const uint32_t v = sad1(__shfl_sync(kFull, fx, s), __shfl_sync(kFull, fy, s));
        if (lane == s) mine = v;
      }
    }
    mine = total(mine);
    nsad += __popc(there);
    p = warp_min(ok ? mine + rate(fx * 4, fy * 4) : kInf);
    if (!(p.cost < bcost)) break;
    bcost = p.cost;
    fbx = __shfl_sync(kFull, fx, p.lane);
    fby = __shfl_sync(kFull, fy, p.lane);
    it = 0;
  }
  const uint32_t int_cost = bcost;
  const int imx = fbx * 4, imy = fby * 4;

  // refine_subpel: P lanes a candidate (the tiles, rounded up to a power of
  // two, at most 32 a warp), 32 / P candidates side by side; lane k gets
  // candidate k's SATD.
  const int tw = w >> 2, nt = tw * (h >> 2), lp = W > 1 || nt >= 32 ? 5 : 32 - __clz(nt - 1), P = 1 << lp;
  const int t0 = W > 1 ? tid : lane & (P - 1), g = lane >> lp, tstep = W > 1 ? STEP : P;
  const bool pow2 = (tw & (tw - 1)) == 0;
  const int tsh = __ffs(tw) - 1;
  auto source_tile = [&](int t, uint32_t (&sw)[4][WPT]) {
    const int ty = pow2 ? t >> tsh : t / tw, tx = t - ty * tw;
#pragma unroll
    for (int rr = 0; rr < 4; ++rr) {
      const S* sp = K.src + (ptrdiff_t)(ty * 4 + rr) * K.src_stride + tx * 4;
#pragma unroll
      for (int q = 0; q < WPT; ++q) sw[rr][q] = source(sp + q * SPW);
    }
  };
  uint32_t first[4][WPT] = {};  // the lane's first tile, most blocks' only one
  if (t0 < nt) source_tile(t0, first);
  auto tile_sum = [&](int mx, int my) -> uint32_t {  // over this lane's tiles
    const S* const pp = plane_at<S>(R, (my & 3) * 4 + (mx & 3), x + (mx >> 2), y + (my >> 2));
    auto tile = [&](int t, const uint32_t (&sw)[4][WPT]) {
      const int ty = pow2 ? t >> tsh : t / tw, tx = t - ty * tw;
      uint32_t pr[4][WPT];
#pragma unroll
      for (int rr = 0; rr < 4; ++rr) ldwords<WPT>(pp + (ptrdiff_t)(ty * 4 + rr) * stride + tx * 4, pr[rr]);
      return satd4x4<WPT>(sw, pr);
    };
    uint32_t acc = t0 < nt ? tile(t0, first) : 0u;
    for (int t = t0 + tstep; t < nt; t += tstep) {
      uint32_t sw[4][WPT];
      source_tile(t, sw);
      acc += tile(t, sw);
    }
    return acc;
  };
  auto satd = [&](int nc, auto vec) -> uint32_t {
    uint32_t got = 0;
    for (int k0 = 0; k0 < nc; k0 += 32 >> lp) {
      const int k = k0 + g;
      int mx, my;
      uint32_t v = k < nc && vec(k, mx, my) ? tile_sum(mx, my) : 0u;
      if (lp == 5) {
        v = __reduce_add_sync(kFull, v);
      } else {
        for (int o = P >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
      }
      const int from = (lane - k0) << lp;
      const uint32_t u = __shfl_sync(kFull, v, from & 31);
      if (lane >= k0 && from < 32) got = u;
    }
    return total(got);
  };
  auto half_vec = [&](int k, int& mx, int& my) {
    const int q = k == 0 ? 4 : k <= 4 ? k - 1 : k, qr = q / 3;
    mx = imx + (q - qr * 3 - 1) * 2;
    my = imy + (qr - 1) * 2;
    return true;
  };
  uint32_t v = satd(9, half_vec);
  int mx, my;
  half_vec(min(lane, 8), mx, my);
  p = warp_min(lane < 9 ? v + rate(mx, my) : kInf);
  uint32_t bc = p.cost, bsatd = __shfl_sync(kFull, v, p.lane);
  int bmx, bmy;
  half_vec(p.lane, bmx, bmy);
  const int hmx = bmx, hmy = bmy, cross = F.quarter_cross;
  auto quarter_vec = [&](int k, int& ax, int& ay) {
    const int q = k < 4 ? k : k + 1, qr = q / 3, dx = q - qr * 3 - 1, dy = qr - 1;
    ax = (int)(int16_t)(hmx + dx);
    ay = (int)(int16_t)(hmy + dy);
    return !(cross != 0 && dx != 0 && dy != 0);
  };
  v = satd(8, quarter_vec);
  const bool ok = quarter_vec(min(lane, 7), mx, my) && lane < 8;
  nsatd += cross ? 4 : 8;
  p = warp_min(ok ? v + rate(mx, my) : kInf);
  if (p.cost < bc) {
    bc = p.cost;
    bsatd = __shfl_sync(kFull, v, p.lane);
    quarter_vec(p.lane, bmx, bmy);
  }
  write_result(out, bmx, bmy, K.r, bc, bsatd, imx, imy, int_cost, nsad, nsatd, tid);
}

// A GIVEN job; false (and the status bit) for one that fails the check.
template <class S>
__device__ bool given_block(const LaunchDesc& L, const FrameDesc& F, int t, int lane, FlatBlock<S>& K) {
  const rme_job* j = &F.jobs[t];
  if (t >= F.ntasks || F.mode != RME_PRED_GIVEN || !given_job_ok(F, j, RME_MAX_SEEDS)) {
    if (lane == 0) atomicOr(L.status, kStatusBadTask);
    return false;
  }
  K.x = j->x;
  K.y = j->y;
  K.w = j->w;
  K.h = j->h;
  K.r = j->ref;
  K.ns = j->nseeds;
  K.p0x = j->mvp[0].x;
  K.p0y = j->mvp[0].y;
  K.p1x = j->mvp[1].x;
  K.p1y = j->mvp[1].y;
  K.sx = lane < K.ns ? j->seeds[lane].x : 0;
  K.sy = lane < K.ns ? j->seeds[lane].y : 0;
  if (F.bi_src) {  // refine_bi: the target block stands in for the source, at twice the multiplier
    K.src = (const S*)F.bi_src + (int64_t)t * (kBiBlock * kBiBlock);
    K.src_stride = kBiBlock;
    K.lam = 2.0f * F.lam;
  } else {
    K.src = plane_at<S>(F.src, 0, K.x, K.y);
    K.src_stride = F.src.stride;
    K.lam = F.lam;
  }
  return true;
}

// AMP unit t (a task index past the 2Nx2N blocks): searched from its CU's own
// 2Nx2N result, AMVP pair [own, 0], seeds [own, mvp0, mvp1].
template <class S>
__device__ void amp_block(const FrameDesc& F, int t, int lane, FlatBlock<S>& K) {
  const int blk = t / F.nref;
  K.r = t - blk * F.nref;
  int la = 0;
  while (la + 1 < F.amp_nlev && blk >= F.amp_base[la + 1]) ++la;
  const int per = 2 * F.amp_nmodes, j = blk - F.amp_base[la], cu = j / per, rem = j - cu * per, part = rem & 1;
  int mode = 0;
  for (int b = 0, k = rem >> 1; b < 4; ++b)
    if ((F.amp >> b) & 1) {
      if (k == 0) {
        mode = b;
        break;
      }
      --k;
    }
  const int N = F.size[la], q = N / 4, cby = cu / F.nbx[la], cbx = cu - cby * F.nbx[la];
  K.x = cbx * N;
  K.y = cby * N;
  K.w = K.h = N;
  if (mode < 2) {
    K.h = (part == (mode == 0)) ? 3 * q : q;
    if (part) K.y += mode == 0 ? q : 3 * q;
  } else {
    K.w = (part == (mode == 2)) ? 3 * q : q;
    if (part) K.x += mode == 2 ? q : 3 * q;
  }
  const uint32_t own = ldcg_u32(&F.out[(int64_t)(F.base[la] + cu) * F.nref + K.r].mv);
  K.p0x = mvx_of(own);
  K.p0y = mvy_of(own);
  K.p1x = K.p1y = 0;
  K.ns = 3;
  K.sx = lane < 2 ? K.p0x : 0;
  K.sy = lane < 2 ? K.p0y : 0;
  K.src = plane_at<S>(F.src, 0, K.x, K.y);
  K.src_stride = F.src.stride;
  K.lam = F.lam;
}

// Searches are taken from L.head: the first `nbig` by CTAs, one at a time,
// the others by warps, `chunk` consecutive ones at a time. GIVEN: entry i of
// L's queue. AMP: the frames' AMP units one frame after another; those of a
// frame's 64x64 CUs are its big ones (their halves of 1024 samples and more),
// numbered first over all frames. HALVES: GIVEN jobs of 8 bits that are all
// blocks of half a warp. They have a kernel of their own: beside the larger
// blocks' code theirs costs those 2 to 10 % (registers), and a list of both
// that takes two loops in turn waits for the second one's instructions (3,000
// 8x8 and 3,000 16x16 jobs 61 -> 79 us). 20,000 8x8 jobs 125 -> 104 us, 600 of
// them 26 -> 22, 20,000 of 8x4, 4x8 and 4x4 104 -> 87.
template <class S, bool AMP, bool WORDS, bool HALVES = false>
__global__ void __launch_bounds__(kFlatWarps * 32, kFlatBlocks) hevc_flat_kernel(LaunchDesc L, int nframes, int64_t nbig,
                                                                                 int chunk) {
  __shared__ uint32_t part[2][kFlatWarps][32];
  __shared__ unsigned long long next;
  const int lane = threadIdx.x & 31;
  constexpr int D = sizeof(S) == 1 ? 0 : 1;  // the frames' counts of this depth
  unsigned long long cnt[5] = {0, 0, 0, 0, 0};
  int f = 0;
  // Search i (or false): by the whole CTA, or by this warp.
  auto search = [&](int64_t i, auto warps) {
    constexpr int W = decltype(warps)::value;
    int t;
    if (AMP) {
      const int64_t j = W > 1 ? i : i - nbig;
      while (f + 1 < nframes && j >= L.frames[f + 1].amp_first[W > 1][D]) ++f;
    } else {
      const uint32_t e = (uint32_t)L.ready[i];
      f = (int)(e >> 24);
      t = (int)(e & 0xffffffu);
    }
    const FrameDesc& F = L.frames[f];
    if (AMP) {
      // The first level's units are the big ones where its blocks are 64x64.
      const int big = F.size[0] == 64 ? F.amp_base[1] : F.amp_base[0];
      t = (W > 1 ? F.amp_base[0] : big) * F.nref + (int)((W > 1 ? i : i - nbig) - F.amp_first[W > 1][D]);
    }
    if ((sizeof(S) == 1) != (F.bd == 8) || F.codec != RME_CODEC_HEVC || t >= F.ntasks) {
      if (lane == 0) atomicOr(L.status, kStatusBadTask);
      return;
    }
    FlatBlock<S> K;
    if (AMP) amp_block<S>(F, t, lane, K);
    else if (!given_block<S>(L, F, t, lane, K)) return;
    uint32_t nsad, nsatd;
    auto* const shared = reinterpret_cast<uint32_t(*)[W][32]>(part);
    if constexpr (HALVES && W == 1)
      flat_search<S, WORDS, false, W, true>(F, K, &F.out[t], shared, nsad, nsatd);
    else if (AMP || ((reinterpret_cast<uintptr_t>(K.src) & 3) == 0 && (K.src_stride * (int)sizeof(S) & 3) == 0))
      flat_search<S, WORDS, true, W, false>(F, K, &F.out[t], shared, nsad, nsatd);
    else
      flat_search<S, WORDS, false, W, false>(F, K, &F.out[t], shared, nsad, nsatd);
    if (W > 1 && threadIdx.x >= 32) return;
    cnt[0] += 1;
    cnt[1] += nsad;
    cnt[2] += nsatd;
    cnt[3] += (unsigned long long)nsad * (K.w * K.h);
    cnt[4] += (unsigned long long)nsatd * (K.w * K.h);
  };
  while (!HALVES && nbig > 0) {
    __syncthreads();  // the last search's sums, and its place, are read
    if (threadIdx.x == 0) next = atomicAdd(L.head, 1ull);
    __syncthreads();
    const unsigned long long i = next;
    if ((int64_t)i >= nbig) break;
    search((int64_t)i, std::integral_constant<int, kFlatWarps>{});
  }
  f = 0;
  for (;;) {
    unsigned long long i0 = 0;
    if (lane == 0) i0 = atomicAdd(L.tail, (unsigned long long)chunk);
    i0 = __shfl_sync(kFull, i0, 0) + (unsigned long long)nbig;
    if ((int64_t)i0 >= L.total) break;
    const int64_t end = min((int64_t)i0 + chunk, L.total);
    for (int64_t i = (int64_t)i0; i < end; ++i) search(i, std::integral_constant<int, 1>{});
  }
  if (lane < 5) atomicAdd(&L.counters[lane], lane == 0 ? cnt[0] : lane == 1 ? cnt[1] : lane == 2 ? cnt[2] : lane == 3 ? cnt[3] : cnt[4]);
}

}  // namespace

cudaError_t launch_hevc_flat(const LaunchDesc& L, int bytes_per_sample, bool amp, bool words, int nframes, int64_t nbig,
                             int nsm, cudaStream_t s, bool halves) {
  const int64_t most = (int64_t)nsm * kFlatBlocks, small = L.total - nbig;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(nbig + (small + kFlatWarps - 1) / kFlatWarps, most));
  // Few takes from the counter while many searches are left for every warp.
  const int chunk = (int)std::max<int64_t>(1, std::min<int64_t>(16, small / (most * kFlatWarps * 16)));
  constexpr int T = kFlatWarps * 32;
  if (bytes_per_sample == 1) {
    if (amp) hevc_flat_kernel<uint8_t, true, true><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
    else if (words && halves) hevc_flat_kernel<uint8_t, false, true, true><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
    else if (words) hevc_flat_kernel<uint8_t, false, true><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
    else hevc_flat_kernel<uint8_t, false, false><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
  } else {
    if (amp) hevc_flat_kernel<uint16_t, true, true><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
    else if (words) hevc_flat_kernel<uint16_t, false, true><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
    else hevc_flat_kernel<uint16_t, false, false><<<grid, T, 0, s>>>(L, nframes, nbig, chunk);
  }
  return cudaGetLastError();
}

}  // namespace rme
