// The lookahead's motion estimation at half resolution, for the HEVC
// encoder's quantiser propagation (encode/h265_cutree.rs) and the H.264
// encoder's (encode/h264_lookahead.rs): the half-resolution plane of a
// picture and its blocks' intra costs, the per-block motion search against
// a reference and the SATD against the average of two displaced blocks.
//
// The search reads the left and above blocks' vectors as seeds, so its
// blocks form a wavefront. A warp owns a row of blocks and searches it left
// to right, its left seed in registers; each block's vector is published as
// one word, and the row below waits (bounded) for that word only. Rows are
// claimed top to bottom from one counter, so a row a warp waits for was
// claimed earlier by a running warp: the wait always ends unless its bound
// runs out, which sets the status word. The winners' SATDs, which no other
// block reads, are a second launch over all blocks at once.
#include <cuda_runtime.h>

#include <algorithm>

#include "rme_internal.h"

namespace rme {
namespace {

constexpr unsigned kAll = 0xffffffffu;

// LowRes::new (h265_cutree.rs:61-110): the 2x2 mean of the picture
// (clamped at its edges) shifted to 8 bits, over whole 8x8 blocks, the
// border replicated: every padded position is the value of its clamped
// position.
template <class S>
__global__ void lowres_build_kernel(const S* __restrict__ pic, int pstride, int w, int h, int bd, LowresDesc L) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y * blockDim.y + threadIdx.y;
  const int rows = L.ph + 2 * kLowresPad;
  if (X >= L.stride || Y >= rows) return;
  const int lw = (w + 1) / 2, lh = (h + 1) / 2;
  const int xx = min(max(X - kLowresPad, 0), L.pw - 1), yy = min(max(Y - kLowresPad, 0), L.ph - 1);
  const int x2 = 2 * min(xx, lw - 1), y2 = 2 * min(yy, lh - 1);
  auto at = [&](int x, int y) { return (int)pic[(ptrdiff_t)min(y, h - 1) * pstride + min(x, w - 1)]; };
  const int s = at(x2, y2) + at(x2 + 1, y2) + at(x2, y2 + 1) + at(x2 + 1, y2 + 1);
  L.plane[(ptrdiff_t)Y * L.stride + X] = (uint8_t)min(((s + 2) >> 2) >> (bd - 8), 255);
}

// The 4x4 Hadamard SATD of sixteen differences, (sum + 1) >> 1
// (dsp/distortion.rs:350-381).
__device__ __forceinline__ uint32_t hadamard_satd(int (&d)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = d[i * 4], q = d[i * 4 + 1], u = d[i * 4 + 2], v = d[i * 4 + 3];
    const int s0 = p + v, s1 = q + u, s2 = q - u, s3 = p - v;
    d[i * 4] = s0 + s1;
    d[i * 4 + 1] = s3 + s2;
    d[i * 4 + 2] = s0 - s1;
    d[i * 4 + 3] = s3 - s2;
  }
  uint32_t sum = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = d[j], q = d[4 + j], u = d[8 + j], v = d[12 + j];
    const int s0 = p + v, s1 = q + u, s2 = q - u, s3 = p - v;
    sum += abs(s0 + s1) + abs(s3 + s2) + abs(s0 - s1) + abs(s3 - s2);
  }
  return (sum + 1) >> 1;
}

// One 4x4 tile's SATD.
template <class S>
__device__ __forceinline__ uint32_t satd4x4_tile(const S* a, int as, const S* b, int bs) {
  int d[16];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) d[r * 4 + c] = (int)a[(ptrdiff_t)r * as + c] - (int)b[(ptrdiff_t)r * bs + c];
  return hadamard_satd(d);
}

template <class S>
__device__ uint32_t satd8x8(const S* a, int as, const S* b, int bs) {
  uint32_t total = 0;
  for (int ty = 0; ty < 2; ++ty)
    for (int tx = 0; tx < 2; ++tx)
      total += satd4x4_tile<S>(a + (ptrdiff_t)(ty * 4) * as + tx * 4, as, b + (ptrdiff_t)(ty * 4) * bs + tx * 4, bs);
  return total;
}

// intra_cost (h265_cutree.rs:118-140), one thread per block: the least SATD
// of the flat, horizontal and vertical predictions from the samples above
// and left, floored at 16.
__global__ void lowres_intra_kernel(LowresDesc L) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= L.bw * L.bh) return;
  const int x = (b % L.bw) * 8, y = (b / L.bw) * 8;
  const uint8_t* src = L.plane + (ptrdiff_t)(y + kLowresPad) * L.stride + x + kLowresPad;
  uint8_t top[8], left[8];
  int st = 0;
  for (int i = 0; i < 8; ++i) {
    top[i] = src[i - L.stride];
    left[i] = src[(ptrdiff_t)i * L.stride - 1];
    st += top[i] + left[i];
  }
  uint8_t pred[64];
  const uint8_t dc = (uint8_t)((st + 8) / 16);
  for (int i = 0; i < 64; ++i) pred[i] = dc;
  uint32_t best = satd8x8<uint8_t>(src, L.stride, pred, 8);
  for (int i = 0; i < 64; ++i) pred[i] = left[i / 8];
  best = min(best, satd8x8<uint8_t>(src, L.stride, pred, 8));
  for (int i = 0; i < 64; ++i) pred[i] = top[i % 8];
  best = min(best, satd8x8<uint8_t>(src, L.stride, pred, 8));
  L.intra[b] = max(best, 16u);
}

// A block's published vector: bit 32 set, the vector in the low half. The
// word carries all a reader needs, so relaxed accesses suffice.
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, uint32_t mv) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(1ull << 32 | mv) : "memory");
}

// A bounded wait for a published word, already loaded once (`w`): at most
// `limit` polls (the first few back to back, the upper row being a block
// ahead), then the status word records the timeout and the wait gives up
// (false). A warp that gave up once waits no more (`lost`).
__device__ __forceinline__ bool wait_word(const unsigned long long* p, unsigned long long& w, uint32_t* status,
                                          bool lost = false, uint32_t limit = kSpinLimit) {
  uint32_t ns = 32;
  for (uint32_t it = 0; (w >> 32) == 0ull; ++it) {
    if (lost || it >= limit) {
      if (!lost) atomicOr(status, kStatusWaitTimeout);
      return false;
    }
    if (it >= 16) {
      __nanosleep(ns);
      if (ns < 256) ns <<= 1;
    }
    w = ld_word(p);
  }
  return true;
}

// The wait of a warp, all of whose lanes hold the word: where one of them gave
// up, all go on with zero and wait no more (their steps and votes must agree).
__device__ __forceinline__ bool wait_above(const unsigned long long* p, unsigned long long& w, uint32_t* status,
                                           bool lost) {
  lost = __any_sync(kAll, !wait_word(p, w, status, lost));
  if (lost) w = 0ull;
  return lost;
}

// |a - b| of four bytes, summed onto acc.
__device__ __forceinline__ uint32_t sad4(uint32_t a, uint32_t b, uint32_t acc) {
  uint32_t r;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(acc));
  return r;
}
// Point k of the rings (4, 2, 1 samples; each (s,0), (-s,0), (0,s), (0,-s)):
// offsets + 4 as hex digits, the lowest first.
__device__ __forceinline__ int ring_x(int k) { return (int)((0x443544264408ull >> (4 * k)) & 15u) - 4; }
__device__ __forceinline__ int ring_y(int k) { return (int)((0x354426440844ull >> (4 * k)) & 15u) - 4; }

// The row a warp claims next: row-major over the pairs (every pair's row 0,
// then every row 1, ...), so that a claim's upper row was claimed before it.
__device__ __forceinline__ bool claim_row(unsigned long long* counter, int npairs, int rows, int lane, int& pair,
                                          int& row) {
  unsigned long long c = 0;
  if (lane == 0) c = atomicAdd(counter, 1ull);
  c = __shfl_sync(kAll, c, 0);
  if (c >= (unsigned long long)npairs * rows) return false;
  row = (int)(c / npairs);
  pair = (int)(c - (unsigned long long)row * npairs);
  return true;
}

// search (h265_cutree.rs:152-216), a warp per row of blocks, two lanes per
// candidate (four rows of the block each). The reference walks a 4-, a 2-
// and a 1-sample ring of four points, a ring again after each move; the
// three rings around a centre are known together, so a pass scores all
// twelve points and resolves them in the reference's order (the first ring
// with a point below the best moves there and the walk goes on at that
// ring; the points counted are those the reference scores). The first pass
// scores the seeds and, around the first of the neighbours' vectors, the
// rings: where that seed wins, as it does in even motion, its rings are
// known already.
//
// Bound by the chain of passes along the wavefront (bw + bh blocks), each a
// chain of dependent instructions: a load, one shuffle and one warp minimum,
// over keys that order the points by ring, cost and place, so that the minimum
// is the decision; what depends on the lane alone is kept. Eight pairs of
// 1080p pictures: 3,010 us when a warp took one block at a time (claim, two
// waits, up to twelve passes, the SATD), 547 us a row a warp with ballots and
// shuffles to decide, 445 us this way, the SATDs included; a row of eight
// bytes by two 8-byte loads instead of three words took 50 us of it (the
// candidates lie on lines of their own, each a pass through L1 a load).
constexpr int kLaWarps = 4;  // rows per CTA: few, so that a launch's rows spread over the SMs
__global__ void __launch_bounds__(kLaWarps * 32) lowres_search_kernel(const LowresDesc* pairs, int npairs,
                                                                      unsigned long long* words_all,
                                                                      unsigned long long* counter, uint32_t* status,
                                                                      rme_mv* mv_all, uint32_t* nsad_all) {
  const int lane = threadIdx.x & 31, q = lane >> 1, half = lane & 1;
  const int bw = pairs[0].bw, bh = pairs[0].bh, n = bw * bh, lim = kLowresPad - 1;
  bool lost = false;
  // This lane's ring point in a first pass (candidates 3..14) and in a later
  // one (0..11).
  const int rx0 = ring_x(min(max(q - 3, 0), 11)), ry0 = ring_y(min(max(q - 3, 0), 11));
  const int rx1 = ring_x(min(q, 11)), ry1 = ring_y(min(q, 11));
  for (int pi, by; claim_row(counter, npairs, bh, lane, pi, by);) {
    const LowresDesc cur = pairs[2 * pi], ref = pairs[2 * pi + 1];
    unsigned long long* words = words_all + (size_t)pi * n + (size_t)by * bw;
    const unsigned long long* up = words - bw;
    const int y = by * 8;
    const uint8_t* srow = cur.plane + (ptrdiff_t)(y + kLowresPad + half * 4) * cur.stride + kLowresPad;
    const uint32_t rstride = (uint32_t)ref.stride;  // a multiple of 8: a block's rows start alike
    const uint32_t rrow = (uint32_t)(y + kLowresPad + half * 4) * rstride + kLowresPad;
    const int ylo = -lim - y, yn = ref.ph + 2 * lim - 8;  // rows a block may be displaced to: ylo .. ylo + yn
    const int xn = ref.pw + 2 * lim - 8;
    uint32_t prev_n = 0;  // the block before's count, stored a block later
    // The first block's source rows and upper vector; later ones are loaded
    // a block ahead (8-byte aligned: x, the pad and the stride are multiples
    // of 8).
    uint2 s[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) s[r] = __ldg(reinterpret_cast<const uint2*>(srow + (ptrdiff_t)r * cur.stride));
    unsigned long long uw = by > 0 ? ld_word(up) : 0ull;
    uint32_t lv = 0;
    for (int bx = 0; bx < bw; ++bx) {
      const int x = bx * 8, xlo = -lim - x;
      const uint32_t rb = rrow + x;
      if (by > 0) lost = wait_above(up + bx, uw, status, lost);
      const uint32_t av = (uint32_t)uw;
      uint2 sn[4] = {};
      unsigned long long un = 0ull;
      if (bx + 1 < bw) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          sn[r] = __ldg(reinterpret_cast<const uint2*>(srow + (ptrdiff_t)r * cur.stride + x + 8));
        if (by > 0) un = ld_word(up + bx + 1);
      }
      auto inplane = [&](int dx, int dy) {
        return (uint32_t)(dx - xlo) <= (uint32_t)xn && (uint32_t)(dy - ylo) <= (uint32_t)yn;
      };
      auto score = [&](bool ok, int dx, int dy) -> uint32_t {
        uint32_t part = 0, odd = 0;
        if (ok) {
          const uint32_t o = rb + (uint32_t)(dy * (int)rstride + dx), sh = (o & 3u) * 8u;
          const bool up = o & 4u;
          uint2 w[4][2];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const uint2* p = reinterpret_cast<const uint2*>(ref.plane + (size_t)((o & ~7u) + r * rstride));
            w[r][0] = __ldg(p);
            w[r][1] = __ldg(p + 1);
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const uint32_t a = up ? w[r][0].y : w[r][0].x, b = up ? w[r][1].x : w[r][0].y,
                           c = up ? w[r][1].y : w[r][1].x;
            part = sad4(s[r].x, __funnelshift_r(a, b, sh), part);
            odd = sad4(s[r].y, __funnelshift_r(b, c, sh), odd);
          }
        }
        part += odd;
        part += __shfl_xor_sync(kAll, part, 1);
        return part + 2u * (uint32_t)min(abs(dx) + abs(dy), 32);
      };
      // Seeds: zero, the left block's vector, the above block's (candidates
      // 0..2); rings around the first neighbour's (candidates 3..14).
      const int ns = 1 + (bx > 0) + (by > 0);
      const uint32_t v1 = bx > 0 ? lv : av;
      const int gx = (int)(int16_t)(v1 & 0xffffu), gy = (int)(int16_t)(v1 >> 16);  // zero with no neighbour
      const int hx = (int)(int16_t)(av & 0xffffu), hy = (int)(int16_t)(av >> 16);
      int dx = q == 0 ? 0 : q == 2 ? hx : q == 1 ? gx : gx + rx0, dy = q == 0 ? 0 : q == 2 ? hy : q == 1 ? gy : gy + ry0;
      bool ok = (q < 3 ? q < ns : q < 15) && inplane(dx, dy);
      uint32_t cost = score(ok, dx, dy);
      uint32_t nsad = ok && q < 3;  // this lane's points scored (two lanes a point)
      // A cost is below 2^15: 64 differences of at most 255 and a penalty of 64.
      uint32_t m = __reduce_min_sync(kAll, ok && q < 3 ? cost << 4 | (uint32_t)q : 0xffffffffu);
      uint32_t bc = m >> 4;
      const int seed = m == 0xffffffffu ? 0 : (int)(m & 15u);  // none in the plane: zero
      int bxm = seed == 0 ? 0 : seed == 1 ? gx : hx, bym = seed == 0 ? 0 : seed == 1 ? gy : hy;
      const int cx = bxm, cy = bym;
      int k = q - 3;  // this lane's ring candidate (0..11 where there is one)
      bool known = bxm == gx && bym == gy;
      for (int ring = 0;;) {  // rings `ring`.. of 0, 1, 2 are left around the best
        if (!known) {
          k = q;
          dx = bxm + rx1;
          dy = bym + ry1;
          ok = k < 12 && (k >> 2) >= ring && (uint32_t)(dx - cx + kLowresRange) <= 2u * kLowresRange &&
               (uint32_t)(dy - cy + kLowresRange) <= 2u * kLowresRange && inplane(dx, dy);
          cost = score(ok, dx, dy);
        }
        known = false;
        // The first ring with a point below the best, its least point, the
        // first of equal ones; the rings before it and it are the ones scored.
        const bool live = ok && k >= 0;
        m = __reduce_min_sync(kAll, live && cost < bc ? (uint32_t)(k >> 2) << 24 | cost << 4 | (uint32_t)k : 0xffffffffu);
        const int at = (int)(m >> 24);  // 255: none
        nsad += live && (k >> 2) <= at;
        if (m == 0xffffffffu) break;
        bc = (m >> 4) & 0xfffffu;
        bxm += ring_x((int)(m & 15u));
        bym += ring_y((int)(m & 15u));
        ring = at;
      }
      lv = (uint32_t)(uint16_t)(int16_t)bxm | (uint32_t)(uint16_t)(int16_t)bym << 16;
      if (lane == 0) {
        st_word(words + bx, lv);
        const size_t o = (size_t)pi * n + (size_t)by * bw + bx;
        *reinterpret_cast<uint32_t*>(mv_all + o) = lv;
        if (bx > 0) nsad_all[o - 1] = prev_n;
      }
      prev_n = __reduce_add_sync(kAll, nsad) >> 1;
#pragma unroll
      for (int r = 0; r < 4; ++r) s[r] = sn[r];
      uw = un;
    }
    if (lane == 0) nsad_all[(size_t)pi * n + (size_t)(by + 1) * bw - 1] = prev_n;
  }
}

// The found vectors' SATDs (both lookaheads), a thread per 4x4 tile, four
// per block.
template <class S>
__global__ void __launch_bounds__(256) lowres_cost_kernel(const LowresDesc* pairs, int npairs, const rme_mv* mv_all,
                                                          uint32_t* cost_all) {
  const int bw = pairs[0].bw, n = bw * pairs[0].bh;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, blk = i >> 2;
  uint32_t sat = 0;
  if (blk < (int64_t)n * npairs) {
    const int pi = (int)(blk / n), b = (int)(blk - (int64_t)pi * n), by = b / bw, bx = b - by * bw;
    const int x = bx * 8 + ((int)i & 1) * 4 + kLowresPad, y = by * 8 + ((int)(i >> 1) & 1) * 4 + kLowresPad;
    const LowresDesc &cur = pairs[2 * pi], &ref = pairs[2 * pi + 1];
    const rme_mv m = mv_all[blk];
    const S* sp = reinterpret_cast<const S*>(cur.plane) + (ptrdiff_t)y * cur.stride + x;
    const S* rp = reinterpret_cast<const S*>(ref.plane) + (ptrdiff_t)(y + m.y) * ref.stride + x + m.x;
    constexpr int W = sizeof(S);  // words of a tile row
    uint32_t a[4][W], c[4][W + 1];
    const uintptr_t u = reinterpret_cast<uintptr_t>(rp);
    const uint32_t sh = (uint32_t)(u & 3) * 8u;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(u & ~uintptr_t(3)) + (ptrdiff_t)r * ref.stride * (int)sizeof(S) / 4;
#pragma unroll
      for (int k = 0; k <= W; ++k) c[r][k] = __ldg(w + k);
#pragma unroll
      for (int k = 0; k < W; ++k) a[r][k] = __ldg(reinterpret_cast<const uint32_t*>(sp + (ptrdiff_t)r * cur.stride) + k);
    }
    int d[16];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = e * (int)sizeof(S) / 4, f = e * 8 * (int)sizeof(S) - 32 * k;
        const uint32_t mask = sizeof(S) == 1 ? 0xffu : 0xffffu;
        d[r * 4 + e] = (int)((a[r][k] >> f) & mask) - (int)((__funnelshift_r(c[r][k], c[r][k + 1], sh) >> f) & mask);
      }
    sat = hadamard_satd(d);
  }
  sat += __shfl_xor_sync(kAll, sat, 1);
  sat += __shfl_xor_sync(kAll, sat, 2);
  if ((i & 3) == 0 && blk < (int64_t)n * npairs) cost_all[blk] = sat;
}

// bi_cost (h265_cutree.rs:222-243), one thread per block.
__global__ void lowres_bi_kernel(LowresDesc cur, LowresDesc r0, LowresDesc r1, const rme_mv* m0, const rme_mv* m1,
                                 uint32_t* cost) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= cur.bw * cur.bh) return;
  const int x = (b % cur.bw) * 8, y = (b / cur.bw) * 8;
  const uint8_t* a = r0.plane + (ptrdiff_t)(y + m0[b].y + kLowresPad) * r0.stride + x + m0[b].x + kLowresPad;
  const uint8_t* c = r1.plane + (ptrdiff_t)(y + m1[b].y + kLowresPad) * r1.stride + x + m1[b].x + kLowresPad;
  uint8_t pred[64];
  for (int yy = 0; yy < 8; ++yy)
    for (int xx = 0; xx < 8; ++xx)
      pred[yy * 8 + xx] = (uint8_t)(((int)a[(ptrdiff_t)yy * r0.stride + xx] + c[(ptrdiff_t)yy * r1.stride + xx] + 1) >> 1);
  cost[b] = satd8x8<uint8_t>(cur.plane + (ptrdiff_t)(y + kLowresPad) * cur.stride + x + kLowresPad, cur.stride, pred, 8);
}

// ---- H.264 (h264_lookahead.rs) ----------------------------------------------

// Lookahead::add (h264_lookahead.rs:87-117): over the macroblock grid (8
// samples per macroblock), each sample the rounded mean of the picture's
// 2x2 square at (2x, 2y), its columns and rows clamped to the picture; the
// border replicated (every padded position takes its clamped position's
// value).
template <class S>
__global__ void lowres_build_h264_kernel(const S* __restrict__ pic, int pstride, int w, int h, LowresDesc L) {
  const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y * blockDim.y + threadIdx.y;
  const int rows = L.ph + 2 * kLowresPad;
  if (X >= L.stride || Y >= rows) return;
  const int xx = min(max(X - kLowresPad, 0), L.pw - 1), yy = min(max(Y - kLowresPad, 0), L.ph - 1);
  const int x0 = min(2 * xx, w - 1), x1 = min(2 * xx + 1, w - 1);
  const S* r0 = pic + (ptrdiff_t)min(2 * yy, h - 1) * pstride;
  const S* r1 = pic + (ptrdiff_t)min(2 * yy + 1, h - 1) * pstride;
  const int s = (int)r0[x0] + r0[x1] + r1[x0] + r1[x1];
  reinterpret_cast<S*>(L.plane)[(ptrdiff_t)Y * L.stride + X] = (S)((s + 2) >> 2);
}

// intra_costs (h264_lookahead.rs:146-222), one thread per block: DC from
// the neighbours there are (the block's own mean with none), vertical where
// there is a row above, horizontal where there is a column to the left, the
// bilinear blend of both edges where both are; the least SATD, plus 12.
template <class S>
__global__ void lowres_intra_h264_kernel(LowresDesc L) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= L.bw * L.bh) return;
  const int bx = b % L.bw, by = b / L.bw;
  const S* src = reinterpret_cast<const S*>(L.plane) + (ptrdiff_t)(by * 8 + kLowresPad) * L.stride + bx * 8 + kLowresPad;
  const bool ht = by > 0, hl = bx > 0;
  int t[8], l[8], st = 0, sl = 0;
  for (int i = 0; i < 8; ++i) {
    t[i] = src[i - L.stride];
    l[i] = src[(ptrdiff_t)i * L.stride - 1];
    st += t[i];
    sl += l[i];
  }
  int dc;
  if (ht && hl) {
    dc = (st + sl + 8) >> 4;
  } else if (ht || hl) {
    dc = ((ht ? st : sl) + 4) >> 3;
  } else {
    int sum = 0;
    for (int yy = 0; yy < 8; ++yy)
      for (int xx = 0; xx < 8; ++xx) sum += src[(ptrdiff_t)yy * L.stride + xx];
    dc = (sum + 32) >> 6;
  }
  S pred[64];
  for (int i = 0; i < 64; ++i) pred[i] = (S)dc;
  uint32_t best = satd8x8<S>(src, L.stride, pred, 8);
  if (ht) {
    for (int i = 0; i < 64; ++i) pred[i] = (S)t[i & 7];
    best = min(best, satd8x8<S>(src, L.stride, pred, 8));
  }
  if (hl) {
    for (int i = 0; i < 64; ++i) pred[i] = (S)l[i >> 3];
    best = min(best, satd8x8<S>(src, L.stride, pred, 8));
  }
  if (ht && hl) {
    for (int yy = 0; yy < 8; ++yy)
      for (int xx = 0; xx < 8; ++xx)
        pred[yy * 8 + xx] = (S)((t[xx] * (8 - yy) + l[yy] * (8 - xx) + t[7] * yy + l[7] * xx + 8) >> 4);
    best = min(best, satd8x8<S>(src, L.stride, pred, 8));
  }
  L.intra[b] = best + 12;
}

// One row of 8 samples at any sample address, as 32-bit words (two for u8,
// four for u16), from aligned loads.
template <class S>
struct Row8;
// By 8-byte loads (as lowres_search_kernel), one more than the row may need:
// a plane's memory goes on behind its last row. (Left out where the row is
// aligned, the predicate costs more than the load: 564 us against 491 for
// eight 8-bit 1080p pairs.)
template <int N>
__device__ __forceinline__ void load_words(const void* p, uint32_t (&out)[N]) {
  const uintptr_t u = reinterpret_cast<uintptr_t>(p);
  const uint2* q = reinterpret_cast<const uint2*>(u & ~uintptr_t(7));
  const uint32_t sh = (uint32_t)(u & 3) * 8u;
  const bool up = u & 4;
  uint32_t w[N + 2] = {};
#pragma unroll
  for (int i = 0; i <= N / 2; ++i) {
    const uint2 v = __ldg(q + i);
    w[2 * i] = v.x;
    w[2 * i + 1] = v.y;
  }
  uint32_t t[N + 1];
#pragma unroll
  for (int i = 0; i <= N; ++i) t[i] = up ? w[i + 1] : w[i];
#pragma unroll
  for (int i = 0; i < N; ++i) out[i] = __funnelshift_r(t[i], t[i + 1], sh);
}
// |a - b| of two 16-bit halves, summed onto acc: the larger less the smaller
// of each and a dot product with ones.
__device__ __forceinline__ uint32_t sad2(uint32_t a, uint32_t b, uint32_t acc) {
  uint32_t hi, lo;
  asm("max.u16x2 %0, %1, %2;" : "=r"(hi) : "r"(a), "r"(b));
  asm("min.u16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(b));
  return __dp2a_lo(hi - lo, 0x0101u, acc);
}
template <>
struct Row8<uint8_t> {
  uint32_t w[2];
  __device__ __forceinline__ void load(const uint8_t* p) { load_words<2>(p, w); }
  __device__ __forceinline__ uint32_t sad(const Row8& o, uint32_t acc) const {
    return sad4(w[1], o.w[1], sad4(w[0], o.w[0], acc));
  }
};
template <>
struct Row8<uint16_t> {
  uint32_t w[4];
  __device__ __forceinline__ void load(const uint16_t* p) { load_words<4>(p, w); }
  __device__ __forceinline__ uint32_t sad(const Row8& o, uint32_t acc) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) acc = sad2(w[i], o.w[i], acc);
    return acc;
  }
};

// search (h264_lookahead.rs:227-376), a warp per row of blocks, two lanes
// per candidate (four rows each). The window is the reference's: 16 samples
// into the border, at most 32 from the block. From the zero vector, the left
// and above blocks' vectors (zero where there is no such block) clamped to
// the window, each scored unless it is the best's point, then the hexagon
// (after a step in direction k only k - 1, k and k + 1 are new), at most 16
// steps, then the eight-point square; the SAD + 2 * min(|mx| + |my|, 64) of
// each point, the first least cost taken when strictly below the best (the
// reference's in-order scoring). A pass scores a hexagon step (candidates
// 0..5) together with the square around the same centre (6..13), which is
// the walk's last step when the hexagon has settled there. As
// lowres_search_kernel a chain of steps: eight 1080p pairs 553 us with rows by
// words, ballots and shuffles, 491 us with 8-byte loads and decisions by keys;
// eight 10-bit 720p pairs 505 -> 369 us.
template <class S>
__global__ void __launch_bounds__(kLaWarps * 32) lowres_search_h264_kernel(const LowresDesc* pairs, int npairs,
                                                                           unsigned long long* words_all,
                                                                           unsigned long long* counter,
                                                                           uint32_t* status, rme_mv* mv_all,
                                                                           uint32_t* nsad_all) {
  const int lane = threadIdx.x & 31, q = lane >> 1, half = lane & 1;
  const int bw = pairs[0].bw, bh = pairs[0].bh, n = bw * bh, lim = kLowresPad - 8;
  // This lane's offset from the centre: a point of the hexagon or of the
  // 3x3 square without its centre.
  auto off_x = [](int k) { return (int)((0x32131321134310ull >> (4 * k)) & 15u) - 2; };
  auto off_y = [](int k) { return (int)((0x33322111442002ull >> (4 * k)) & 15u) - 2; };
  const int ofx = off_x(min(q, 13)), ofy = off_y(min(q, 13));
  bool lost = false;
  for (int pi, by; claim_row(counter, npairs, bh, lane, pi, by);) {
    const LowresDesc cur = pairs[2 * pi], ref = pairs[2 * pi + 1];
    unsigned long long* words = words_all + (size_t)pi * n + (size_t)by * bw;
    const unsigned long long* up = words - bw;
    const int y = by * 8;
    const S* srow = reinterpret_cast<const S*>(cur.plane) + (ptrdiff_t)(y + kLowresPad + half * 4) * cur.stride + kLowresPad;
    const S* rrow = reinterpret_cast<const S*>(ref.plane) + (ptrdiff_t)(y + kLowresPad + half * 4) * ref.stride + kLowresPad;
    const int ly = max(-y - lim, -2 * kLowresRange), hy = min(cur.ph - 8 - y + lim, 2 * kLowresRange);
    Row8<S> s[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) s[r].load(srow + (ptrdiff_t)r * cur.stride);
    unsigned long long uw = by > 0 ? ld_word(up) : 0ull;
    uint32_t lv = 0;
    for (int bx = 0; bx < bw; ++bx) {
      const int x = bx * 8;
      const S* rb = rrow + x;
      if (by > 0) lost = wait_above(up + bx, uw, status, lost);
      const uint32_t av = (uint32_t)uw;
      Row8<S> sn[4];
      unsigned long long un = 0ull;
      const int xn = bx + 1 < bw ? x + 8 : x;
#pragma unroll
      for (int r = 0; r < 4; ++r) sn[r].load(srow + (ptrdiff_t)r * cur.stride + xn);
      if (by > 0 && bx + 1 < bw) un = ld_word(up + bx + 1);
      const int lx = max(-x - lim, -2 * kLowresRange), hx = min(cur.pw - 8 - x + lim, 2 * kLowresRange);
      auto score = [&](bool ok, int dx, int dy) -> uint32_t {
        uint32_t part = 0, odd = 0;
        if (ok) {
          Row8<S> a[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) a[r].load(rb + (ptrdiff_t)(dy + r) * ref.stride + dx);
#pragma unroll
          for (int r = 0; r < 4; ++r) (r & 1 ? odd : part) = s[r].sad(a[r], r & 1 ? odd : part);
        }
        part += odd;
        part += __shfl_xor_sync(kAll, part, 1);
        return ok ? part + 2u * (uint32_t)min(abs(dx) + abs(dy), 64) : 0xffffffffu;
      };
      auto inwin = [&](int dx, int dy) { return dx >= lx && dx <= hx && dy >= ly && dy <= hy; };
      // The zero vector and the two candidates, scored at once, resolved in
      // the reference's order.
      const int c0x = min(max((int)(int16_t)(lv & 0xffffu), lx), hx), c0y = min(max((int)(int16_t)(lv >> 16), ly), hy);
      const int c1x = min(max((int)(int16_t)(av & 0xffffu), lx), hx), c1y = min(max((int)(int16_t)(av >> 16), ly), hy);
      int dx = q == 1 ? c0x : q == 2 ? c1x : 0, dy = q == 1 ? c0y : q == 2 ? c1y : 0;
      const uint32_t sc = score(q < 3, dx, dy);
      const uint32_t z = __shfl_sync(kAll, sc, 0), k0 = __shfl_sync(kAll, sc, 2), k1 = __shfl_sync(kAll, sc, 4);
      uint32_t bc = z, nsad = 1;
      int bxm = 0, bym = 0;
      if (c0x != 0 || c0y != 0) {
        ++nsad;
        if (k0 < bc) {
          bc = k0;
          bxm = c0x;
          bym = c0y;
        }
      }
      if (c1x != bxm || c1y != bym) {
        ++nsad;
        if (k1 < bc) {
          bc = k1;
          bxm = c1x;
          bym = c1y;
        }
      }
      uint32_t live = 0x3f, lsad = 0;  // the hexagon's new points; this lane's points scored (two lanes a point)
      for (int it = 0;; ++it) {
        dx = bxm + ofx;
        dy = bym + ofy;
        const bool ok = (q < 6 ? it < kLowresRange && ((live >> q) & 1) : q < 14) && inwin(dx, dy);
        const uint32_t cost = score(ok, dx, dy);
        // Keys of cost and place: the minimum is the decision. (A cost is below
        // 2^19: 64 differences of at most 4095 and a penalty of 128.)
        const uint32_t key = ok ? cost << 4 | (uint32_t)q : 0xffffffffu;
        uint32_t m = __reduce_min_sync(kAll, q < 6 ? key : 0xffffffffu);
        lsad += ok && q < 6;
        const bool step = m >> 4 < bc;
        if (!step) {  // settled: the square around the hexagon's centre
          lsad += ok && q >= 6;
          m = __reduce_min_sync(kAll, q < 6 ? 0xffffffffu : key);
        }
        const int k = (int)(m & 15u);
        if (m >> 4 < bc) {
          bc = m >> 4;
          bxm += off_x(k);
          bym += off_y(k);
        }
        if (!step) break;
        const uint32_t r = 7u << (k + 5);
        live = (r | r >> 6 | r >> 12) & 0x3f;
      }
      lv = (uint32_t)(uint16_t)(int16_t)bxm | (uint32_t)(uint16_t)(int16_t)bym << 16;
      if (lane == 0) st_word(words + bx, lv);
      nsad += __reduce_add_sync(kAll, lsad) >> 1;
      if (lane == 0) {
        const size_t o = (size_t)pi * n + (size_t)by * bw + bx;
        *reinterpret_cast<uint32_t*>(mv_all + o) = lv;
        nsad_all[o] = nsad;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) s[r] = sn[r];
      uw = un;
    }
  }
}

// The average-of-two cost of estimate() (h264_lookahead.rs:417-432), one
// thread per block: the SATD against the rounded average of the blocks the
// two vectors point at.
template <class S>
__global__ void lowres_bi_h264_kernel(LowresDesc cur, LowresDesc r0, LowresDesc r1, const rme_mv* m0, const rme_mv* m1,
                                      uint32_t* cost) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= cur.bw * cur.bh) return;
  const int x = (b % cur.bw) * 8, y = (b / cur.bw) * 8;
  const S* a = reinterpret_cast<const S*>(r0.plane) + (ptrdiff_t)(y + m0[b].y + kLowresPad) * r0.stride + x + m0[b].x +
               kLowresPad;
  const S* c = reinterpret_cast<const S*>(r1.plane) + (ptrdiff_t)(y + m1[b].y + kLowresPad) * r1.stride + x + m1[b].x +
               kLowresPad;
  S pred[64];
  for (int yy = 0; yy < 8; ++yy)
    for (int xx = 0; xx < 8; ++xx)
      pred[yy * 8 + xx] = (S)(((int)a[(ptrdiff_t)yy * r0.stride + xx] + c[(ptrdiff_t)yy * r1.stride + xx] + 1) >> 1);
  const S* src = reinterpret_cast<const S*>(cur.plane) + (ptrdiff_t)(y + kLowresPad) * cur.stride + x + kLowresPad;
  cost[b] = satd8x8<S>(src, cur.stride, pred, 8);
}

// The wavefront's wait on a word nothing publishes, with a short poll limit:
// the failure path of a dependency that never completes, taken on purpose.
__global__ void probe_wait_kernel(const unsigned long long* word, uint32_t limit, uint32_t* status) {
  if ((threadIdx.x & 31) == 0) {
    unsigned long long w = ld_word(word);
    wait_word(word, w, status, false, limit);
  }
}

}  // namespace

cudaError_t launch_probe_wait(const unsigned long long* word, uint32_t limit, uint32_t* status, cudaStream_t s) {
  probe_wait_kernel<<<1, 32, 0, s>>>(word, limit, status);
  return cudaGetLastError();
}

cudaError_t launch_lowres_build(const DevPlanes& pic, int bd, int w, int h, const LowresDesc& L, cudaStream_t s) {
  dim3 blk(32, 8), grd((L.stride + 31) / 32, (L.ph + 2 * kLowresPad + 7) / 8);
  if (L.h264) {
    if (bd == 8) {
      lowres_build_h264_kernel<uint8_t><<<grd, blk, 0, s>>>((const uint8_t*)pic.base + pic.origin, pic.stride, w, h, L);
      lowres_intra_h264_kernel<uint8_t><<<(L.bw * L.bh + 127) / 128, 128, 0, s>>>(L);
    } else {
      lowres_build_h264_kernel<uint16_t>
          <<<grd, blk, 0, s>>>((const uint16_t*)pic.base + pic.origin, pic.stride, w, h, L);
      lowres_intra_h264_kernel<uint16_t><<<(L.bw * L.bh + 127) / 128, 128, 0, s>>>(L);
    }
    return cudaGetLastError();
  }
  if (bd == 8)
    lowres_build_kernel<uint8_t><<<grd, blk, 0, s>>>((const uint8_t*)pic.base + pic.origin, pic.stride, w, h, bd, L);
  else
    lowres_build_kernel<uint16_t><<<grd, blk, 0, s>>>((const uint16_t*)pic.base + pic.origin, pic.stride, w, h, bd, L);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  lowres_intra_kernel<<<(L.bw * L.bh + 127) / 128, 128, 0, s>>>(L);
  return cudaGetLastError();
}

cudaError_t launch_lowres_search(const LowresDesc* pairs, int npairs, const LowresDesc& first,
                                 unsigned long long* words, unsigned long long* counter, uint32_t* status,
                                 uint32_t* cost, rme_mv* mv, uint32_t* nsad, int max_ctas, cudaStream_t s) {
  const int64_t rows = (int64_t)first.bh * npairs, tiles = (int64_t)first.bw * first.bh * npairs * 4;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(max_ctas, (rows + kLaWarps - 1) / kLaWarps));
  const unsigned cgrid = (unsigned)((tiles + 255) / 256);
  if (!first.h264)
    lowres_search_kernel<<<grid, kLaWarps * 32, 0, s>>>(pairs, npairs, words, counter, status, mv, nsad);
  else if (first.bytes == 1)
    lowres_search_h264_kernel<uint8_t><<<grid, kLaWarps * 32, 0, s>>>(pairs, npairs, words, counter, status, mv, nsad);
  else
    lowres_search_h264_kernel<uint16_t><<<grid, kLaWarps * 32, 0, s>>>(pairs, npairs, words, counter, status, mv, nsad);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (first.bytes == 1)
    lowres_cost_kernel<uint8_t><<<cgrid, 256, 0, s>>>(pairs, npairs, mv, cost);
  else
    lowres_cost_kernel<uint16_t><<<cgrid, 256, 0, s>>>(pairs, npairs, mv, cost);
  return cudaGetLastError();
}

cudaError_t launch_lowres_bi(const LowresDesc& cur, const LowresDesc& r0, const LowresDesc& r1, const rme_mv* m0,
                             const rme_mv* m1, uint32_t* cost, cudaStream_t s) {
  const int grid = (cur.bw * cur.bh + 127) / 128;
  if (!cur.h264)
    lowres_bi_kernel<<<grid, 128, 0, s>>>(cur, r0, r1, m0, m1, cost);
  else if (cur.bytes == 1)
    lowres_bi_h264_kernel<uint8_t><<<grid, 128, 0, s>>>(cur, r0, r1, m0, m1, cost);
  else
    lowres_bi_h264_kernel<uint16_t><<<grid, 128, 0, s>>>(cur, r0, r1, m0, m1, cost);
  return cudaGetLastError();
}

}  // namespace rme
