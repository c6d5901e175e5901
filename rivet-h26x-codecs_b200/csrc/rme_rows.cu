// The HEVC STANDALONE search in its row form (frames without AMP units): a
// group of threads owns a row of blocks of one size and reference and
// searches it left to right.
//
// The STANDALONE rule makes a block read its left and upper neighbours of
// its size and its parent one size up, so each size is a wavefront, and a
// frame's time is the longest chain of blocks through them: nothing here is
// bound by bandwidth or by the number of operations, all of it by the
// latency of one block's dependent steps. Hence
//   - no queue between blocks: a finished block publishes its vector as one
//     word (tag, vector), and a block waits (bounded) for its upper and
//     parent words only, loaded a block ahead; its left vector is at hand.
//     A wait that runs out ends its group's row, its CTA and, by the status
//     word, soon the launch;
//   - several warps a block and few steps: an 8x8 block has 64 threads, a
//     16x16 or 32x32 block 128, a 64x64 block 256, so that a step is a few
//     loads a thread, a short sum and one barrier. More threads would repeat
//     the decisions, which every warp of a group takes, for less: 128 threads
//     an 8x8 block or 256 a 16x16 block gain 0 to 4 % on one 1080p frame and
//     lose 8 to 20 % on launches of two to forty; half as many threads lose
//     10 to 60 %;
//   - speculation instead of dependence: the first step of an 8x8 or 16x16
//     block scores all seeds and, around the two likeliest, the twelve points
//     two diamond rounds can reach; later steps, and those of larger blocks,
//     score two or three rounds at once;
//   - a 32x32 or 64x64 block's diamond reads a window staged in shared memory
//     while the seeds are scored, a thread its words' twelve candidates;
//   - the next block's source is on its way while a block is searched;
//   - 128 registers a thread, two CTAs an SM: three (80 registers) lose 8 to
//     25 % at every launch size.
// Which candidates are scored, in which order they win and how many are
// counted is the reference's walk (h265_me.rs:3749-3922), as hevc_task runs
// it with one warp. Search kernel, one B200, before (dataflow or a warp a
// row, the faster) and now: one 1080p frame of two references 3.8 -> 1.6 ms,
// 850x478 1.59 -> 0.60 ms, twelve 1080p frames 13.4 -> 7.8 ms, one 2160p
// 10-bit frame of four references 33 -> 10.4 ms. Rows read by 8-byte loads
// (fewer passes through L1, more selections) lose 1 to 8 %, the sub-sample
// planes brought into L1 ahead 0 to 8 %: issue and latency bind, not the loads.
//
// A CTA is 256 threads: one row of 64x64 blocks, two of 32x32 or 16x16, four
// of 8x8. Rows are taken in the order the host pushed them, each after the
// rows it reads, so the owner of a row that is waited for is always running.
#include <algorithm>

#include "rme_search_impl.cuh"

namespace rme {
namespace {

constexpr int kRowThreads = 256;

// Threads that share a block of N x N samples.
constexpr int row_group(int n) { return n == 64 ? 256 : n == 8 ? 64 : 128; }

// A step's candidates of an 8x8 or 16x16 block: 32 slots.
constexpr int kSlots = 32;
constexpr uint32_t kNoKey = 0xffffffffu;  // a slot without a candidate

template <class S, int N>
struct SmallSmem {
  uint32_t src[2][N * N * sizeof(S) / 4];
  uint32_t key[2][kSlots];  // cost << 5 | slot (a cost is below 2^26: at most 64 * 64 * 4095 and the largest rate)
  uint32_t satd[2][16];     // half, quarter
  volatile uint32_t lost;   // a wait of the group gave up
};

// The points three rounds of the small diamond can reach, in an order in
// which, whichever way the rounds before moved, a round's new points come in
// the reference's order ((1,0), (-1,0), (0,1), (0,-1) around the new best):
// the centre, the first round (1..4), then (2,0), (-2,0), (1,1), (1,-1),
// (-1,1), (-1,-1), (0,2), (0,-2) (5..12), then (3,0), (-3,0), (2,1), (2,-1),
// (-2,1), (-2,-1), (1,2), (1,-2), (-1,2), (-1,-2), (0,3), (0,-3) (13..24).
// Offsets + 3 as hex digits, 16 points a word, the lowest digit first.
__device__ __forceinline__ int around_x(int q) {
  return (int)(((q < 16 ? 0x5063322441533243ull : 0x332244115ull) >> (4 * (q & 15))) & 15u) - 3;
}
__device__ __forceinline__ int around_y(int q) {
  return (int)(((q < 16 ? 0x4331524243324333ull : 0x061515242ull) >> (4 * (q & 15))) & 15u) - 3;
}
// The second round's new points after the first moved in direction j.
__device__ __forceinline__ constexpr uint32_t second_round(int j) {
  return j == 0 ? 0x1a0u : j == 1 ? 0x640u : j == 2 ? 0xa80u : 0x1500u;
}
// The third round's points after the second moved to point 5 + k: all four
// (the first round's points among them, which cannot win: they cost no less
// than the point the first round moved to), and the new ones.
__constant__ uint32_t c_third[8] = {
    1u << 13 | 1u << 1 | 1u << 15 | 1u << 16, 1u << 14 | 1u << 2 | 1u << 17 | 1u << 18,
    1u << 15 | 1u << 3 | 1u << 19 | 1u << 1,  1u << 16 | 1u << 4 | 1u << 1 | 1u << 20,
    1u << 3 | 1u << 17 | 1u << 21 | 1u << 2,  1u << 4 | 1u << 18 | 1u << 2 | 1u << 22,
    1u << 19 | 1u << 21 | 1u << 23 | 1u << 3, 1u << 20 | 1u << 22 | 1u << 4 | 1u << 24};

// Waits for another row's published word, already loaded once (`w`): at most
// L.wait_polls polls, then the status word's timeout bit; fewer once the launch
// has failed elsewhere. Returns the word, of another tag where it gave up. (The
// first polls follow one another, later ones back off, as wait_word's.)
__device__ __noinline__ unsigned long long poll_published(const LaunchDesc& L, const unsigned long long* p, uint32_t tag,
                                                          unsigned long long w) {
  uint32_t ns = 32;
  for (uint32_t it = 0; (uint32_t)(w >> 32) != tag; ++it) {
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
// Sets the group's `lost` (shared memory) where it gave up. All of a group must
// then know before a step whose number the words decide (a walk's): with
// different words some would wait at a barrier for ever. A small block's warps
// each wait by themselves, read `lost` behind the first step's barrier and end
// the row there; a large block's words are waited for by one warp and read from
// shared memory by all (a barrier more, few registers: there the check cost
// spills).
__device__ __forceinline__ void wait_published(const LaunchDesc& L, const unsigned long long* p, uint32_t tag,
                                               unsigned long long& w, volatile uint32_t& lost) {
  if ((uint32_t)(w >> 32) == tag) return;
  w = poll_published(L, p, tag, w);
  if ((uint32_t)(w >> 32) != tag) lost = 1u;
}

// What a row's blocks share, read once.
template <class S>
struct RowInfo {
  const DevPlanes src, ref;
  unsigned long long* mvf;
  rme_result* out;
  const uint32_t tag;
  const int nref, r, nbx, base;          // this level
  const int pnbx, pbase, pshift;         // the parents' level, log2 of its size (pnbx 0: none over this row)
  const int width, height, padm, range, rings, cross;
  const float lam;
};
template <class S>
__device__ __forceinline__ RowInfo<S> row_info(const FrameDesc& F, int l, int r, int y) {
  int psize = l > 0 ? F.size[l - 1] : 0;
  if (psize && y / psize >= F.nby[l - 1]) psize = 0;
  return RowInfo<S>{F.src,    F.ref[r],  F.mvf,
                    F.out,    F.tag,     F.nref,
                    r,        F.nbx[l],  F.base[l],
                    psize ? F.nbx[l - 1] : 0, psize ? F.base[l - 1] + (y / psize) * F.nbx[l - 1] : 0, 31 - __clz(psize | 1),
                    F.width,  F.height,  F.pad - 4,
                    F.search_range, F.search_rings, F.quarter_cross, F.lam};
}

// The totals of a thread's rows (thread 0 of each group counts).
struct RowCount {
  uint32_t tasks = 0, sad = 0, satd = 0, area = 0;
};

// A row of 8x8 or 16x16 blocks by T threads. False, for the whole group, where
// a wait gave up (the launch has failed).
template <class S, int N, int T>
__device__ bool small_row(const LaunchDesc& L, const FrameDesc& F, int l, int r, int row, SmallSmem<S, N>& sm, int tid,
                          int bar, RowCount& cnt) {
  constexpr int SPW = 4 / (int)sizeof(S), WR = N / SPW, NSRC = N * WR, TW = N / 4, NT = TW * TW, WPT = 4 / SPW;
  constexpr int PS = (NSRC + T - 1) / T;  // source words a thread stages
  const int y = row * N, lane = tid & 31;
  const RowInfo<S> I = row_info<S>(F, l, r, y);
  const unsigned long long* const up = I.mvf + ((ptrdiff_t)(I.base + (row - 1) * I.nbx)) * I.nref + I.r;
  const unsigned long long* const par = I.mvf + (ptrdiff_t)I.pbase * I.nref + I.r;
  const int stride = I.ref.stride, range = I.range;
  const float lam = I.lam;
  // The word of the parent of the block at x, or null where there is none.
  auto parent_of = [&](int x) -> const unsigned long long* {
    const int px = x >> I.pshift;
    return px < I.pnbx ? par + (ptrdiff_t)px * I.nref : nullptr;
  };
  auto load_src = [&](int bx, uint32_t (&v)[PS]) {  // aligned: N and the pad are whole words
#pragma unroll
    for (int k = 0; k < PS; ++k) {
      const int i = tid + k * T;
      v[k] = i < NSRC ? RME_LD32(reinterpret_cast<const uint32_t*>(plane_at<S>(I.src, 0, bx * N, y + i / WR)) + i % WR)
                      : 0u;
    }
  };
  auto store_src = [&](uint32_t* dst, const uint32_t (&v)[PS]) {
#pragma unroll
    for (int k = 0; k < PS; ++k)
      if (tid + k * T < NSRC) dst[tid + k * T] = v[k];
  };
  uint32_t nsrc[PS];
  load_src(0, nsrc);
  store_src(sm.src[0], nsrc);
  if (tid == 0) sm.lost = 0u;
  unsigned long long uw = row > 0 ? ld_relaxed64(up) : 0ull, pw = 0ull;
  if (const unsigned long long* p = parent_of(0)) pw = ld_relaxed64(p);
  uint32_t lv = 0;
  int buf = 0;  // the key buffer of the next step
  // This thread's slot of a step, and its place around a centre: as one of
  // the first step's two (slots 1..13 and 16..28), as the only one (0..12).
  const int slot = tid / (T / kSlots), q2 = slot < 16 ? slot - 1 : slot - 16;
  const bool in2 = q2 >= 0 && q2 < 13;
  const int ax = around_x(in2 ? q2 : 0), ay = around_y(in2 ? q2 : 0), cxo = around_x(slot), cyo = around_y(slot);
  group_sync<T>(bar);
  for (int bx = 0; bx < I.nbx; ++bx) {
    const int x = bx * N;
    const uint32_t* const src = sm.src[bx & 1];
    if (row > 0) wait_published(L, up + (ptrdiff_t)bx * I.nref, I.tag, uw, sm.lost);
    const unsigned long long* const pp = parent_of(x);
    if (pp) wait_published(L, pp, I.tag, pw, sm.lost);
    __syncwarp();
    const uint32_t uv = (uint32_t)uw, pv = pp ? (uint32_t)pw : 0u;
    // The next block's words and source, on their way during the search.
    if (bx + 1 < I.nbx) {
      if (row > 0) uw = ld_relaxed64(up + (ptrdiff_t)(bx + 1) * I.nref);
      if (const unsigned long long* p = parent_of(x + N)) pw = ld_relaxed64(p);
      load_src(bx + 1, nsrc);
    }
    // The AMVP pair (left, upper when another; zero-filled) and the seeds
    // [zero, mvp0, mvp1, parent], floored to whole samples and clamped.
    uint32_t m0 = 0, m1 = 0;
    if (bx > 0) {
      m0 = lv;
      if (row > 0 && uv != lv) m1 = uv;
    } else if (row > 0) {
      m0 = uv;
    }
    const int p0x = mvx_of(m0), p0y = mvy_of(m0), p1x = mvx_of(m1), p1y = mvy_of(m1);
    const int lox = -I.padm - x, hix = I.width + I.padm - N - x, loy = -I.padm - y, hiy = I.height + I.padm - N - y;
    auto to_x = [&](int v) { return min(max(v >> 2, lox), hix); };
    auto to_y = [&](int v) { return min(max(v >> 2, loy), hiy); };
    const int zx = to_x(0), zy = to_y(0), ux = to_x(p0x), uy = to_y(p0y), vx = to_x(p1x), vy = to_y(p1y);
    const int wx = to_x(mvx_of(pv)), wy = to_y(mvy_of(pv));
    // A seed on an earlier one's point is not scored again (`tried`).
    const bool k1 = ux != zx || uy != zy, k2 = (vx != zx || vy != zy) && (vx != ux || vy != uy);
    const bool k3 = pp && (wx != zx || wy != zy) && (wx != ux || wy != uy) && (wx != vx || wy != vy);
    uint32_t nsad = 1u + k1 + k2 + k3, nsatd = 9;
    const S* const org = plane_at<S>(I.ref, 0, x, y);
    auto inside = [&](int fx, int fy) { return fx >= lox && fx <= hix && fy >= loy && fy <= hiy; };
    // A candidate's SAD over its slot's LPC lanes (rows sub, sub + LPC, ...)
    // and its key into the slot `at`, then the barrier; lane i of every warp
    // gets slot i's key.
    auto score = [&](auto lanes, int at, bool ok, int fx, int fy) -> uint32_t {
      constexpr int LPC = decltype(lanes)::value, RPL = N / LPC, UN = RPL * WR <= 16 ? RPL : 16 / WR;
      const int sub = tid % LPC;
      uint32_t acc = 0;
      // The key but for the distortion, worked out while the loads are on
      // their way (behind the sum it would lengthen the step).
      const uint32_t low = hevc_rate(lam, fx * 4, fy * 4, p0x, p0y, p1x, p1y) << 5 | (uint32_t)at;
      if (ok) {
        const S* rp = org + (ptrdiff_t)(fy + sub) * stride + fx;
#pragma unroll
        for (int k0 = 0; k0 < RPL; k0 += UN) {
          uint32_t a[UN][WR];
#pragma unroll
          for (int k = 0; k < UN; ++k) ldwords<WR>(rp + (ptrdiff_t)(k0 + k) * LPC * stride, a[k]);
#pragma unroll
          for (int k = 0; k < UN; ++k)
#pragma unroll
            for (int c = 0; c < WR; ++c) acc = vsad(src[(sub + (k0 + k) * LPC) * WR + c], a[k][c], acc, S());
        }
      }
#pragma unroll
      for (int o = LPC >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
      uint32_t* c = sm.key[buf];
      buf ^= 1;
      if (sub == 0) c[at] = ok ? (acc << 5) + low : kNoKey;
      group_sync<T>(bar);
      return c[lane];
    };
    // First step. Slot 0 the zero seed; 1..13 mvp0 with the points around
    // it; 14 mvp1 where the parent takes 16..28, else 16..28 mvp1 with the
    // points around it.
    const int gx = pp ? wx : vx, gy = pp ? wy : vy;
    uint32_t key;
    {
      const bool a = slot < 16;
      int fx = (a ? ux : gx) + ax, fy = (a ? uy : gy) + ay;
      bool ok = in2 && (ax | ay) != 0 ? abs(ax) <= range && abs(ay) <= range && inside(fx, fy) : in2;
      if (slot == 0) {
        fx = zx;
        fy = zy;
        ok = true;
      } else if (slot == 14) {
        fx = vx;
        fy = vy;
        ok = pp != nullptr;
      }
      key = score(std::integral_constant<int, T / kSlots>{}, slot, ok, fx, fy);
    }
    const bool lost = sm.lost != 0u;
    // The best seed, the first in order (slots 0, 1, 14, 16) of least cost.
    uint32_t best = __reduce_min_sync(kFull, (0x14003u >> lane) & 1u ? key : kNoKey);
    const int s0 = (int)(best & 31u);
    const int ox = s0 == 0 ? zx : s0 == 1 ? ux : s0 == 14 ? vx : gx, oy = s0 == 0 ? zy : s0 == 1 ? uy : s0 == 14 ? vy : gy;
    int fbx = ox, fby = oy;        // the best whole-sample point
    uint32_t bcost = best >> 5;
    int base = ox == ux && oy == uy ? 1 : ox == gx && oy == gy ? 16 : -1;  // its points' slots, where scored
    // The diamond, two rounds a step.
    if (lost) break;
    for (int it = 0, rings = 0;;) {
      while (it < 2 * range) {
        if (base < 0) {
          const int fx = fbx + cxo, fy = fby + cyo;
          const bool ok = slot > 0 && slot < 25 && abs(fx - ox) <= range && abs(fy - oy) <= range && inside(fx, fy);
          key = score(std::integral_constant<int, T / kSlots>{}, slot, ok, fx, fy);
          base = 0;
        }
        // The first round's minimum and, for each way it can move, the
        // second's: five minima that wait for nothing but the keys.
        const uint32_t there = __ballot_sync(kFull, key != kNoKey) >> base;  // bit q: point q is scored
        const int q = lane - base;
        const uint32_t bit = q >= 0 && q < (base == 0 ? 25 : 13) ? 1u << q : 0u;
        const uint32_t m1 = __reduce_min_sync(kFull, bit & 0x1eu ? key : kNoKey);
        uint32_t m2, second;
        {
          uint32_t mj[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) mj[j] = __reduce_min_sync(kFull, bit & second_round(j) ? key : kNoKey);
          const int j = (int)(m1 & 31u) - base - 1;
          m2 = j == 0 ? mj[0] : j == 1 ? mj[1] : j == 2 ? mj[2] : mj[3];
          second = second_round(j);
        }
        const int left = 2 * range - it;  // rounds allowed, this one the first
        nsad += __popc(there & 0x1eu);
        if (!(m1 >> 5 < bcost)) break;
        uint32_t won = m1;
        ++it;
        bool more = left > 1;
        if (more) {
          nsad += 1u + __popc(there & second);  // the fourth point is the old best
          more = m2 >> 5 < m1 >> 5;
        }
        if (more) {
          won = m2;
          ++it;
          more = left > 2;
          if (more && base == 0) {
            const uint32_t third = c_third[(m2 & 31u) - 5u];
            nsad += __popc(there & third);
            const uint32_t m3 = __reduce_min_sync(kFull, bit & third & ~0x1eu ? key : kNoKey);
            more = m3 >> 5 < m2 >> 5;
            if (more) {
              won = m3;
              ++it;
            }
          }
        }
        const int qw = (int)(won & 31u) - base;
        bcost = won >> 5;
        fbx += around_x(qw);
        fby += around_y(qw);
        if (!more) break;
        base = -1;
      }
      if (rings >= I.rings) break;
      ++rings;
      // The 24 ring points at 4, 8, 16 around the settled point, in order;
      // a move restarts the diamond.
      auto ring_x = [](int k) {
        const int d = k < 8 ? 4 : k < 16 ? 8 : 16, c = k & 7;
        return c == 0 || c == 4 || c == 6 ? d : c == 1 || c == 5 || c == 7 ? -d : 0;
      };
      auto ring_y = [](int k) {
        const int d = k < 8 ? 4 : k < 16 ? 8 : 16, c = k & 7;
        return c == 2 || c == 4 || c == 5 ? d : c == 3 || c == 6 || c == 7 ? -d : 0;
      };
      const int fx = fbx + ring_x(slot), fy = fby + ring_y(slot);
      const bool ok = slot < 24 && abs(fx - ox) <= range && abs(fy - oy) <= range && inside(fx, fy);
      key = score(std::integral_constant<int, T / kSlots>{}, slot, ok, fx, fy);
      nsad += __popc(__ballot_sync(kFull, key != kNoKey));
      const uint32_t m = __reduce_min_sync(kFull, key);
      if (!(m >> 5 < bcost)) break;
      bcost = m >> 5;
      fbx += ring_x((int)(m & 31u));
      fby += ring_y((int)(m & 31u));
      it = 0;
      base = -1;
    }
    const uint32_t int_cost = bcost;
    const int imx = fbx * 4, imy = fby * 4;

    // refine_subpel: the start and the half ring in one step, then the
    // quarter ring around the winner; a thread per 4x4 tile, NT threads a
    // candidate. at(k, dx, dy): candidate k's offset from the whole-sample
    // point in quarter samples, and whether it is scored. Returns lane i's
    // candidate's key.
    const S* const whole = org + (ptrdiff_t)fby * stride + fbx;
    auto satd = [&](auto count, auto at) -> uint32_t {
      constexpr int NC = decltype(count)::value;
      uint32_t* kb = sm.key[buf];
      buf ^= 1;
#pragma unroll
      for (int j0 = 0; j0 < NC * NT; j0 += T) {
        const int j = j0 + tid, k = j / NT, tile = j % NT, ty = tile / TW, tx = tile % TW;
        if (j0 + (tid & ~31) >= NC * NT) break;  // none of the warp's
        int dx = 0, dy = 0;
        uint32_t v = 0, low = 0;
        const bool ok = k < NC && at(k, dx, dy);
        if (ok) {
          const S* q = whole + (int64_t)((dy & 3) * 4 + (dx & 3)) * I.ref.plane_elems +
                       (ptrdiff_t)((dy >> 2) + ty * 4) * stride + ((dx >> 2) + tx * 4);
          uint32_t pr[4][WPT], sw[4][WPT];
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) ldwords<WPT>(q + (ptrdiff_t)rr * stride, pr[rr]);
          low = hevc_rate(lam, imx + dx, imy + dy, p0x, p0y, p1x, p1y);
#pragma unroll
          for (int rr = 0; rr < 4; ++rr)
#pragma unroll
            for (int w = 0; w < WPT; ++w) sw[rr][w] = src[(ty * 4 + rr) * WR + tx * WPT + w];
          v = satd4x4<WPT>(sw, pr);
        }
#pragma unroll
        for (int o = NT >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        if (tile == 0 && k < NC) {
          kb[k] = ok ? (v + low) << 5 | (uint32_t)k : kNoKey;
          sm.satd[NC == 8][k] = v;
        }
      }
      group_sync<T>(bar);
      return lane < NC ? kb[lane] : kNoKey;
    };
    auto half_at = [](int k, int& dx, int& dy) {
      const int q = k == 0 ? 4 : k <= 4 ? k - 1 : k, qy = q / 3;
      dx = (q - qy * 3 - 1) * 2;
      dy = (qy - 1) * 2;
      return true;
    };
    uint32_t m = __reduce_min_sync(kFull, satd(std::integral_constant<int, 9>{}, half_at));
    int hdx, hdy;
    half_at((int)(m & 31u), hdx, hdy);
    int bmx = imx + hdx, bmy = imy + hdy;
    uint32_t bc = m >> 5, bsatd = sm.satd[0][m & 31u];
    const int cross = I.cross;
    auto quarter_at = [&](int k, int& dx, int& dy) {
      const int q = k < 4 ? k : k + 1, qy = q / 3, ex = q - qy * 3 - 1, ey = qy - 1;
      dx = hdx + ex;
      dy = hdy + ey;
      return !(cross != 0 && ex != 0 && ey != 0);
    };
    store_src(sm.src[(bx + 1) & 1], nsrc);
    const uint32_t qkey = satd(std::integral_constant<int, 8>{}, quarter_at);
    nsatd += cross ? 4 : 8;
    m = __reduce_min_sync(kFull, qkey);
    if (m != kNoKey && m >> 5 < bc) {
      int dx, dy;
      bc = m >> 5;
      bsatd = sm.satd[1][m & 31u];
      quarter_at((int)(m & 31u), dx, dy);
      bmx = imx + dx;
      bmy = imy + dy;
    }
    lv = (uint32_t)(uint16_t)(int16_t)bmx | (uint32_t)(uint16_t)(int16_t)bmy << 16;
    if (tid == 0) {
      const ptrdiff_t t = (ptrdiff_t)(I.base + row * I.nbx + bx) * I.nref + I.r;
      st_relaxed64(I.mvf + t, (unsigned long long)I.tag << 32 | lv);
      write_result(I.out + t, bmx, bmy, I.r, bc, bsatd, imx, imy, int_cost, nsad, nsatd, 0);
      cnt.tasks += 1;
      cnt.sad += nsad;
      cnt.satd += nsatd;
    }
  }
  cnt.area = N * N;
  group_sync<T>(bar);  // the last block's keys and source are read: the buffers may be reused
  return sm.lost == 0u;
}

// A 32x32 or 64x64 block's window: the reference's integer plane around a
// centre, kMargin samples beyond the block on every side, as the aligned
// words that hold it. A diamond step from any point within kMargin - 2 of the
// centre reads the window only.
constexpr int kMargin = 8;
template <class S, int N>
struct BigSmem {
  static constexpr int ROWS = N + 2 * kMargin, WRW = (N + 2 * kMargin) * (int)sizeof(S) / 4 + 1;
  uint32_t src[2][N * N * sizeof(S) / 4];
  uint32_t win[ROWS * WRW];
  uint32_t cost[3][32];  // a step's distortions, summed over the warps; in turn, the next one cleared a step ahead
  uint32_t word[2];        // the upper and the parent block's vectors
  volatile uint32_t lost;  // a wait gave up
};

// A row of 32x32 or 64x64 blocks by T threads: a thread has PW words of the
// block for the SADs (a warp's lanes side by side in a row) and a 4x4 tile
// for the SATDs, and scores every candidate of a step on them; the warps'
// sums meet in shared memory, one barrier a step. False as small_row (where
// a wait gave up the row goes on, and its later waits give up at once).
template <class S, int N, int T>
__device__ bool big_row(const LaunchDesc& L, const FrameDesc& F, int l, int r, int row, BigSmem<S, N>& sm, int tid,
                        int bar, RowCount& cnt) {
  constexpr int B = (int)sizeof(S), SPW = 4 / B, WR = N / SPW, NSRC = N * WR, PW = NSRC / T, NW = B == 1 ? 3 : 4;
  constexpr int TW = N / 4, NT = TW * TW, WPT = 4 / SPW, WRW = BigSmem<S, N>::WRW, ROWS = BigSmem<S, N>::ROWS;
  static_assert(NSRC % T == 0 && T % WR == 0 && T % NT == 0 && PW <= 16, "a thread's words and tile");
  const int y = row * N, lane = tid & 31, wd = tid % WR, row0 = tid / WR * PW;
  const RowInfo<S> I = row_info<S>(F, l, r, y);
  const unsigned long long* const up = I.mvf + ((ptrdiff_t)(I.base + (row - 1) * I.nbx)) * I.nref + I.r;
  const unsigned long long* const par = I.mvf + (ptrdiff_t)I.pbase * I.nref + I.r;
  const int stride = I.ref.stride, range = I.range, plane = (int)I.ref.plane_elems;
  const float lam = I.lam;
  auto parent_of = [&](int x) -> const unsigned long long* {
    const int px = x >> I.pshift;
    return px < I.pnbx ? par + (ptrdiff_t)px * I.nref : nullptr;
  };
  // This thread's words: word wd of rows row0 .. row0 + PW - 1.
  auto load_src = [&](int bx, uint32_t (&v)[PW]) {
    const uint32_t* o = reinterpret_cast<const uint32_t*>(plane_at<S>(I.src, 0, bx * N, y + row0)) + wd;
#pragma unroll
    for (int k = 0; k < PW; ++k) v[k] = RME_LD32(o + (ptrdiff_t)k * I.src.stride * B / 4);
  };
  uint32_t sw[PW];
  load_src(0, sw);
  unsigned long long uw = row > 0 ? ld_relaxed64(up) : 0ull, pw = 0ull;
  if (const unsigned long long* p = parent_of(0)) pw = ld_relaxed64(p);
  uint32_t lv = 0;
  int buf = 0;
  if (tid < 32) sm.cost[0][tid] = 0u;
  if (tid == 0) sm.lost = 0u;
  group_sync<T>(bar);
  // After a step's sums are in `mine` (lane k: candidate k's over this warp):
  // the totals, lane k candidate k's.
  auto total = [&](uint32_t mine, int nc) -> uint32_t {
    uint32_t* c = sm.cost[buf];
    const int nx = buf == 2 ? 0 : buf + 1;
    if (lane < nc) atomicAdd(&c[lane], mine);
    if (tid < 32) sm.cost[nx][tid] = 0u;
    buf = nx;
    group_sync<T>(bar);
    return c[lane];
  };
  for (int bx = 0; bx < I.nbx; ++bx) {
    const int x = bx * N;
    uint32_t* const src = sm.src[bx & 1];
#pragma unroll
    for (int k = 0; k < PW; ++k) src[(row0 + k) * WR + wd] = sw[k];
    const unsigned long long* const pp = parent_of(x);
    if (tid < 32) {
      if (row > 0) wait_published(L, up + (ptrdiff_t)bx * I.nref, I.tag, uw, sm.lost);
      if (pp) wait_published(L, pp, I.tag, pw, sm.lost);
      __syncwarp();
      if (lane == 0) {
        sm.word[0] = (uint32_t)uw;
        sm.word[1] = pp ? (uint32_t)pw : 0u;
      }
      if (bx + 1 < I.nbx) {
        if (row > 0) uw = ld_relaxed64(up + (ptrdiff_t)(bx + 1) * I.nref);
        if (const unsigned long long* p = parent_of(x + N)) pw = ld_relaxed64(p);
      }
    }
    group_sync<T>(bar);
    const uint32_t uv = sm.word[0], pv = sm.word[1];
    uint32_t m0 = 0, m1 = 0;
    if (bx > 0) {
      m0 = lv;
      if (row > 0 && uv != lv) m1 = uv;
    } else if (row > 0) {
      m0 = uv;
    }
    const int p0x = mvx_of(m0), p0y = mvy_of(m0), p1x = mvx_of(m1), p1y = mvy_of(m1);
    const int lox = -I.padm - x, hix = I.width + I.padm - N - x, loy = -I.padm - y, hiy = I.height + I.padm - N - y;
    const S* const org = plane_at<S>(I.ref, 0, x, y);
    auto inside = [&](int fx, int fy) { return fx >= lox && fx <= hix && fy >= loy && fy <= hiy; };
    auto rate = [&](int mx, int my) { return hevc_rate(lam, mx, my, p0x, p0y, p1x, p1y); };
    // Seeds [zero, mvp0, mvp1, parent], lane i the i-th: floored, clamped, a
    // seed on an earlier one's point left out.
    const uint32_t sv = lane == 1 ? m0 : lane == 2 ? m1 : lane == 3 ? pv : 0u;
    const int sx = min(max(mvx_of(sv) >> 2, lox), hix), sy = min(max(mvy_of(sv) >> 2, loy), hiy);
    bool keep = lane < (pp ? 4 : 3);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int jx = __shfl_sync(kFull, sx, j), jy = __shfl_sync(kFull, sy, j);
      keep = keep && !(j < lane && jx == sx && jy == sy);
    }
    const uint32_t kept = __ballot_sync(kFull, keep);
    // The window around the likeliest seed is staged while the seeds are
    // scored: plane words clamped to the plane (a point there is no candidate).
    int scx, scy;
    uint32_t woff;
    auto stage = [&](int cx, int cy) {
      scx = cx;
      scy = cy;
      const int e0 = I.ref.origin + (y + cy - kMargin) * stride + x + cx - kMargin;  // may lie before the plane
      const int w0 = (e0 * B) >> 2;
      woff = (uint32_t)(e0 * B) & 3u;
      const uint32_t* base = reinterpret_cast<const uint32_t*>(I.ref.base);
      const int rs = stride * B / 4, last = plane * B / 4 - 1;
      for (int i = tid; i < ROWS * WRW; i += T) {
        const int rr = i / WRW, ww = i - rr * WRW;
        sm.win[i] = RME_LD32(base + min(max(w0 + rr * rs + ww, 0), last));
      }
    };
    {
      const int gl = pp ? 3 : 1;
      stage(__shfl_sync(kFull, sx, gl), __shfl_sync(kFull, sy, gl));
    }
    uint32_t nsad = __popc(kept), nsatd = 9;
    uint32_t mine = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      if (!((kept >> s) & 1u)) continue;
      const int fx = __shfl_sync(kFull, sx, s), fy = __shfl_sync(kFull, sy, s);
      const S* rp = org + (ptrdiff_t)(fy + row0) * stride + fx + wd * SPW;
      uint32_t a[PW], acc = 0;
#pragma unroll
      for (int k = 0; k < PW; ++k) a[k] = ldw(rp + (ptrdiff_t)k * stride);
#pragma unroll
      for (int k = 0; k < PW; ++k) acc = sad_add(sw[k], a[k], acc, S());
      acc = __reduce_add_sync(kFull, sad_sum(acc, S()));
      if (lane == s) mine = acc;
    }
    uint32_t c = total(mine, 4);
    c = keep ? c + rate(sx * 4, sy * 4) : kInf;
    Pick p = warp_min(c);
    uint32_t bcost = p.cost;
    int fbx = __shfl_sync(kFull, sx, p.lane), fby = __shfl_sync(kFull, sy, p.lane);
    const int ox = fbx, oy = fby;
    // The diamond, two rounds a step: the twelve points around the best from
    // the window (lane q: point q + 1 of the order around_x has).
    for (int it = 0, rings = 0;;) {
      while (it < 2 * range) {
        if (abs(fbx - scx) > kMargin - 2 || abs(fby - scy) > kMargin - 2) {
          group_sync<T>(bar);  // the window's last readers are done
          stage(fbx, fby);
          group_sync<T>(bar);
        }
        uint32_t acc[12];
#pragma unroll
        for (int q = 0; q < 12; ++q) acc[q] = 0u;
        // The byte offset of dx = -2 in a window row, and for each dx whether
        // its samples begin in the first or the second word from there.
        const uint32_t b0 = woff + (uint32_t)((fbx - scx + kMargin - 2) * B);
        // The thread's rows follow one another: five rows of words are kept,
        // each row read once.
        const uint32_t* const wp = sm.win + (fby - scy + kMargin + row0) * WRW + (b0 >> 2) + wd;
        uint32_t w[5][NW];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < NW; ++j) w[i][j] = wp[(i - 2) * WRW + j];
#pragma unroll
        for (int k = 0; k < PW; ++k) {
#pragma unroll
          for (int j = 0; j < NW; ++j) w[(k + 4) % 5][j] = wp[(k + 2) * WRW + j];
          auto at = [&](int dx, int dy) {  // the four (two) samples at dx, dy
            const uint32_t (&v)[NW] = w[(k + dy + 2) % 5];
            const uint32_t o = (b0 & 3u) + (uint32_t)((dx + 2) * B), sh = (o & 3u) * 8u;
            const int j = (int)(o >> 2);
            const uint32_t lo = B == 1 ? (j ? v[1] : v[0]) : (j == 0 ? v[0] : j == 1 ? v[1] : v[2]);
            const uint32_t hi = B == 1 ? (j ? v[2] : v[1]) : (j == 0 ? v[1] : j == 1 ? v[2] : v[NW - 1]);
            return __funnelshift_r(lo, hi, sh);
          };
          const uint32_t s = sw[k];
          acc[0] = sad_add(s, at(1, 0), acc[0], S());
          acc[1] = sad_add(s, at(-1, 0), acc[1], S());
          acc[2] = sad_add(s, at(0, 1), acc[2], S());
          acc[3] = sad_add(s, at(0, -1), acc[3], S());
          acc[4] = sad_add(s, at(2, 0), acc[4], S());
          acc[5] = sad_add(s, at(-2, 0), acc[5], S());
          acc[6] = sad_add(s, at(1, 1), acc[6], S());
          acc[7] = sad_add(s, at(1, -1), acc[7], S());
          acc[8] = sad_add(s, at(-1, 1), acc[8], S());
          acc[9] = sad_add(s, at(-1, -1), acc[9], S());
          acc[10] = sad_add(s, at(0, 2), acc[10], S());
          acc[11] = sad_add(s, at(0, -2), acc[11], S());
        }
        mine = 0;
#pragma unroll
        for (int q = 0; q < 12; ++q) {
          const uint32_t v = __reduce_add_sync(kFull, sad_sum(acc[q], S()));
          if (lane == q) mine = v;
        }
        c = total(mine, 12);
        const int q = lane + 1, fx = fbx + around_x(q & 15), fy = fby + around_y(q & 15);
        const bool ok = lane < 12 && abs(fx - ox) <= range && abs(fy - oy) <= range && inside(fx, fy);
        c = ok ? c + rate(fx * 4, fy * 4) : kInf;
        const uint32_t there = __ballot_sync(kFull, ok) << 1;  // bit q: point q is scored
        nsad += __popc(there & 0x1eu);
        p = warp_min(lane < 4 ? c : kInf);
        if (!(p.cost < bcost)) break;
        bcost = p.cost;
        const int q1 = p.lane + 1;
        const uint32_t second = second_round(q1 - 1);
        if (++it >= 2 * range) {
          fbx += around_x(q1);
          fby += around_y(q1);
          break;
        }
        nsad += 1u + __popc(there & second);  // the fourth point is the old best
        p = warp_min((second >> q) & 1u ? c : kInf);
        if (!(p.cost < bcost)) {
          fbx += around_x(q1);
          fby += around_y(q1);
          break;
        }
        bcost = p.cost;
        fbx += around_x(p.lane + 1);
        fby += around_y(p.lane + 1);
        ++it;
      }
      if (rings >= I.rings) break;
      ++rings;
      // The 24 ring points at 4, 8, 16 around the settled point, in order.
      auto ring_x = [](int k) {
        const int d = k < 8 ? 4 : k < 16 ? 8 : 16, e = k & 7;
        return e == 0 || e == 4 || e == 6 ? d : e == 1 || e == 5 || e == 7 ? -d : 0;
      };
      auto ring_y = [](int k) {
        const int d = k < 8 ? 4 : k < 16 ? 8 : 16, e = k & 7;
        return e == 2 || e == 4 || e == 5 ? d : e == 3 || e == 6 || e == 7 ? -d : 0;
      };
      auto allowed = [&](int fx, int fy) {
        return abs(fx - ox) <= range && abs(fy - oy) <= range && inside(fx, fy);
      };
      mine = 0;
      for (int k = 0; k < 24; ++k) {
        const int fx = fbx + ring_x(k), fy = fby + ring_y(k);
        if (!allowed(fx, fy)) continue;
        const S* rp = org + (ptrdiff_t)(fy + row0) * stride + fx + wd * SPW;
        uint32_t acc = 0;
#pragma unroll
        for (int j = 0; j < PW; ++j) acc = sad_add(sw[j], ldw(rp + (ptrdiff_t)j * stride), acc, S());
        acc = __reduce_add_sync(kFull, sad_sum(acc, S()));
        if (lane == k) mine = acc;
      }
      c = total(mine, 24);
      const int fx = fbx + ring_x(min(lane, 23)), fy = fby + ring_y(min(lane, 23));
      const bool ok = lane < 24 && allowed(fx, fy);
      nsad += __popc(__ballot_sync(kFull, ok));
      p = warp_min(ok ? c + rate(fx * 4, fy * 4) : kInf);
      if (!(p.cost < bcost)) break;
      bcost = p.cost;
      fbx += ring_x(p.lane);
      fby += ring_y(p.lane);
      it = 0;
    }
    const uint32_t int_cost = bcost;
    const int imx = fbx * 4, imy = fby * 4;
    // The next block's source, on its way during the refinement.
    if (bx + 1 < I.nbx) load_src(bx + 1, sw);

    // refine_subpel: T / NT candidates at a time, a thread per 4x4 tile.
    const int tile = tid % NT, ty = tile / TW, tx = tile % TW, cg = tid / NT;
    uint32_t st[4][WPT];
#pragma unroll
    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
      for (int w = 0; w < WPT; ++w) st[rr][w] = src[(ty * 4 + rr) * WR + tx * WPT + w];
    auto satd = [&](auto count, auto vec) -> uint32_t {
      constexpr int NC = decltype(count)::value, CG = T / NT;
      uint32_t got = 0;
#pragma unroll 2
      for (int k0 = 0; k0 < NC; k0 += CG) {
        const int k = k0 + cg;
        int mx, my;
        uint32_t v = 0;
        if (k < NC && vec(k, mx, my)) {  // the same for a warp's lanes
          const S* q = plane_at<S>(I.ref, (my & 3) * 4 + (mx & 3), x + (mx >> 2) + tx * 4, y + (my >> 2) + ty * 4);
          uint32_t pr[4][WPT];
#pragma unroll
          for (int rr = 0; rr < 4; ++rr) ldwords<WPT>(q + (ptrdiff_t)rr * stride, pr[rr]);
          v = satd4x4<WPT>(st, pr);
        }
        v = __reduce_add_sync(kFull, v);
        if (lane == k) got = v;
      }
      return total(got, NC);
    };
    auto half_vec = [&](int k, int& mx, int& my) {
      const int q = k == 0 ? 4 : k <= 4 ? k - 1 : k, qy = q / 3;
      mx = imx + (q - qy * 3 - 1) * 2;
      my = imy + (qy - 1) * 2;
      return true;
    };
    uint32_t v = satd(std::integral_constant<int, 9>{}, half_vec);
    int mx, my;
    half_vec(min(lane, 8), mx, my);
    p = warp_min(lane < 9 ? v + rate(mx, my) : kInf);
    uint32_t bc = p.cost, bsatd = __shfl_sync(kFull, v, p.lane);
    int bmx, bmy;
    half_vec(p.lane, bmx, bmy);
    const int hmx = bmx, hmy = bmy, cross = I.cross;
    auto quarter_vec = [&](int k, int& ax, int& ay) {
      const int q = k < 4 ? k : k + 1, qy = q / 3, dx = q - qy * 3 - 1, dy = qy - 1;
      ax = (int)(int16_t)(hmx + dx);
      ay = (int)(int16_t)(hmy + dy);
      return !(cross != 0 && dx != 0 && dy != 0);
    };
    v = satd(std::integral_constant<int, 8>{}, quarter_vec);
    const bool ok = quarter_vec(min(lane, 7), mx, my) && lane < 8;
    nsatd += cross ? 4 : 8;
    p = warp_min(ok ? v + rate(mx, my) : kInf);
    if (p.cost < bc) {
      bc = p.cost;
      bsatd = __shfl_sync(kFull, v, p.lane);
      quarter_vec(p.lane, bmx, bmy);
    }
    lv = (uint32_t)(uint16_t)(int16_t)bmx | (uint32_t)(uint16_t)(int16_t)bmy << 16;
    if (tid == 0) {
      const ptrdiff_t t = (ptrdiff_t)(I.base + row * I.nbx + bx) * I.nref + I.r;
      st_relaxed64(I.mvf + t, (unsigned long long)I.tag << 32 | lv);
      write_result(I.out + t, bmx, bmy, I.r, bc, bsatd, imx, imy, int_cost, nsad, nsatd, 0);
      cnt.tasks += 1;
      cnt.sad += nsad;
      cnt.satd += nsatd;
    }
  }
  cnt.area = N * N;
  group_sync<T>(bar);
  return sm.lost == 0u;
}

template <class S>
constexpr size_t row_smem_bytes() {
  return std::max({(size_t)(kRowThreads / row_group(64)) * sizeof(BigSmem<S, 64>),
                   (size_t)(kRowThreads / row_group(32)) * sizeof(BigSmem<S, 32>),
                   (size_t)(kRowThreads / row_group(16)) * sizeof(SmallSmem<S, 16>),
                   (size_t)(kRowThreads / row_group(8)) * sizeof(SmallSmem<S, 8>)});
}

template <class S>
__global__ void __launch_bounds__(kRowThreads, 2) hevc_row_kernel(LaunchDesc L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t entry;
  const int tid = threadIdx.x;
  const uint32_t epoch = __ldg(L.epoch);
  bool lost = false;  // a wait of this thread's group gave up
  for (;;) {
    if (__syncthreads_or(lost)) break;  // the launch has failed (status set)
    if (tid == 0) {
      const unsigned long long idx = atomicAdd(L.head, 1ull);
      entry = idx >= (unsigned long long)L.total ? kPopDone : pop_slot(L, idx, epoch);
    }
    __syncthreads();
    const uint32_t e = entry;
    if (e == kPopDone) break;
    if (e == 0xffffffffu) continue;  // the wait ran out (status set)
    const int f = (int)(e >> 24);
    const FrameDesc& F = L.frames[f];
    int l, r, row;
    if ((sizeof(S) == 1) != (F.bd == 8) || !row_ok(F, e & 0xffffffu, l, r, row, true)) {
      if (tid == 0) atomicOr(L.status, kStatusBadTask);
      continue;
    }
    // The entry's row and the rows after it, a group each.
    const int N = F.size[l], T = row_group(N), g = tid / T, gt = tid % T, mine = row + g, bar = 1 + g;
    if (mine >= F.nby[l]) continue;
    RowCount cnt;
    if (N == 8)
      lost = !small_row<S, 8, row_group(8)>(L, F, l, r, mine, reinterpret_cast<SmallSmem<S, 8>*>(smem_raw)[g], gt, bar,
                                            cnt);
    else if (N == 16)
      lost = !small_row<S, 16, row_group(16)>(L, F, l, r, mine, reinterpret_cast<SmallSmem<S, 16>*>(smem_raw)[g], gt, bar,
                                            cnt);
    else if (N == 32)
      lost = !big_row<S, 32, row_group(32)>(L, F, l, r, mine, reinterpret_cast<BigSmem<S, 32>*>(smem_raw)[g], gt, bar,
                                            cnt);
    else
      lost = !big_row<S, 64, row_group(64)>(L, F, l, r, mine, reinterpret_cast<BigSmem<S, 64>*>(smem_raw)[g], gt, bar,
                                            cnt);
    if (gt == 0) {
      atomicAdd(&L.counters[0], (unsigned long long)cnt.tasks);
      atomicAdd(&L.counters[1], (unsigned long long)cnt.sad);
      atomicAdd(&L.counters[2], (unsigned long long)cnt.satd);
      atomicAdd(&L.counters[3], (unsigned long long)cnt.sad * cnt.area);
      atomicAdd(&L.counters[4], (unsigned long long)cnt.satd * cnt.area);
    }
  }
}

}  // namespace

int hevc_row_rows(int size) { return kRowThreads / row_group(size); }

int hevc_row_blocks_per_sm(int bytes_per_sample) {
  int n = 0;
  cudaError_t e;
  if (bytes_per_sample == 1) {
    e = cudaFuncSetAttribute(hevc_row_kernel<uint8_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)row_smem_bytes<uint8_t>());
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, hevc_row_kernel<uint8_t>, kRowThreads,
                                                        row_smem_bytes<uint8_t>());
  } else {
    e = cudaFuncSetAttribute(hevc_row_kernel<uint16_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)row_smem_bytes<uint16_t>());
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, hevc_row_kernel<uint16_t>, kRowThreads,
                                                        row_smem_bytes<uint16_t>());
  }
  return e == cudaSuccess && n > 0 ? n : 1;
}

cudaError_t launch_hevc_rows(const LaunchDesc& L, int bytes_per_sample, int grid, cudaStream_t s) {
  if (bytes_per_sample == 1)
    hevc_row_kernel<uint8_t><<<grid, kRowThreads, row_smem_bytes<uint8_t>(), s>>>(L);
  else
    hevc_row_kernel<uint16_t><<<grid, kRowThreads, row_smem_bytes<uint16_t>(), s>>>(L);
  return cudaGetLastError();
}

}  // namespace rme
