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
//     parent words only, loaded a block ahead; its left vector is at hand;
//   - many threads a block and few steps: an 8x8 block has 128 threads, a
//     16x16 or 32x32 block 256, a 64x64 block 512, so that a step is a
//     handful of loads a thread, one shuffle sum and one barrier;
//   - speculation instead of dependence for 8x8 and 16x16 blocks: every
//     seed's SAD and those of the twelve points two diamond rounds around it
//     can reach are scored together;
//   - the next block's source is on its way while a block is searched.
// Which candidates are scored, in which order they win and how many are
// counted is the reference's walk (h265_me.rs:3749-3922), as hevc_task runs
// it with one warp.
//
// A CTA is 512 threads: one row of 64x64 blocks, two of 32x32 or 16x16, four
// of 8x8. Rows are taken in the order the host pushed them, each after the
// rows it reads, so the owner of a row that is waited for is always running.
#include <algorithm>

#include "rme_search_impl.cuh"

namespace rme {
namespace {

constexpr int kRowThreads = 512;

// Threads that share a block of N x N samples.
constexpr int row_group(int n) { return n == 64 ? 512 : n == 8 ? 128 : 256; }

constexpr int kSeeds = 4;          // zero, the AMVP pair, the parent
constexpr int kAround = 16;        // slots per centre: the centre, its 12 points, three empty
constexpr int kSlotCosts = kSeeds * kAround;

template <class S, int N>
struct SmallSmem {
  uint32_t src[2][N * N * sizeof(S) / 4];
  uint32_t cost[2][kSlotCosts];
};

// The points two rounds of the small diamond can reach, in an order in
// which, whichever way the first round moves, the second round's new points
// come in the reference's order ((1,0), (-1,0), (0,1), (0,-1) around the new
// best): the centre, the first round, (2,0), (-2,0), (1,1), (1,-1), (-1,1),
// (-1,-1), (0,2), (0,-2). Offsets + 2 as hex digits, slot 0 the lowest.
constexpr unsigned long long kAroundX = 0x2211330422132ull, kAroundY = 0x0413132213222ull;
__device__ __forceinline__ int around_x(int q) { return (int)((kAroundX >> (4 * q)) & 15u) - 2; }
__device__ __forceinline__ int around_y(int q) { return (int)((kAroundY >> (4 * q)) & 15u) - 2; }
// The second round's new points after the first moved in direction j.
__device__ __forceinline__ uint32_t second_round(int j) {
  return j == 0 ? 0x1a0u : j == 1 ? 0x640u : j == 2 ? 0xa80u : 0x1500u;
}

// What a row's blocks share, read once.
template <class S>
struct RowInfo {
  const DevPlanes src, ref;
  unsigned long long* mvf;
  rme_result* out;
  const uint32_t tag;
  const int nref, r, nbx, base;          // this level
  const int pnbx, pbase, psize;          // the parents' level (psize 0: none over this row)
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
                    psize ? F.nbx[l - 1] : 0, psize ? F.base[l - 1] + (y / psize) * F.nbx[l - 1] : 0, psize,
                    F.width,  F.height,  F.pad - 4,
                    F.search_range, F.search_rings, F.quarter_cross, F.lam};
}

// The totals of a thread's rows (thread 0 of each group counts).
struct RowCount {
  unsigned long long tasks = 0, sad = 0, satd = 0, sad_samples = 0, satd_samples = 0;
};

// A row of 8x8 or 16x16 blocks by T threads.
template <class S, int N, int T>
__device__ void small_row(const LaunchDesc& L, const FrameDesc& F, int l, int r, int row, SmallSmem<S, N>& sm, int tid,
                          int bar, RowCount& cnt) {
  constexpr int SPW = 4 / (int)sizeof(S), WR = N / SPW, NSRC = N * WR, TW = N / 4, NT = TW * TW, WPT = 4 / SPW;
  const int y = row * N, lane = tid & 31;
  const RowInfo<S> I = row_info<S>(F, l, r, y);
  const unsigned long long* const up = I.mvf + ((ptrdiff_t)(I.base + (row - 1) * I.nbx)) * I.nref + I.r;
  const unsigned long long* const par = I.mvf + (ptrdiff_t)I.pbase * I.nref + I.r;
  const int stride = I.ref.stride;
  const float lam = I.lam;
  // The word of the parent of the block at x, or null where there is none.
  auto parent_of = [&](int x) -> const unsigned long long* {
    const int px = I.psize ? x / I.psize : 0;
    return I.psize && px < I.pnbx ? par + (ptrdiff_t)px * I.nref : nullptr;
  };
  auto load_src = [&](int bx) -> uint32_t {  // word tid of the block (aligned: N and the pad are whole words)
    return RME_LD32(reinterpret_cast<const uint32_t*>(plane_at<S>(I.src, 0, bx * N, y + tid / WR)) + tid % WR);
  };
  if (tid < NSRC) sm.src[0][tid] = load_src(0);
  unsigned long long uw = row > 0 ? ld_relaxed64(up) : 0ull, pw = 0ull;
  if (const unsigned long long* p = parent_of(0)) pw = ld_relaxed64(p);
  uint32_t lv = 0;
  int buf = 0;  // the cost buffer of the next step
  const int slot = tid / (T / kSlotCosts), aq = slot & (kAround - 1), ax = around_x(aq), ay = around_y(aq);
  const int slot16 = tid / (T / kAround), bx16 = around_x(slot16), by16 = around_y(slot16);
  group_sync<T>(bar);
  for (int bx = 0; bx < I.nbx; ++bx) {
    const int x = bx * N;
    const uint32_t* const src = sm.src[bx & 1];
    if (row > 0) uw = wait_word(L, up + (ptrdiff_t)bx * I.nref, I.tag, uw);
    const unsigned long long* const pp = parent_of(x);
    if (pp) pw = wait_word(L, pp, I.tag, pw);
    __syncwarp();
    const uint32_t uv = (uint32_t)uw, pv = pp ? (uint32_t)pw : 0u;
    // The next block's words and source, on their way during the search.
    uint32_t nsrc = 0;
    if (bx + 1 < I.nbx) {
      if (row > 0) uw = ld_relaxed64(up + (ptrdiff_t)(bx + 1) * I.nref);
      if (const unsigned long long* p = parent_of(x + N)) pw = ld_relaxed64(p);
      if (tid < NSRC) nsrc = load_src(bx + 1);
    }
    // The AMVP pair (left, upper when another; zero-filled) and the seeds
    // [zero, mvp0, mvp1, parent], floored to whole samples and clamped.
    int p0x = 0, p0y = 0, p1x = 0, p1y = 0;
    if (bx > 0) {
      p0x = mvx_of(lv);
      p0y = mvy_of(lv);
      if (row > 0 && uv != lv) {
        p1x = mvx_of(uv);
        p1y = mvy_of(uv);
      }
    } else if (row > 0) {
      p0x = mvx_of(uv);
      p0y = mvy_of(uv);
    }
    const int lox = -I.padm - x, hix = I.width + I.padm - N - x, loy = -I.padm - y, hiy = I.height + I.padm - N - y;
    int kx[kSeeds], ky[kSeeds];
    uint32_t kept = 0;
    {
      const int sx[kSeeds] = {0, p0x, p1x, mvx_of(pv)}, sy[kSeeds] = {0, p0y, p1y, mvy_of(pv)};
#pragma unroll
      for (int i = 0; i < kSeeds; ++i) {
        kx[i] = min(max(sx[i] >> 2, lox), hix);
        ky[i] = min(max(sy[i] >> 2, loy), hiy);
        bool dup = i == 3 && !pp;
#pragma unroll
        for (int j = 0; j < i; ++j) dup |= kx[j] == kx[i] && ky[j] == ky[i];
        kept |= (dup ? 0u : 1u) << i;
      }
    }
    auto seed_x = [&](int i) { return i == 0 ? kx[0] : i == 1 ? kx[1] : i == 2 ? kx[2] : kx[3]; };
    auto seed_y = [&](int i) { return i == 0 ? ky[0] : i == 1 ? ky[1] : i == 2 ? ky[2] : ky[3]; };
    const S* const org = plane_at<S>(I.ref, 0, x, y);
    uint32_t nsad = __popc(kept), nsatd = 9;
    // A candidate's SAD over LPC lanes (rows sub, sub + LPC, ...) and its
    // cost into its slot, then the barrier: every cost in `costs`.
    const uint32_t* costs = nullptr;
    auto score = [&](auto lanes, int at, bool ok, int fx, int fy) {
      constexpr int LPC = decltype(lanes)::value, RPL = N / LPC;
      const int sub = tid % LPC;
      uint32_t acc = 0;
      if (ok) {
        const S* rp = org + (ptrdiff_t)(fy + sub) * stride + fx;
        if constexpr (RPL * WR <= 16) {  // every load before any use
          uint32_t a[RPL][WR];
#pragma unroll
          for (int k = 0; k < RPL; ++k) ldwords<WR>(rp + (ptrdiff_t)k * LPC * stride, a[k]);
#pragma unroll
          for (int k = 0; k < RPL; ++k)
#pragma unroll
            for (int c = 0; c < WR; ++c) acc = vsad(src[(sub + k * LPC) * WR + c], a[k][c], acc, S());
        } else {
#pragma unroll 2
          for (int k = 0; k < RPL; ++k) {
            uint32_t a[WR];
            ldwords<WR>(rp + (ptrdiff_t)k * LPC * stride, a);
#pragma unroll
            for (int c = 0; c < WR; ++c) acc = vsad(src[(sub + k * LPC) * WR + c], a[c], acc, S());
          }
        }
      }
#pragma unroll
      for (int o = LPC >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(kFull, acc, o);
      uint32_t* c = sm.cost[buf];
      buf ^= 1;
      if (sub == 0) c[at] = ok ? acc + hevc_rate(lam, fx * 4, fy * 4, p0x, p0y, p1x, p1y) : kInf;
      group_sync<T>(bar);
      costs = c;
    };
    // Every seed with the points two rounds around it.
    const int range = I.range;
    {
      const int i = slot / kAround, sx = seed_x(i), sy = seed_y(i), fx = sx + ax, fy = sy + ay;
      const bool ok = ((kept >> i) & 1u) && aq < 13 &&
                      (aq == 0 || (abs(ax) <= range && abs(ay) <= range && fx >= lox && fx <= hix && fy >= loy && fy <= hiy));
      score(std::integral_constant<int, T / kSlotCosts>{}, slot, ok, fx, fy);
    }
    int ox, oy, mxw, myw;  // the best seed; the best whole-sample point
    uint32_t bcost, c;
    {
      const Pick p = warp_min(lane < kSeeds ? costs[lane * kAround] : kInf);
      bcost = p.cost;
      mxw = ox = seed_x(p.lane);
      myw = oy = seed_y(p.lane);
      c = lane < kAround ? costs[p.lane * kAround + lane] : kInf;
    }
    int it = 0, rings = 0;
    for (bool known = true;;) {
      // The diamond, two rounds a step, from the costs `c` of the points
      // around the best (lane q: point q).
      while (it < 2 * range) {
        if (!known) {
          const int fx = mxw + bx16, fy = myw + by16;
          const bool ok = slot16 > 0 && slot16 < 13 && abs(fx - ox) <= range && abs(fy - oy) <= range && fx >= lox &&
                          fx <= hix && fy >= loy && fy <= hiy;
          score(std::integral_constant<int, T / kAround>{}, slot16, ok, fx, fy);
          c = lane < kAround ? costs[lane] : kInf;
        }
        known = false;
        const uint32_t in1 = lane >= 1 && lane <= 4 ? c : kInf;
        nsad += __popc(__ballot_sync(kFull, in1 != kInf));
        Pick p = warp_min(in1);
        if (!(p.cost < bcost)) break;
        const int j = p.lane - 1;
        bcost = p.cost;
        mxw += around_x(p.lane);
        myw += around_y(p.lane);
        if (++it >= 2 * range) break;
        const int cx = mxw - around_x(p.lane), cy = myw - around_y(p.lane);
        const uint32_t in2 = (second_round(j) >> lane) & 1u ? c : kInf;
        nsad += 1u + __popc(__ballot_sync(kFull, in2 != kInf));  // the fourth point is the old best
        p = warp_min(in2);
        if (!(p.cost < bcost)) break;
        bcost = p.cost;
        mxw = cx + around_x(p.lane);
        myw = cy + around_y(p.lane);
        ++it;
      }
      if (rings >= I.rings) break;
      ++rings;
      // The 24 ring points at 4, 8, 16 around the settled point, in order;
      // a move restarts the diamond.
      const int k = tid / (T / 32), rr = k < 8 ? 4 : k < 16 ? 8 : 16;
      auto ring_x = [](int q, int d) { return q == 0 || q == 4 || q == 6 ? d : q == 1 || q == 5 || q == 7 ? -d : 0; };
      auto ring_y = [](int q, int d) { return q == 2 || q == 4 || q == 5 ? d : q == 3 || q == 6 || q == 7 ? -d : 0; };
      const int fx = mxw + ring_x(k & 7, rr), fy = myw + ring_y(k & 7, rr);
      const bool ok = k < 24 && abs(fx - ox) <= range && abs(fy - oy) <= range && fx >= lox && fx <= hix && fy >= loy &&
                      fy <= hiy;
      score(std::integral_constant<int, T / 32>{}, k, ok, fx, fy);
      c = lane < 24 ? costs[lane] : kInf;
      nsad += __popc(__ballot_sync(kFull, c != kInf));
      const Pick p = warp_min(c);
      if (!(p.cost < bcost)) break;
      bcost = p.cost;
      const int pr = p.lane < 8 ? 4 : p.lane < 16 ? 8 : 16;
      mxw += ring_x(p.lane & 7, pr);
      myw += ring_y(p.lane & 7, pr);
      it = 0;
    }
    const uint32_t int_cost = bcost;
    const int imx = mxw * 4, imy = myw * 4;

    // refine_subpel: the start and the half ring in one step, then the
    // quarter ring around the winner; a thread per 4x4 tile, NT threads a
    // candidate.
    auto satd = [&](int nc, auto vec) {
      const int k = tid / NT, tile = tid % NT, ty = tile / TW, tx = tile % TW;
      int mx, my;
      uint32_t v = 0;
      if (k < nc && vec(k, mx, my)) {
        const S* q = plane_at<S>(I.ref, (my & 3) * 4 + (mx & 3), x + (mx >> 2) + tx * 4, y + (my >> 2) + ty * 4);
        uint32_t pw4[4][WPT];
#pragma unroll
        for (int rr = 0; rr < 4; ++rr) ldwords<WPT>(q + (ptrdiff_t)rr * stride, pw4[rr]);
        uint32_t sw[4][WPT];
#pragma unroll
        for (int rr = 0; rr < 4; ++rr)
#pragma unroll
          for (int w = 0; w < WPT; ++w) sw[rr][w] = src[(ty * 4 + rr) * WR + tx * WPT + w];
        v = satd4x4<WPT>(sw, pw4);
      }
#pragma unroll
      for (int o = NT >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
      uint32_t* cb = sm.cost[buf];
      buf ^= 1;
      if (tile == 0 && k < nc) cb[k] = v;
      group_sync<T>(bar);
      costs = cb;
    };
    auto half_vec = [&](int k, int& mx, int& my) {
      const int q = k == 0 ? 4 : k <= 4 ? k - 1 : k;
      mx = imx + (q % 3 - 1) * 2;
      my = imy + (q / 3 - 1) * 2;
      return true;
    };
    satd(9, half_vec);
    int bmx, bmy;
    uint32_t bc, bsatd;
    {
      int mx = imx, my = imy;
      uint32_t v = 0, cost = kInf;
      if (lane < 9) {
        half_vec(lane, mx, my);
        v = costs[lane];
        cost = v + hevc_rate(lam, mx, my, p0x, p0y, p1x, p1y);
      }
      const Pick p = warp_min(cost);
      bc = p.cost;
      bsatd = __shfl_sync(kFull, v, p.lane);
      bmx = __shfl_sync(kFull, mx, p.lane);
      bmy = __shfl_sync(kFull, my, p.lane);
    }
    const int hmx = bmx, hmy = bmy, cross = I.cross;
    auto quarter_vec = [&](int k, int& mx, int& my) {
      const int q = k < 4 ? k : k + 1, dx = q % 3 - 1, dy = q / 3 - 1;
      mx = (int)(int16_t)(hmx + dx);
      my = (int)(int16_t)(hmy + dy);
      return !(cross != 0 && dx != 0 && dy != 0);
    };
    if (tid < NSRC) sm.src[(bx + 1) & 1][tid] = nsrc;
    satd(8, quarter_vec);
    {
      int mx = 0, my = 0;
      uint32_t v = 0, cost = kInf;
      bool ok = false;
      if (lane < 8) ok = quarter_vec(lane, mx, my);
      if (ok) {
        v = costs[lane];
        cost = v + hevc_rate(lam, mx, my, p0x, p0y, p1x, p1y);
      }
      nsatd += __popc(__ballot_sync(kFull, ok));
      const Pick p = warp_min(cost);
      if (p.cost < bc) {
        bc = p.cost;
        bsatd = __shfl_sync(kFull, v, p.lane);
        bmx = __shfl_sync(kFull, mx, p.lane);
        bmy = __shfl_sync(kFull, my, p.lane);
      }
    }
    lv = (uint32_t)(uint16_t)(int16_t)bmx | (uint32_t)(uint16_t)(int16_t)bmy << 16;
    if (tid == 0) {
      const ptrdiff_t t = (ptrdiff_t)(I.base + row * I.nbx + bx) * I.nref + I.r;
      st_relaxed64(I.mvf + t, (unsigned long long)I.tag << 32 | lv);
      write_result(I.out + t, bmx, bmy, I.r, bc, bsatd, imx, imy, int_cost, nsad, nsatd, 0);
      cnt.tasks += 1;
      cnt.sad += nsad;
      cnt.satd += nsatd;
      cnt.sad_samples += (unsigned long long)nsad * (N * N);
      cnt.satd_samples += (unsigned long long)nsatd * (N * N);
    }
  }
  group_sync<T>(bar);  // the last block's costs and source are read: the buffers may be reused
}

// A row of 32x32 or 64x64 blocks by T threads: the group search (GroupSmem,
// its window behind it), its counts in the GroupSmem.
template <class S, int N, int T>
__device__ void big_row(const LaunchDesc& L, const FrameDesc& F, int f, int l, int r, int row, GroupSmem<S>& gs,
                        int tid, int bar) {
  const int nbx = F.nbx[l], t0 = (F.base[l] + row * nbx) * F.nref + r;
  for (int bx = 0; bx < nbx; ++bx) hevc_group_task<S, N, true, T>(L, F, f, t0 + bx * F.nref, gs, tid, bar);
  group_sync<T>(bar);
}

template <class S, int N>
constexpr size_t big_bytes() {
  return (sizeof(GroupSmem<S>) + (size_t)WinGeo<S, N>::ROWS * WinGeo<S, N>::WRW * 4 + 15) / 16 * 16;
}
template <class S>
constexpr size_t row_smem_bytes() {
  return std::max({big_bytes<S, 64>(), 2 * big_bytes<S, 32>(), 2 * sizeof(SmallSmem<S, 16>), 4 * sizeof(SmallSmem<S, 8>)});
}

template <class S>
__global__ void __launch_bounds__(kRowThreads, 2) hevc_row_kernel(LaunchDesc L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t entry;
  const int tid = threadIdx.x;
  const uint32_t epoch = __ldg(L.epoch);
  RowCount cnt;
  for (;;) {
    __syncthreads();
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
    if ((sizeof(S) == 1) != (F.bd == 8) || !row_ok(F, e & 0xffffffu, l, r, row)) {
      if (tid == 0) atomicOr(L.status, kStatusBadTask);
      continue;
    }
    // The entry's row and the rows after it, a group each.
    const int N = F.size[l], T = row_group(N), g = tid / T, gt = tid % T, mine = row + g, bar = 1 + g;
    if (mine >= F.nby[l]) continue;
    if (N == 8) {
      small_row<S, 8, row_group(8)>(L, F, l, r, mine, reinterpret_cast<SmallSmem<S, 8>*>(smem_raw)[g], gt, bar, cnt);
    } else if (N == 16) {
      small_row<S, 16, row_group(16)>(L, F, l, r, mine, reinterpret_cast<SmallSmem<S, 16>*>(smem_raw)[g], gt, bar, cnt);
    } else {
      GroupSmem<S>& gs = *reinterpret_cast<GroupSmem<S>*>(smem_raw + (N == 32 ? g * big_bytes<S, 32>() : 0));
      if (gt < 6) gs.cnt[gt] = 0;
      if (N == 32) big_row<S, 32, row_group(32)>(L, F, f, l, r, mine, gs, gt, bar);
      else big_row<S, 64, row_group(64)>(L, F, f, l, r, mine, gs, gt, bar);
      if (gt < 5) atomicAdd(&L.counters[gt], gs.cnt[gt]);
    }
  }
  if (cnt.tasks != 0) {
    atomicAdd(&L.counters[0], cnt.tasks);
    atomicAdd(&L.counters[1], cnt.sad);
    atomicAdd(&L.counters[2], cnt.satd);
    atomicAdd(&L.counters[3], cnt.sad_samples);
    atomicAdd(&L.counters[4], cnt.satd_samples);
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
