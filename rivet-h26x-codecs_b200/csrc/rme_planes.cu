// Per-reference plane builds on the device.
//
// A reference picture is searched by every block of every picture that
// predicts from it, so — as the reference's encoders do on the CPU — its
// sub-sample planes are computed once, when it is uploaded:
//   H.264  build_hpel / hpel_planes (encode/h264_hpel.rs:95-189): the
//          horizontal (b), vertical (h) and centre (j) half-sample planes.
//   HEVC   HalfPlanes::new (encode/h265_search.rs:79-170): the fifteen
//          fractional phases, each the exact uni-predicted sample of
//          8.5.3.3.3.1 (8-tap, shift1 = Min(4, BitDepth-8), second pass
//          >> 6, (x + offset) >> (14 - BitDepth) and clip).
// The reference's planes hold a copy of the integer sample where a filter
// window would leave the padded plane, and HalfPlanes stops REACH samples
// outside the picture; neither region is ever read by a search whose
// window rules hold (search_bounds, clamp_pos), so here every position is
// computed over the edge-replicated plane, which gives the reference's
// value wherever the reference computes one.
#include <cuda_runtime.h>

#include <algorithm>

#include "rme_internal.h"

namespace rme {
namespace {

// The padded plane of a picture: position (x, y) the sample of its clamped
// position. A thread writes one aligned 16-byte chunk of a row: from inside
// the picture as four words at any byte address, across its sides sample by
// sample. In place (src is the plane's own visible picture) only the border
// is written, and it reads only the visible picture. A thread a sample took
// 7.9 us for the border of a 1080p picture; this way the whole plane from a
// packed picture takes 4.1 us, the border alone 3.8.
template <class S>
__global__ void __launch_bounds__(256) pad_plane_kernel(const S* __restrict__ src, int w, int h, int sstride,
                                                        S* __restrict__ dst, int dstride, int prow, int pad,
                                                        bool in_place) {
  constexpr int N = 16 / (int)sizeof(S);  // samples of a chunk
  const int x = (blockIdx.x * 32 + threadIdx.x) * N, y = blockIdx.y * 8 + threadIdx.y;
  if (x >= dstride || y >= prow) return;
  const S* row = src + (int64_t)min(max(y - pad, 0), h - 1) * sstride;
  const int sx = x - pad;  // the source column of the chunk's first sample
  const bool own = in_place && y >= pad && y < pad + h;
  S* d = dst + (int64_t)y * dstride + x;
  if (sx >= 0 && sx + N <= w) {
    if (own) return;
    const uintptr_t u = reinterpret_cast<uintptr_t>(row + sx);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(u & ~uintptr_t(3));
    const uint32_t sh = (uint32_t)(u & 3) * 8u;
    uint32_t v[5];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = q[k];
    v[4] = sh ? q[4] : 0u;  // holds samples of the chunk only when the address is odd
    uint4 o;
    o.x = __funnelshift_r(v[0], v[1], sh);
    o.y = __funnelshift_r(v[1], v[2], sh);
    o.z = __funnelshift_r(v[2], v[3], sh);
    o.w = __funnelshift_r(v[3], v[4], sh);
    *reinterpret_cast<uint4*>(d) = o;
    return;
  }
#pragma unroll 4
  for (int k = 0; k < N; ++k) {
    const int c = sx + k;
    if (!(own && c >= 0 && c < w)) d[k] = row[min(max(c, 0), w - 1)];
  }
}

__device__ __forceinline__ int tap6(int a, int b, int c, int d, int e, int f) {
  return a + f - 5 * (b + e) + 20 * (c + d);
}

// b, h, j of every padded position (x, y): reads of G clamped to the padded
// plane, i.e. of the edge-replicated picture.
template <class S>
__global__ void h264_hpel_kernel(const S* __restrict__ g, S* __restrict__ pb, S* __restrict__ ph, S* __restrict__ pj,
                                 int stride, int prow, int pcol, int maxv) {
  constexpr int TX = 32, TY = 8;
  __shared__ int tile[TY + 5][TX + 5];  // G over rows y-2..y+TY+2, cols x-2..x+TX+2
  __shared__ int vin[TY][TX + 5];       // vertical six-tap, unclipped
  int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
  int tid = threadIdx.y * TX + threadIdx.x;
  for (int i = tid; i < (TY + 5) * (TX + 5); i += TX * TY) {
    int ty = i / (TX + 5), tx = i % (TX + 5);
    int gx = min(max(x0 + tx - 2, 0), pcol - 1), gy = min(max(y0 + ty - 2, 0), prow - 1);
    tile[ty][tx] = g[(int64_t)gy * stride + gx];
  }
  __syncthreads();
  for (int i = tid; i < TY * (TX + 5); i += TX * TY) {
    int ty = i / (TX + 5), tx = i % (TX + 5);
    vin[ty][tx] = tap6(tile[ty][tx], tile[ty + 1][tx], tile[ty + 2][tx], tile[ty + 3][tx], tile[ty + 4][tx],
                       tile[ty + 5][tx]);
  }
  __syncthreads();
  int tx = threadIdx.x, ty = threadIdx.y, x = x0 + tx, y = y0 + ty;
  if (x >= pcol || y >= prow) return;
  const int* r = &tile[ty + 2][tx];
  int b = tap6(r[0], r[1], r[2], r[3], r[4], r[5]);
  int v = vin[ty][tx + 2];
  const int* q = &vin[ty][tx];
  int j = tap6(q[0], q[1], q[2], q[3], q[4], q[5]);
  int64_t o = (int64_t)y * stride + x;
  pb[o] = (S)min(max((b + 16) >> 5, 0), maxv);
  ph[o] = (S)min(max((v + 16) >> 5, 0), maxv);
  pj[o] = (S)min(max((j + 512) >> 10, 0), maxv);
}

// The luma taps of a quarter fraction as two words of four signed bytes, and
// as four pairs in the low halves' bytes of words (dp4a and dp2a operands):
// {-1, 4, -10, 58, 17, -5, 1, 0}, {-1, 4, -11, 40, 40, -11, 4, -1},
// {0, 1, -5, 17, 58, -10, 4, -1}.
constexpr uint32_t byte4(int a, int b, int c, int d) {
  return (uint32_t)(uint8_t)a | (uint32_t)(uint8_t)b << 8 | (uint32_t)(uint8_t)c << 16 | (uint32_t)(uint8_t)d << 24;
}
template <int F>
struct Taps;
template <>
struct Taps<1> {
  static constexpr uint32_t lo = byte4(-1, 4, -10, 58), hi = byte4(17, -5, 1, 0);
};
template <>
struct Taps<2> {
  static constexpr uint32_t lo = byte4(-1, 4, -11, 40), hi = byte4(40, -11, 4, -1);
};
template <>
struct Taps<3> {
  static constexpr uint32_t lo = byte4(0, 1, -5, 17), hi = byte4(58, -10, 4, -1);
};
// Four unsigned bytes by four signed ones, added to c.
__device__ __forceinline__ int dot4(uint32_t a, uint32_t b, int c) {
  int r;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
// The eight taps (signed bytes in `lo`, `hi`) on four words of two signed
// 16-bit values, added to c.
__device__ __forceinline__ int dot8(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3, uint32_t lo, uint32_t hi, int c) {
  asm("dp2a.lo.s32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(p0), "r"(lo));
  asm("dp2a.hi.s32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(p1), "r"(lo));
  asm("dp2a.lo.s32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(p2), "r"(hi));
  asm("dp2a.hi.s32.s32 %0, %1, %2, %0;" : "+r"(c) : "r"(p3), "r"(hi));
  return c;
}

// Four output samples, each v[i] clamped to 0..maxv, as words.
__device__ __forceinline__ void put4(uint8_t* q, const int (&v)[4], uint32_t) {
  uint32_t r;
  asm("{ .reg .b32 t; cvt.pack.sat.u8.s32.b32 t, %4, %3, 0; cvt.pack.sat.u8.s32.b32 %0, %2, %1, t; }"
      : "=r"(r)
      : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
  *reinterpret_cast<uint32_t*>(q) = r;
}
__device__ __forceinline__ void put4(uint16_t* q, const int (&v)[4], uint32_t maxv2) {
  uint2 r;
  asm("cvt.pack.sat.u16.s32 %0, %1, %2;" : "=r"(r.x) : "r"(v[1]), "r"(v[0]));
  asm("cvt.pack.sat.u16.s32 %0, %1, %2;" : "=r"(r.y) : "r"(v[3]), "r"(v[2]));
  asm("min.u16x2 %0, %0, %1;" : "+r"(r.x) : "r"(maxv2));
  asm("min.u16x2 %0, %0, %1;" : "+r"(r.y) : "r"(maxv2));
  *reinterpret_cast<uint2*>(q) = r;
}

// One row's samples x - 4 .. x + 7 (x a multiple of 4) as words. Columns
// outside the padded plane take the border's value, which the outermost
// words hold (the border is a replicated edge wider than a word): a word
// outside is read at the first or the last whole word.
template <class S>
struct RowWords {
  uint32_t w[3 * sizeof(S)];
};
template <class S>
__device__ __forceinline__ RowWords<S> load_row(const S* row, const int (&col)[3]) {
  RowWords<S> r;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if constexpr (sizeof(S) == 1) {
      r.w[i] = *reinterpret_cast<const uint32_t*>(row + col[i]);
    } else {
      const uint2 v = *reinterpret_cast<const uint2*>(row + col[i]);
      r.w[2 * i] = v.x;
      r.w[2 * i + 1] = v.y;
    }
  }
  return r;
}

// The row's horizontal pass of fraction FX at x .. x + 3 (FX 0: the samples),
// 16-bit values in order.
template <int FX>
__device__ __forceinline__ void horizontal(const RowWords<uint8_t>& r, int, int (&h)[4]) {
  if constexpr (FX == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = (int)((r.w[1] >> (8 * i)) & 0xffu);
  } else {
    // Bytes x + i - 3 .. x + i and x + i + 1 .. x + i + 4.
    const uint32_t a[8] = {__funnelshift_r(r.w[0], r.w[1], 8),  __funnelshift_r(r.w[0], r.w[1], 16),
                           __funnelshift_r(r.w[0], r.w[1], 24), r.w[1],
                           __funnelshift_r(r.w[1], r.w[2], 8),  __funnelshift_r(r.w[1], r.w[2], 16),
                           __funnelshift_r(r.w[1], r.w[2], 24), r.w[2]};
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = dot4(a[i + 4], Taps<FX>::hi, dot4(a[i], Taps<FX>::lo, 0));
  }
}
template <int FX>
__device__ __forceinline__ void horizontal(const RowWords<uint16_t>& r, int shift1, int (&h)[4]) {
  if constexpr (FX == 0) {
    h[0] = (int)(r.w[2] & 0xffffu);
    h[1] = (int)(r.w[2] >> 16);
    h[2] = (int)(r.w[3] & 0xffffu);
    h[3] = (int)(r.w[3] >> 16);
  } else {
    uint32_t o[5];  // samples x - 3 + 2k, x - 2 + 2k
#pragma unroll
    for (int k = 0; k < 5; ++k) o[k] = __funnelshift_r(r.w[k], r.w[k + 1], 16);
    constexpr uint32_t lo = Taps<FX>::lo, hi = Taps<FX>::hi;
    h[0] = dot8(o[0], o[1], o[2], o[3], lo, hi, 0) >> shift1;
    h[1] = dot8(r.w[1], r.w[2], r.w[3], r.w[4], lo, hi, 0) >> shift1;
    h[2] = dot8(o[1], o[2], o[3], o[4], lo, hi, 0) >> shift1;
    h[3] = dot8(r.w[2], r.w[3], r.w[4], r.w[5], lo, hi, 0) >> shift1;
  }
}

// One warp's share of a tile: the phases of horizontal fraction FX over 128
// columns and `rows` rows. A lane has four columns: it runs down the
// rows, keeping the horizontal pass of the last eight as words of two rows
// (p[i][k]: rows k and k + 1 of the window), from which each vertical pass
// is four dot products of pairs. The rounding of 8.5.3.3.3.1 (>> shift1 or
// >> 6, then + round and >> shift3) is one addition and one shift: nested
// floors are the floor of the quotient.
constexpr int kPhaseTX = 128;
template <class S, int FX>
__device__ __forceinline__ void phase_columns(const S* g, S* planes, int64_t plane_elems, int stride, int prow, int pcol,
                                              int bd, int x, int y0, int rows) {
  const int shift1 = min(bd, 12) - 8, shift3 = 14 - bd, round3 = 1 << (shift3 - 1);
  const uint32_t maxv2 = ((1u << bd) - 1u) * 0x10001u;
  const int vshift = FX == 0 ? shift1 + shift3 : 6 + shift3, vround = round3 << (FX == 0 ? shift1 : 6);
  uint32_t p[4][7];
  int last[4];
  const int edge = pcol / 4 * 4 - 4, col[3] = {max(x - 4, 0), min(x, edge), min(x + 4, edge)};
  auto row_of = [&](int y) { return g + (int64_t)min(max(y, 0), prow - 1) * stride; };
  horizontal<FX>(load_row<S>(row_of(y0 - 3), col), shift1, last);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    int h[4];
    horizontal<FX>(load_row<S>(row_of(y0 - 2 + k), col), shift1, h);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[i][k] = __byte_perm((uint32_t)last[i], (uint32_t)h[i], 0x5410);
      last[i] = h[i];
    }
  }
  RowWords<S> next = load_row<S>(row_of(y0 + 4), col);
  S* out = planes + (int64_t)y0 * stride + x;
#pragma unroll (sizeof(S) == 1 ? 2 : 1)
  for (int r = 0; r < rows; ++r) {
    int h[4];
    horizontal<FX>(next, shift1, h);
    next = load_row<S>(row_of(y0 + r + 5), col);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      p[i][6] = __byte_perm((uint32_t)last[i], (uint32_t)h[i], 0x5410);
      last[i] = h[i];
    }
    int v[4];
    if (FX != 0) {  // the row itself: window row 3
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = ((int)(int16_t)(p[i][3] & 0xffffu) + round3) >> shift3;
      put4(out + (int64_t)FX * plane_elems, v, maxv2);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = dot8(p[i][0], p[i][2], p[i][4], p[i][6], Taps<1>::lo, Taps<1>::hi, vround) >> vshift;
    put4(out + (int64_t)(4 + FX) * plane_elems, v, maxv2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = dot8(p[i][0], p[i][2], p[i][4], p[i][6], Taps<2>::lo, Taps<2>::hi, vround) >> vshift;
    put4(out + (int64_t)(8 + FX) * plane_elems, v, maxv2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      v[i] = dot8(p[i][0], p[i][2], p[i][4], p[i][6], Taps<3>::lo, Taps<3>::hi, vround) >> vshift;
    put4(out + (int64_t)(12 + FX) * plane_elems, v, maxv2);
    out += stride;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 6; ++k) p[i][k] = p[i][k + 1];
  }
}

// The fifteen phases of every padded position: a CTA of two warps, two of the
// horizontal fractions (grid z the other two), over a tile of 128 x
// `strip` positions. At most 64 registers a thread: the resident engine leaves
// 2,048 on each of an SM's four schedulers, one warp's at 64, so a picture's
// planes are built while the engine runs (with more, no warp could start until
// it left, and it waits for the planes). Bound by issue: about 5 instructions
// an output sample, where a multiply-add per tap and the passes' round trip
// through shared memory took about 50. One 1080p reference 61 -> 21 us, one of
// 2160p at 10 bits 203 -> 85 us (3.3 TB/s written), one of 360p 13 -> 8 us; up
// to 94 registers, with half as many warps an SM, were no faster.
template <class S>
__global__ void __launch_bounds__(64, 16) hevc_phase_kernel(const S* g, S* planes, int64_t plane_elems, int stride,
                                                            int prow, int pcol, int bd, int strip) {
  const int x = blockIdx.x * kPhaseTX + (threadIdx.x & 31) * 4, y0 = blockIdx.y * strip;
  if (x >= pcol) return;
  const int rows = min(strip, prow - y0);
  const int fx = blockIdx.z * 2 + (threadIdx.x >> 5);
  if (fx == 0) phase_columns<S, 0>(g, planes, plane_elems, stride, prow, pcol, bd, x, y0, rows);
  else if (fx == 1) phase_columns<S, 1>(g, planes, plane_elems, stride, prow, pcol, bd, x, y0, rows);
  else if (fx == 2) phase_columns<S, 2>(g, planes, plane_elems, stride, prow, pcol, bd, x, y0, rows);
  else phase_columns<S, 3>(g, planes, plane_elems, stride, prow, pcol, bd, x, y0, rows);
}

}  // namespace

cudaError_t load_plane_kernels() {
  cudaError_t e = load_kernel(pad_plane_kernel<uint8_t>);
  if (e == cudaSuccess) e = load_kernel(pad_plane_kernel<uint16_t>);
  if (e == cudaSuccess) e = load_kernel(h264_hpel_kernel<uint8_t>);
  if (e == cudaSuccess) e = load_kernel(h264_hpel_kernel<uint16_t>);
  if (e == cudaSuccess) e = load_kernel(hevc_phase_kernel<uint8_t>);
  if (e == cudaSuccess) e = load_kernel(hevc_phase_kernel<uint16_t>);
  return e;
}

cudaError_t launch_pad_plane(const void* src, int bd, int w, int h, int sstride, DevPlanes dst, int ch, int pad,
                             cudaStream_t s) {
  const int prow = ch + 2 * pad, bps = bd == 8 ? 1 : 2, chunks = dst.stride * bps / 16;
  const bool in_place = src == static_cast<const uint8_t*>(dst.base) + (size_t)dst.origin * bps;
  dim3 blk(32, 8), grd((chunks + 31) / 32, (prow + 7) / 8);
  prefer_max_shared(pad_plane_kernel<uint8_t>);
  prefer_max_shared(pad_plane_kernel<uint16_t>);
  if (bd == 8)
    pad_plane_kernel<uint8_t><<<grd, blk, 0, s>>>((const uint8_t*)src, w, h, sstride, (uint8_t*)dst.base, dst.stride,
                                                  prow, pad, in_place);
  else
    pad_plane_kernel<uint16_t><<<grd, blk, 0, s>>>((const uint16_t*)src, w, h, sstride, (uint16_t*)dst.base,
                                                   dst.stride, prow, pad, in_place);
  return cudaGetLastError();
}

cudaError_t launch_h264_hpel(DevPlanes p, int bd, int cw, int ch, int pad, cudaStream_t s) {
  int prow = ch + 2 * pad, pcol = cw + 2 * pad;
  dim3 blk(32, 8), grd((pcol + 31) / 32, (prow + 7) / 8);
  prefer_max_shared(h264_hpel_kernel<uint8_t>);
  prefer_max_shared(h264_hpel_kernel<uint16_t>);
  if (bd == 8) {
    auto b = (uint8_t*)p.base;
    h264_hpel_kernel<uint8_t><<<grd, blk, 0, s>>>(b, b + p.plane_elems, b + 2 * p.plane_elems, b + 3 * p.plane_elems,
                                                  p.stride, prow, pcol, 255);
  } else {
    auto b = (uint16_t*)p.base;
    h264_hpel_kernel<uint16_t><<<grd, blk, 0, s>>>(b, b + p.plane_elems, b + 2 * p.plane_elems,
                                                   b + 3 * p.plane_elems, p.stride, prow, pcol, (1 << bd) - 1);
  }
  return cudaGetLastError();
}

cudaError_t launch_hevc_phases(DevPlanes p, int bd, int w, int h, int pad, cudaStream_t s) {
  int prow = h + 2 * pad, pcol = w + 2 * pad;
  // Strips as long as one wave of warps allows (32 an SM), 8 to 64 rows: a
  // strip filters seven rows more than it writes, and a second wave that is
  // nearly empty costs as much as the first (strips for half a wave: 1080p at
  // 10 bits 30.9 us against 26.7, 2160p 58.7 against 57.4).
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int cols = (pcol + kPhaseTX - 1) / kPhaseTX, strips = std::max(1, nsm * 32 / (4 * cols));
  const int strip = std::min(64, std::max(8, (prow + strips - 1) / strips));
  dim3 blk(64), grd(cols, (prow + strip - 1) / strip, 2);
  prefer_max_shared(hevc_phase_kernel<uint8_t>);
  prefer_max_shared(hevc_phase_kernel<uint16_t>);
  if (bd == 8)
    hevc_phase_kernel<uint8_t><<<grd, blk, 0, s>>>((const uint8_t*)p.base, (uint8_t*)p.base, p.plane_elems, p.stride,
                                                   prow, pcol, bd, strip);
  else
    hevc_phase_kernel<uint16_t><<<grd, blk, 0, s>>>((const uint16_t*)p.base, (uint16_t*)p.base, p.plane_elems,
                                                    p.stride, prow, pcol, bd, strip);
  return cudaGetLastError();
}

}  // namespace rme
