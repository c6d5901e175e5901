// H.264 GIVEN jobs: one warp per job (h264_task's GIVEN path), jobs taken
// from the launch's queue, largest blocks first. (STANDALONE frames run in
// rows: rme_h264.cu, rme_rows.cu; HEVC's GIVEN jobs and AMP units:
// rme_flat.cu; the resident engine runs every kind as tasks.)
//
// What a job computes is the reference's search, step for step:
//   Search::int_search (encode/h264_hpel.rs:789-952) and Search::refine
//   (956-1021): predictor plus deduplicated candidates (rounded
//   (m + 2) >> 2, clamped to search_bounds), UMH cross and hexagon rings,
//   small diamond or the hexagon with its three-new-points continuation, the
//   square; half- then quarter-sample rings that skip points within one step
//   of the previous centre; SAD / SATD + MvCostTable rate, strict <.
//
// The reference scores one candidate at a time and takes it when strictly
// cheaper than the best so far. Every candidate of a step is known before
// the step (each ring is around a centre fixed for the step), so here a
// warp scores them together: a group of lanes per candidate computes its
// distortion and its rate, and the step's outcome is the warp minimum:
// the lowest-indexed candidate among those of least cost, taken when below
// the best. That is exactly the sequential strict-< walk: it ends on the
// least cost, and on the first candidate reaching it.
#include <algorithm>

#include "rme_search_impl.cuh"

namespace rme {
namespace {

// MINB is the number of resident blocks the register allocation is bounded
// for: 2 leaves more registers per thread (few long jobs run faster), 4 keeps
// more warps resident (many jobs hide more latency); the host's tuner picks
// per sample width and job count.
template <class S, int MINB>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, MINB) given_kernel(LaunchDesc L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpSmem<S>& sm = reinterpret_cast<WarpSmem<S>*>(smem_raw)[warp];
  if (lane < 5) sm.cnt[lane] = 0;
  __syncwarp();
  for (;;) {
    unsigned long long idx = 0;
    if (lane == 0) idx = atomicAdd(L.head, 1ull);
    idx = __shfl_sync(kFull, idx, 0);
    if (idx >= (unsigned long long)L.total) break;
    const uint32_t e = (uint32_t)L.ready[idx];
    const int f = (int)(e >> 24), t = (int)(e & 0xffffffu);
    const FrameDesc& F = L.frames[f];
    // A job of another kind, or past its frame, is a host bug: flag it and
    // skip it rather than read out of bounds.
    if (t >= F.ntasks || (sizeof(S) == 1) != (F.bd == 8) || F.codec != RME_CODEC_H264 || F.mode != RME_PRED_GIVEN) {
      if (lane == 0) atomicOr(L.status, kStatusBadTask);
      continue;
    }
    h264_task<S>(L, F, f, t, sm, lane);
    __syncwarp();
  }
  __syncwarp();
  if (lane < 5) atomicAdd(&L.counters[lane], sm.cnt[lane]);
}

template <class S>
size_t smem_bytes() {
  return sizeof(WarpSmem<S>) * kWarpsPerBlock;
}

template <class S, int MINB>
int blocks_per_sm() {
  int n = 0;
  cudaError_t e =
      cudaFuncSetAttribute(given_kernel<S, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<S>());
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, given_kernel<S, MINB>, kWarpsPerBlock * 32, smem_bytes<S>());
  return e == cudaSuccess && n > 0 ? n : 1;
}

// The shared-memory share of the SM's unified L1 that MINB blocks need
// (percent, rounded up): the rest stays L1 data cache, which the reference
// reads hit.
template <class S, int MINB>
int carveout_pct() {
  static int pct = -1;
  if (pct < 0) {
    int dev = 0, smem_sm = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        smem_sm <= 0) {
      cudaGetLastError();
      return 100;
    }
    const long need = (long)MINB * ((long)smem_bytes<S>() + 1024);
    pct = (int)std::min<long>(100, (need * 100 + smem_sm - 1) / smem_sm);
  }
  return pct;
}

template <class S, int MINB>
cudaError_t launch(const LaunchDesc& L, int grid, cudaStream_t s) {
  cudaError_t e =
      cudaFuncSetAttribute(given_kernel<S, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<S>());
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(given_kernel<S, MINB>, cudaFuncAttributePreferredSharedMemoryCarveout,
                           carveout_pct<S, MINB>());
  if (e != cudaSuccess) return e;
  given_kernel<S, MINB><<<grid, kWarpsPerBlock * 32, smem_bytes<S>(), s>>>(L);
  return cudaGetLastError();
}

template <class S>
int bps_variant(int v) {
  return v == 0 ? blocks_per_sm<S, 2>() : v == 2 ? blocks_per_sm<S, 4>() : blocks_per_sm<S, 3>();
}
template <class S>
cudaError_t launch_variant(const LaunchDesc& L, int v, int grid, cudaStream_t s) {
  return v == 0 ? launch<S, 2>(L, grid, s) : v == 2 ? launch<S, 4>(L, grid, s) : launch<S, 3>(L, grid, s);
}

}  // namespace

int h264_given_blocks_per_sm(int bytes_per_sample, int variant) {
  return bytes_per_sample == 1 ? bps_variant<uint8_t>(variant) : bps_variant<uint16_t>(variant);
}

cudaError_t launch_h264_given(const LaunchDesc& L, int bytes_per_sample, int variant, int grid, cudaStream_t s) {
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>(grid, (L.total + kWarpsPerBlock - 1) / kWarpsPerBlock));
  return bytes_per_sample == 1 ? launch_variant<uint8_t>(L, variant, g, s) : launch_variant<uint16_t>(L, variant, g, s);
}

}  // namespace rme
