// schedule.cu - work order of the raster.
//
// The reference dispatches one workgroup per tile in row-major order
// (GaussianSplatRenderer.ts:1259-1265).  Per-tile raster cost spans orders of
// magnitude, and a long tile that starts late stretches the whole pass, so
// the raster's workers pull tiles from a queue ordered by decreasing
// expected cost (longest-processing-time first).  The order only changes
// which worker renders a tile and when; every pixel's arithmetic is unchanged.
//
// Key-count schedule: expected cost = the tile's key count (the plain
// schedule the learned one falls back to).  Learned schedule: expected cost
// = the cost MLP's prediction (learned.cu).  Up to kOrderTiles tiles are
// ordered by one block (order_kernel), more by a radix sort of 16-bit keys.
//
// Both also split: the tiles whose expected cost per work item exceeds half of
// a raster worker's fair share of the frame (the head of the order) are shaded
// as two items per 8x8 pixel block, so a tile far heavier than the rest does not
// leave one worker running alone at the end of the raster.
#include "gs3d_internal.cuh"

namespace gs3d {
namespace {

constexpr int kThreads = 256;

// key = 0xffff - min(count, 0xffff): ascending key order = descending count;
// two 8-bit passes sort it.  The expected cost is the key count.
__global__ void __launch_bounds__(kThreads)
    keycount_keys_kernel(const uint32_t* __restrict__ tile_offsets, uint32_t num_tiles,
                         uint32_t* __restrict__ keys, uint32_t* __restrict__ ids,
                         float* __restrict__ est) {
  const uint32_t t = blockIdx.x * kThreads + threadIdx.x;
  if (t >= num_tiles) return;
  const uint32_t lo = __ldg(tile_offsets + t), hi = __ldg(tile_offsets + t + 1);
  const uint32_t n = hi > lo ? hi - lo : 0u;
  keys[t] = 0xffffu - min(n, 0xffffu);
  ids[t] = t;
  est[t] = (float)n;
}

// One block: the sum of the expected costs, then the count of tiles above
// half of a raster worker's fair share (deterministic: fixed per-thread order,
// fixed tree reduction).
constexpr int kHeavyThreads = 1024;
__global__ void __launch_bounds__(kHeavyThreads)
    heavy_count_kernel(const float* __restrict__ est, uint32_t n, uint32_t workers,
                       uint32_t items_per_tile, float floor, uint32_t all,
                       uint32_t* __restrict__ heavy) {
  __shared__ float s_sum[kHeavyThreads / 32];
  __shared__ uint32_t s_cnt[kHeavyThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (all) {
    if (threadIdx.x == 0) *heavy = n;
    return;
  }
  float sum = 0.0f;
  for (uint32_t t = threadIdx.x; t < n; t += kHeavyThreads) sum += __ldg(est + t);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  float total = 0.0f;
  for (int w = 0; w < kHeavyThreads / 32; ++w) total += s_sum[w];
  // a work item costs about est; the frame about sum(est) * items_per_tile
  const float thr =
      fmaxf(0.5f * total * (float)items_per_tile / (float)max(workers, 1u), floor);
  uint32_t cnt = 0;
  for (uint32_t t = threadIdx.x; t < n; t += kHeavyThreads) cnt += __ldg(est + t) > thr ? 1u : 0u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  if (lane == 0) s_cnt[warp] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t c = 0;
    for (int w = 0; w < kHeavyThreads / 32; ++w) c += s_cnt[w];
    *heavy = c;
  }
}

// The whole order in one block, for up to kOrderTiles tiles: buckets of 1/32
// octave of the expected cost, largest first (any order inside a bucket: the
// queue needs long tiles early, not an exact sort), and the tiles to split.
// Costs are walked three times (sum; bucket and heavy counts; placement)
// instead of six launches for keys, heavy count, histogram and two digit
// passes.
constexpr int kOrderThreads = 1024;
constexpr uint32_t kBuckets = 1024;  // 32 octaves
__device__ __forceinline__ uint32_t cost_bucket(float est) {
  // bits of 1 + est in [1, 2^32]: exponent and five bits of mantissa
  const uint32_t b = (__float_as_uint(fminf(fmaxf(est, 0.0f), 4.29e9f) + 1.0f) >> 18) - (127u << 5);
  return kBuckets - 1u - min(b, kBuckets - 1u);
}
template <bool LEARNED>
__global__ void __launch_bounds__(kOrderThreads)
    order_kernel(const uint32_t* __restrict__ tile_offsets, const float* __restrict__ pred,
                 const SchedGate* __restrict__ gate, uint32_t n, uint32_t workers,
                 uint32_t items_per_tile, float floor_keys, float floor_cost, uint32_t split_all,
                 uint32_t* __restrict__ order, uint32_t* __restrict__ heavy) {
  __shared__ uint32_t s_bucket[kBuckets];
  __shared__ float s_sum[kOrderThreads / 32];
  __shared__ uint32_t s_warp[kOrderThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  after_predecessor(tile_offsets, pred, gate);
  const bool learned = LEARNED && gate->use_learned != 0u;
  auto cost = [&](uint32_t t) -> float {
    if (learned) return expm1f(fminf(fmaxf(__ldg(pred + t), 0.0f), 15.99f));
    const uint32_t lo = __ldg(tile_offsets + t), hi = __ldg(tile_offsets + t + 1);
    return hi > lo ? (float)(hi - lo) : 0.0f;
  };
  s_bucket[tid] = 0u;
  __syncthreads();
  float sum = 0.0f;
  for (uint32_t t = tid; t < n; t += kOrderThreads) {
    const float c = cost(t);
    sum += c;
    atomicAdd(&s_bucket[cost_bucket(c)], 1u);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  float total = 0.0f;
  for (int w = 0; w < kOrderThreads / 32; ++w) total += s_sum[w];
  // a work item costs about the tile's cost; the frame about total * items
  const float thr = fmaxf(0.5f * total * (float)items_per_tile / (float)max(workers, 1u),
                          learned ? floor_cost : floor_keys);
  // bucket starts (a bucket a thread)
  {
    const uint32_t c = s_bucket[tid];
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += s_warp[w];
    s_bucket[tid] = before + inc - c;
  }
  __syncthreads();
  uint32_t over = 0;
  for (uint32_t t = tid; t < n; t += kOrderThreads) {
    const float c = cost(t);
    order[atomicAdd(&s_bucket[cost_bucket(c)], 1u)] = t;
    over += c > thr ? 1u : 0u;
  }
  over = __reduce_add_sync(0xffffffffu, over);
  __syncthreads();  // s_warp is rewritten
  if (lane == 0) s_warp[warp] = over;
  __syncthreads();
  if (tid == 0) {
    uint32_t c = 0;
    for (int w = 0; w < kOrderThreads / 32; ++w) c += s_warp[w];
    *heavy = split_all ? n : c;
  }
}

}  // namespace

cudaError_t launch_order(uint32_t schedule, const uint32_t* tile_offsets, const float* pred,
                         const SchedGate* gate, uint32_t num_tiles, uint32_t workers,
                         uint32_t items_per_tile, bool split_all, uint32_t* order,
                         uint32_t* heavy, LaunchStream s) {
  if (schedule == GS3D_SCHEDULE_LEARNED)
    launch_after(order_kernel<true>, 1, kOrderThreads, 0, s, tile_offsets, pred, gate, num_tiles,
                 workers, items_per_tile, (float)kHeavyKeys, (float)kHeavyCost,
                 split_all ? 1u : 0u, order, heavy);
  else
    launch_after(order_kernel<false>, 1, kOrderThreads, 0, s, tile_offsets, nullptr, nullptr,
                 num_tiles, workers, items_per_tile, (float)kHeavyKeys, (float)kHeavyCost,
                 split_all ? 1u : 0u, order, heavy);
  return cudaGetLastError();
}

cudaError_t launch_heavy_count(const float* est, uint32_t n, uint32_t workers,
                               uint32_t items_per_tile, float floor, bool all, uint32_t* heavy,
                               cudaStream_t s) {
  heavy_count_kernel<<<1, kHeavyThreads, 0, s>>>(est, n, workers, items_per_tile, floor,
                                                 all ? 1u : 0u, heavy);
  return cudaGetLastError();
}

cudaError_t launch_schedule(uint32_t schedule, const uint32_t* tile_offsets, uint32_t num_tiles,
                            const uint32_t* num_tiles_dev, uint32_t* keys_a, uint32_t* order_a,
                            uint32_t* keys_b, uint32_t* order_b, float* est, uint32_t* status,
                            Ctrl* ctrl, uint32_t workers, uint32_t items_per_tile, bool split_all,
                            int sm_count, cudaStream_t s) {
  if (num_tiles == 0) return cudaSuccess;
  cudaError_t e = cudaSuccess;
  if (schedule == GS3D_SCHEDULE_KEY_COUNT) {
    keycount_keys_kernel<<<(num_tiles + kThreads - 1) / kThreads, kThreads, 0, s>>>(
        tile_offsets, num_tiles, keys_a, order_a, est);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  e = launch_heavy_count(est, num_tiles, workers, items_per_tile,
                         schedule == GS3D_SCHEDULE_LEARNED ? (float)kHeavyCost : (float)kHeavyKeys,
                         split_all, &ctrl->raster_heavy, s);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(ctrl->sched_counter, 0, sizeof(ctrl->sched_counter), s);
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(ctrl->sched_hist, 0, sizeof(ctrl->sched_hist), s);
  if (e != cudaSuccess) return e;
  SortPlan plan{};
  plan.passes = 2;
  plan.word[0] = plan.word[1] = 1;
  plan.shift[0] = 0;
  plan.shift[1] = 8;
  plan.nbits[0] = plan.nbits[1] = 8;
  // two passes: the result is back in keys_a / order_a
  return launch_sort_u32(plan, num_tiles_dev, num_tiles, keys_a, order_a, keys_b, order_b,
                         status, &ctrl->sched_hist[0][0], ctrl->sched_counter, &ctrl->error,
                         sm_count, s);
}

}  // namespace gs3d
