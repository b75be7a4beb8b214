// depth_sort.cu - the fused rebin's order of the splat-views by depth: a stable
// LSD radix sort of the 32-bit depth keys bits(-depth) with their ids.
//
// The same onesweep scheme as sort.cu (decoupled look-back per digit, ranking
// by ballots, partitions fetched by bulk copies), with the digits fitted to the
// frame: the preprocess leaves the smallest and the largest key, and depths
// whose keys span less than 2^27 (farthest / nearest below 2^16, any view of a
// usual near and far plane) are sorted as key - smallest in three passes of 9
// bits; other frames (NaN depths among them) in four passes of 8 bits of the key
// itself.  Which of the two is decided on the device, by every kernel from the
// same two words; the fourth pass returns at once where three suffice, and the
// sorted arrays are then the B buffers (DepthSorted).
//
// With 512 bins every one of a block's 512 threads owns a digit in the offset
// and look-back phases (of 256 bins, half of them idled there).
//
// Culled splats carry key 2^32 - 1 and are capped to the last key of the span:
// they sort last, and where they tie with a splat at its very end they have no
// refs to put in front of it.
//
// Measured (GB300), 4 x 8-bit passes -> these, histogram included: 24M splat-views
// 795 -> 653 us, 3M 177 -> 120, 400k 79 -> 47, 20k 69 -> 29.  A pass moves 16 bytes
// a key; what bounds it is the ranking (issue slots 53% busy) and, below 1M
// keys, the chain of one partition.
#include <algorithm>
#include <mutex>

#include "gs3d_internal.cuh"

namespace gs3d {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
// Keys a thread ranks: 10 (12, as 8-bit passes take, would leave one block per
// SM beside the 16 KB of per-warp counts).  While partitions of 4 keys a thread
// number at most one per SM, a pass is bound by one partition's chain, of which
// ranking is 0.3 us a key: sort of 20k splats 37 -> 29 us, 100k 41 -> 34 (400k
// with 4 keys 46 -> 47; 6 keys up to two partitions per SM: 43, but a 500k frame
// with others beside it 464 -> 468).
constexpr int kItems = 10, kItemsSmall = 4;
template <int ITEMS>
constexpr uint32_t part_of() {
  return (uint32_t)(kThreads * ITEMS);
}
constexpr uint32_t kSmallSplats = 152 * part_of<kItemsSmall>();
constexpr uint32_t kBins = 512;                // one per thread
constexpr int kBits = 9;
constexpr uint32_t kFlagAgg = 1u, kFlagInc = 2u;
constexpr uint32_t kValueMask = (1u << 30) - 1u;
constexpr int kLookback = 16;
template <int ITEMS>
constexpr size_t buf_of() {
  return (size_t)part_of<ITEMS>() * 2 * sizeof(uint32_t);
}
template <int ITEMS>
constexpr size_t smem_of() {
  return 2 * buf_of<ITEMS>() + (size_t)kWarps * kBins * sizeof(uint16_t);
}

// Digit p of a key under the frame's mapping.
struct Digits {
  uint32_t base, cap, shift, mask;
  __device__ __forceinline__ uint32_t operator()(uint32_t key) const {
    return (min(key - base, cap) >> shift) & mask;
  }
};
__device__ __forceinline__ Digits digits_of(const DepthRange* range, int p) {
  const uint32_t lo = ~__ldg(&range->max_not), hi = __ldg(&range->max);
  return depth_three_passes(lo, hi) ? Digits{lo, (1u << (3 * kBits)) - 1u, (uint32_t)(kBits * p), kBins - 1u}
                                    : Digits{0u, 0xffffffffu, (uint32_t)(8 * p), 255u};
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Exclusive scan over the block's 512 values; one barrier (two calls are a
// barrier apart).
__device__ __forceinline__ uint32_t block_exclusive(uint32_t x, uint32_t* s_wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t inc = warp_inclusive(x, lane);
  if (lane == 31) s_wsum[warp] = inc;
  __syncthreads();
  const uint32_t w = lane < kWarps ? s_wsum[lane] : 0u;
  const uint32_t before = __shfl_sync(0xffffffffu, warp_inclusive(w, lane) - w, warp);
  return before + inc - x;
}

// Histograms of every digit place, and the clear of the passes' look-back
// status and of what later kernels of the frame want zeroed (a memset costs a
// launch: the six of a frame were 12 us of a 20k-splat frame's 160).  Sixteen keys a thread a round, loaded before the first add.
constexpr int kHistThreads = 256, kHistItems = 16;
__global__ void __launch_bounds__(kHistThreads)
    depth_histogram_kernel(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ count,
                           const DepthRange* __restrict__ range, uint32_t* __restrict__ g_hist,
                           uint32_t* __restrict__ status, size_t status_stride,
                           uint32_t part, ClearList clear) {
  __shared__ uint32_t s_hist[kDepthPasses][kBins];
  after_predecessor(keys, count, range);
  for (int k = threadIdx.x; k < kDepthPasses * (int)kBins; k += kHistThreads)
    (&s_hist[0][0])[k] = 0u;
  __syncthreads();
  const uint32_t n = *count;
  const size_t gtid = (size_t)blockIdx.x * kHistThreads + threadIdx.x;
  const size_t gstride = (size_t)gridDim.x * kHistThreads;
  const size_t words = (size_t)((n + part - 1) / part) * kBins;
  for (int p = 0; p < kDepthPasses; ++p)
    for (size_t k = gtid; k < words; k += gstride) status[p * status_stride + k] = 0u;
#pragma unroll
  for (int c = 0; c < ClearList::kMax; ++c)
    for (size_t k = gtid; k < clear.words[c]; k += gstride) clear.p[c][k] = 0u;
  Digits d[kDepthPasses];
#pragma unroll
  for (int p = 0; p < kDepthPasses; ++p) d[p] = digits_of(range, p);
  const bool four = d[0].base == 0u && d[0].mask == 255u;
  for (size_t b = (size_t)blockIdx.x * kHistThreads * kHistItems; b < n;
       b += gstride * kHistItems) {
    uint32_t key[kHistItems];
#pragma unroll
    for (int i = 0; i < kHistItems; ++i) {
      const size_t k = b + (size_t)i * kHistThreads + threadIdx.x;
      key[i] = k < n ? __ldg(keys + k) : 0u;
    }
#pragma unroll
    for (int i = 0; i < kHistItems; ++i) {
      const bool in = b + (size_t)i * kHistThreads + threadIdx.x < n;
      // culled splats share one key: one add per warp
      const bool last = in && key[i] == 0xffffffffu;
      const uint32_t lasts = __ballot_sync(0xffffffffu, last);
      const bool add = last ? (threadIdx.x & 31) == (uint32_t)(__ffs(lasts) - 1) : in;
      const uint32_t by = last ? (uint32_t)__popc(lasts) : 1u;
      if (add) {
#pragma unroll
        for (int p = 0; p < kDepthPasses; ++p)
          if (p < 3 || four) atomicAdd(&s_hist[p][d[p](key[i])], by);
      }
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < kDepthPasses * (int)kBins; k += kHistThreads) {
    const uint32_t v = (&s_hist[0][0])[k];
    if (v) atomicAdd(g_hist + k, v);
  }
}

// One pass.  Partitions are claimed in order, late (after the look-back of the
// current one), and fetched into the other buffer while the current one is
// written out; barriers and waits as in sort.cu's onesweep_kernel.
template <int ITEMS>
__global__ void __launch_bounds__(kThreads, 2)
    depth_pass_kernel(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ ids_in,
                      uint32_t* __restrict__ keys_out, uint32_t* __restrict__ ids_out,
                      const uint32_t* __restrict__ count_in, const DepthRange* __restrict__ range,
                      int pass, const uint32_t* __restrict__ hist, uint32_t* __restrict__ status,
                      uint32_t* __restrict__ part_counter, uint32_t* __restrict__ err) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr size_t kBuf = buf_of<ITEMS>();
  constexpr uint32_t kPart = part_of<ITEMS>();
  // [kWarps][512] per-warp digit counts, then positions of the warps' items
  uint16_t* s_whist = reinterpret_cast<uint16_t*>(smem + 2 * kBuf);
  __shared__ uint32_t s_dest[kBins];
  __shared__ uint32_t s_wsum[kWarps];
  __shared__ uint32_t s_part[2];
  __shared__ uint64_t s_bar[2];
  after_predecessor(count_in, range, hist);
  const Digits digit = digits_of(range, pass);
  if (pass == 3 && digit.mask != 255u) return;  // three passes did
  if (blockDim.x != kThreads) {  // the indexing below is written for this block size
    if (threadIdx.x == 0) latch_error(err, DEVERR_RANGE);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t n = *count_in;
  const uint32_t num_parts = (n + kPart - 1) / kPart;
  auto claim_into = [&](int b) {  // one thread
    const uint32_t part = atomicAdd(part_counter, 1u);
    s_part[b] = part;  // published by the arrive below (release)
    if (part < num_parts) {
      unsigned char* buf = smem + b * kBuf;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&s_bar[b], (uint32_t)kBuf);
      bulk_g2s(buf, keys_in + (size_t)part * kPart, kPart * 4u, &s_bar[b]);
      bulk_g2s(buf + kPart * 4, ids_in + (size_t)part * kPart, kPart * 4u, &s_bar[b]);
    } else {
      mbar_arrive(&s_bar[b]);
    }
  };
  if (tid == 0) {
    mbar_init(&s_bar[0], 1);
    mbar_init(&s_bar[1], 1);
    fence_mbar_init();
    claim_into(0);  // under way while the bucket bases are summed
  }
  const uint32_t bucket = block_exclusive(__ldg(hist + tid), s_wsum);  // this thread's digit
  int b = 0;
  uint32_t phase0 = 0, phase1 = 0;
  for (;;) {
    uint16_t* wh = s_whist + warp * kBins;
    // this warp's count row; its previous readers finished before barrier C
    reinterpret_cast<uint4*>(wh)[lane] = make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4*>(wh)[lane + 32] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    uint32_t* s_keys = reinterpret_cast<uint32_t*>(smem + b * kBuf);
    uint32_t* s_ids = s_keys + kPart;
    const bool landed = mbar_wait(&s_bar[b], b ? phase1 : phase0);
    if (b) phase1 ^= 1u; else phase0 ^= 1u;
    const uint32_t part = landed ? s_part[b] : num_parts;
    const uint32_t count = part < num_parts ? min(kPart, n - part * kPart) : 0u;

    uint32_t key[ITEMS], id[ITEMS], dr[ITEMS];  // dr: digit | rank in warp << 9
    const uint32_t wloc = warp * (32u * ITEMS) + lane;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint32_t loc = wloc + i * 32u;
      const bool in = loc < count;
      key[i] = in ? s_keys[loc] : 0u;
      id[i] = in ? s_ids[loc] : 0u;
      // past the end: the last digit, after every item of it
      dr[i] = in ? digit(key[i]) : digit.mask;
    }
    // (the last fetch of a block finds no partition left)
    if (__any_sync(0xffffffffu, part < num_parts)) {
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const uint32_t d = dr[i];
        uint32_t peers = 0xffffffffu;
#pragma unroll
        for (int k = 0; k < kBits; ++k) {
          const uint32_t bit = (d >> k) & 1u;
          const uint32_t bal = __ballot_sync(0xffffffffu, bit);
          peers &= bit ? bal : ~bal;
        }
        const uint32_t prior = wh[d];
        __syncwarp();
        if ((__ffs(peers) - 1) == lane) wh[d] = (uint16_t)(prior + __popc(peers));
        __syncwarp();
        dr[i] = d | ((prior + __popc(peers & lanemask_lt())) << kBits);
      }
    }
    // A: counts complete, input buffer read, the fetch had landed for everyone
    if (!__syncthreads_and(landed)) {  // bounded wait gave up: stop this block
      if (tid == 0) {
        latch_error(err, DEVERR_TIMEOUT);
        mbar_wait(&s_bar[b], b ? phase1 ^ 1u : phase0 ^ 1u);  // one more bounded wait
      }
      break;
    }
    if (part >= num_parts) break;  // every thread read the same id

    // ---- this thread's digit: total, publication, start in the partition ----
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) total += s_whist[w * kBins + tid];
    const uint32_t pub = (uint32_t)tid == digit.mask ? total - (kPart - count) : total;
    uint32_t* st = status + (size_t)part * kBins + tid;
    st_relaxed_u32(st, ((part == 0 ? kFlagInc : kFlagAgg) << 30) | pub);
    const uint32_t dstart = block_exclusive(total, s_wsum);
    {
      uint32_t run = dstart;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const uint32_t t = s_whist[w * kBins + tid];
        s_whist[w * kBins + tid] = (uint16_t)run;
        run += t;
      }
    }
    __syncthreads();  // B: positions complete

    // ---- reorder the partition in place ----
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const uint32_t pos = wh[dr[i] & (kBins - 1u)] + (dr[i] >> kBits);
      s_keys[pos] = key[i];
      s_ids[pos] = id[i];
    }

    // ---- decoupled look-back, a digit a thread ----
    uint32_t excl = 0;
    bool ok = true;
    if (part > 0) {
      int pp = (int)part - 1;
      bool found = false;
      while (!found && ok && pp >= 0) {
        uint32_t lw[kLookback];
#pragma unroll
        for (int k = 0; k < kLookback; ++k)
          lw[k] = (pp - k >= 0) ? ld_relaxed_u32(status + (size_t)(pp - k) * kBins + tid)
                                : (kFlagInc << 30);
#pragma unroll
        for (int k = 0; k < kLookback; ++k) {
          if (found || !ok) break;
          uint32_t spins = 0;
          while ((lw[k] >> 30) == 0u) {  // not published yet: poll this one
            if (++spins > kSpinLimit) {
              ok = false;
              break;
            }
            if (spins > 16) __nanosleep(32);
            lw[k] = ld_relaxed_u32(status + (size_t)(pp - k) * kBins + tid);
          }
          if (!ok) break;
          excl += lw[k] & kValueMask;
          if ((lw[k] >> 30) == kFlagInc) found = true;
        }
        pp -= kLookback;
      }
      st_relaxed_u32(st, (kFlagInc << 30) | ((excl + pub) & kValueMask));
    }
    s_dest[tid] = bucket + excl - dstart;
    // C: partition reordered, destinations resolved
    if (!__syncthreads_and(ok)) {  // nothing written for this partition
      if (tid == 0) latch_error(err, DEVERR_TIMEOUT);
      break;  // no fetch is in flight: the next claim comes after this barrier
    }
    // the other buffer's last readers (previous write-out) passed barrier A
    if (tid == kThreads - 1) claim_into(b ^ 1);
    for (uint32_t j = tid; j < count; j += kThreads) {
      const uint32_t k = s_keys[j];
      const uint32_t dst = s_dest[digit(k)] + j;
      if (dst < n) {
        keys_out[dst] = k;
        ids_out[dst] = s_ids[j];
      } else {
        latch_error(err, DEVERR_RANGE);
      }
    }
    b ^= 1;
  }
}

template <int ITEMS>
cudaError_t pass_setup(int* per_sm) {
  // once per device and instance; contexts on other host threads may launch
  // concurrently
  static std::mutex mu;
  static int v[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = current_device(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (v[dev] == 0) {
    e = cudaFuncSetAttribute(depth_pass_kernel<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem_of<ITEMS>());
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, depth_pass_kernel<ITEMS>, kThreads,
                                                      smem_of<ITEMS>());
    if (e != cudaSuccess) return e;
    v[dev] = n > 0 ? n : 1;
  }
  *per_sm = v[dev];
  return cudaSuccess;
}

size_t parts_of(uint32_t n, uint32_t part) { return ((size_t)n + part - 1) / part; }

template <int ITEMS>
cudaError_t run_sort(const uint32_t* count, uint32_t n, const DepthRange* range, uint32_t* keys_a,
                     uint32_t* ids_a, uint32_t* keys_b, uint32_t* ids_b, uint32_t* status,
                     uint32_t* g_hist, uint32_t* part_counters, uint32_t* err,
                     const ClearList& clear, int sm_count, LaunchStream s) {
  int per_sm = 0;
  cudaError_t e = pass_setup<ITEMS>(&per_sm);
  if (e != cudaSuccess) return e;
  constexpr uint32_t part = part_of<ITEMS>();
  const size_t parts = std::max<size_t>(parts_of(n, part), 1);
  const size_t stride = parts * kBins;
  const size_t rounds = std::max<size_t>(parts_of(n, kHistThreads * kHistItems), 1);
  launch_after(depth_histogram_kernel, (unsigned)std::min<size_t>((size_t)sm_count * 8, rounds),
               kHistThreads, 0, s, keys_a, count, range, g_hist, status, stride, part, clear);
  const unsigned grid = (unsigned)std::min<size_t>((size_t)sm_count * per_sm, parts);
  for (int p = 0; p < kDepthPasses; ++p) {
    const bool even = p % 2 == 0;
    launch_after(depth_pass_kernel<ITEMS>, grid, kThreads, smem_of<ITEMS>(), s,
                 even ? keys_a : keys_b, even ? ids_a : ids_b, even ? keys_b : keys_a,
                 even ? ids_b : ids_a, count, range, p, g_hist + (size_t)p * kBins,
                 status + p * stride, part_counters + p, err);
  }
  return cudaGetLastError();
}

}  // namespace

size_t depth_sort_capacity(uint32_t n) { return (size_t)n + part_of<kItems>(); }
// enough for every smaller count too
size_t depth_sort_status_words(uint32_t n) {
  const size_t parts = std::max(parts_of(std::min(n, kSmallSplats), part_of<kItemsSmall>()),
                                parts_of(n, part_of<kItems>()));
  return (parts + 1) * kBins * kDepthPasses;
}

cudaError_t launch_sort_depth(const uint32_t* count, uint32_t capacity, const DepthRange* range,
                              uint32_t* keys_a, uint32_t* ids_a, uint32_t* keys_b,
                              uint32_t* ids_b, uint32_t* status, uint32_t* g_hist,
                              uint32_t* part_counters, uint32_t* err, const ClearList& clear,
                              int sm_count, LaunchStream s) {
  const auto run = capacity <= kSmallSplats ? run_sort<kItemsSmall> : run_sort<kItems>;
  return run(count, capacity, range, keys_a, ids_a, keys_b, ids_b, status, g_hist, part_counters,
             err, clear, sm_count, s);
}

}  // namespace gs3d
