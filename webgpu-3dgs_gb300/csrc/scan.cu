// scan.cu - stage 2 of the rebin: exclusive prefix scan of splat_ref_counts.
//
// Replaces the reference's three dispatches prefix_scan_local / _blocks / _add
// (src/shaders/compute/prefix_scan_*.wgsl, scan_core.wgsl), whose middle phase
// is a single thread walking every block sum, with one single-pass kernel:
// tiles of 2048 counts are claimed in order through an atomic ticket, scanned
// with warp shuffles, and chained by decoupled look-back on a per-tile status
// word.  Output contract of prefix_scan_blocks.wgsl:41-42 is kept:
// offsets[n] = ref_counter[0] = total.
//
// Status words are 64-bit: [63:34] launch epoch, [33:32] flag, [31:0] value.
// Entries carrying another epoch than the launch's read as "not ready"; the
// depth sort's first kernel also zeroes the words, since a replayed graph repeats
// its epoch.  Prefixes are summed in
// 64 bits; a total that does not fit 32 bits saturates at 0xffffffff and
// latches DEVERR_CAPACITY (no rebin can hold that many refs).
#include "gs3d_internal.cuh"

namespace gs3d {
namespace {

constexpr int kThreads = 256;
constexpr int kItems = 8;
constexpr uint32_t kTile = kThreads * kItems;  // 2048 counts per tile
constexpr uint32_t kFlagAgg = 1u, kFlagInc = 2u;

__device__ __forceinline__ unsigned long long pack(uint32_t epoch, uint32_t flag, uint32_t v) {
  return ((unsigned long long)epoch << 34) | ((unsigned long long)flag << 32) | v;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// What is scanned: counts (through a permutation where gather is given); the
// cells covered by splat-views (cells8: from one-word rectangles, cells16: from
// the projected records); tile counts, written in tile_offsets' convention.
enum class Scan { counts, cells8, cells16, tiles };

struct ScanExtra {
  const uint32_t* rect8;
  const gs3d_projected_splat* proj;
  unsigned long long* ref_total;  // cells: the refs are added; tiles: read
};

// Cells and refs of a splat-view's tile rectangle [x0, x1] x [y0, y1].
__device__ __forceinline__ uint32_t rect_cells(uint32_t x0, uint32_t y0, uint32_t x1, uint32_t y1,
                                               unsigned long long& refs) {
  refs += (unsigned long long)(x1 - x0 + 1) * (y1 - y0 + 1);
  return (x1 / kCellSide - x0 / kCellSide + 1) * (y1 / kCellSide - y0 / kCellSide + 1);
}

template <Scan KIND>
__global__ void __launch_bounds__(kThreads)
    scan_kernel(const uint32_t* __restrict__ in, DepthSorted order, ScanExtra ex,
                uint32_t* __restrict__ out, uint32_t n, unsigned long long* __restrict__ status,
                uint32_t* __restrict__ ticket, uint32_t epoch, uint32_t* __restrict__ total_out,
                uint32_t* __restrict__ err) {
  __shared__ uint32_t s_tile, s_prefix;
  __shared__ uint32_t s_warp[kThreads / 32];
  __shared__ unsigned long long s_refs[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  after_predecessor(in, order.range, ex.rect8, ex.proj);
  const uint32_t* gather = order.range != nullptr ? order.ids() : nullptr;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t num_tiles = (n + kTile - 1) / kTile;
  const size_t base = (size_t)tile * kTile + (size_t)threadIdx.x * kItems;

  // 128-bit accesses need 16-byte aligned buffers (caller-provided pointers
  // may be offset); otherwise the scalar path is taken
  const bool vec_in = (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
  const bool vec_out = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  uint32_t v[kItems];
  if (KIND == Scan::cells8 || KIND == Scan::cells16) {
    unsigned long long refs = 0;
    uint32_t id[kItems], rect[kItems] = {};
#pragma unroll
    for (int k = 0; k < kItems; ++k) id[k] = (base + k < n) ? __ldg(gather + base + k) : 0u;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      v[k] = 0u;
      if (base + k >= n) continue;
      if (KIND == Scan::cells8) {
        const uint32_t r = rect[k] = __ldg(ex.rect8 + id[k]);
        const uint32_t x0 = r & 0xffu, y0 = (r >> 8) & 0xffu;
        if (r != kCulledRect)
          v[k] = rect_cells(x0, y0, x0 + ((r >> 16) & 0xffu), y0 + (r >> 24), refs);
      } else if (__ldg(in + id[k]) != 0u) {
        const uint4 r = __ldg(reinterpret_cast<const uint4*>(ex.proj + id[k]) + 3);
        v[k] = rect_cells(r.x, r.y, r.z, r.w, refs);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) refs += __shfl_xor_sync(0xffffffffu, refs, o);
    if (lane == 0) s_refs[warp] = refs;
    // Rectangles in depth order for the emit (whole groups of 8 fit the array).
    // The gather is what bounds this kernel: one L2 request a splat-view, 100 G
    // a second (24M splat-views 264 us; wider look-back windows and tiles of
    // 1024 to 8192 made no difference).
    if (KIND == Scan::cells8 && base < n) {
      uint4* r4 = reinterpret_cast<uint4*>(order.rects() + base);
      r4[0] = make_uint4(rect[0], rect[1], rect[2], rect[3]);
      r4[1] = make_uint4(rect[4], rect[5], rect[6], rect[7]);
    }
  } else if (gather != nullptr) {  // counts read through a permutation (fused rebin)
#pragma unroll
    for (int k = 0; k < kItems; ++k) v[k] = (base + k < n) ? __ldg(in + __ldg(gather + base + k)) : 0u;
  } else if (vec_in && base + kItems <= n) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(in + base));
    const uint4 b = __ldg(reinterpret_cast<const uint4*>(in + base) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < kItems; ++k) v[k] = (base + k < n) ? __ldg(in + base + k) : 0u;
  }
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) sum += v[k];

  const uint32_t winc = warp_inclusive(sum, lane);
  if (lane == 31) s_warp[warp] = winc;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < kThreads / 32 ? s_warp[lane] : 0u;
    const uint32_t wi = warp_inclusive(w, lane);
    if (lane < kThreads / 32) s_warp[lane] = wi - w;  // exclusive warp offsets
    const uint32_t tile_total = __shfl_sync(0xffffffffu, wi, kThreads / 32 - 1);
    if ((KIND == Scan::cells8 || KIND == Scan::cells16) && lane == 0) {
      unsigned long long refs = 0;
#pragma unroll
      for (int w8 = 0; w8 < kThreads / 32; ++w8) refs += s_refs[w8];
      if (refs) atomicAdd(ex.ref_total, refs);
    }

    // ---- decoupled look-back (warp 0) ----
    unsigned long long excl = 0;
    if (tile == 0) {
      if (lane == 0) st_relaxed_u64(status, pack(epoch, kFlagInc, tile_total));
    } else {
      if (lane == 0) st_relaxed_u64(status + tile, pack(epoch, kFlagAgg, tile_total));
      int pred = (int)tile - 1;
      bool timed_out = false;
      while (true) {
        const int idx = pred - lane;
        uint32_t flag = kFlagInc, val = 0;
        uint32_t spins = 0;
        while (true) {
          if (idx >= 0) {
            const unsigned long long w64 = ld_relaxed_u64(status + idx);
            flag = ((uint32_t)(w64 >> 34) == epoch) ? (uint32_t)(w64 >> 32) & 3u : 0u;
            val = (uint32_t)w64;
          } else {
            flag = kFlagInc;
            val = 0;
          }
          if (__all_sync(0xffffffffu, flag != 0u)) break;
          if (++spins > kSpinLimit) {
            timed_out = true;
            break;
          }
          if (spins > 32) __nanosleep(64);
        }
        if (__any_sync(0xffffffffu, timed_out)) {
          if (lane == 0) latch_error(err, DEVERR_TIMEOUT);
          break;
        }
        const uint32_t inc_mask = __ballot_sync(0xffffffffu, flag == kFlagInc);
        if (inc_mask) {
          const int first = __ffs(inc_mask) - 1;  // nearest inclusive predecessor
          unsigned long long x = lane <= first ? val : 0u;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
          excl += x;
          break;
        }
        unsigned long long x = val;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        excl += x;
        pred -= 32;
      }
    }
    const unsigned long long inc = excl + tile_total;
    const bool overflow = inc > 0xffffffffull;
    const uint32_t inc32 = overflow ? 0xffffffffu : (uint32_t)inc;
    if (lane == 0) {
      if (tile > 0) st_relaxed_u64(status + tile, pack(epoch, kFlagInc, inc32));
      if (overflow) latch_error(err, DEVERR_CAPACITY);
      s_prefix = overflow ? 0xffffffffu : (uint32_t)excl;
      if (tile == num_tiles - 1) {
        *total_out = inc32;
        if (KIND != Scan::tiles) out[n] = inc32;
      }
    }
  }
  __syncthreads();

  uint32_t run = s_prefix + s_warp[warp] + (winc - sum);
  uint32_t o[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    o[k] = run;
    run += v[k];
  }
  if (KIND == Scan::tiles) {
    // a tile after the last populated one keeps 0: its predecessor is empty and
    // every ref lies before it
    const unsigned long long all = *ex.ref_total;
    uint32_t before = base > 0 && base < n ? __ldg(in + base - 1) : 1u;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      if (base + k + 1 == n) out[n] = v[k] ? o[k] + v[k] : 0u;
      if (o[k] == all && before == 0u) o[k] = 0u;
      before = v[k];
    }
  }
  if (vec_out && base + kItems <= n) {
    reinterpret_cast<uint4*>(out + base)[0] = make_uint4(o[0], o[1], o[2], o[3]);
    reinterpret_cast<uint4*>(out + base)[1] = make_uint4(o[4], o[5], o[6], o[7]);
  } else {
#pragma unroll
    for (int k = 0; k < kItems; ++k)
      if (base + k < n) out[base + k] = o[k];
  }
}

__global__ void scan_empty_kernel(uint32_t* out, uint32_t* total_out) {
  out[0] = 0u;
  *total_out = 0u;
}

}  // namespace

size_t scan_status_words(uint32_t n) { return (n + kTile - 1) / kTile + 1; }

cudaError_t launch_scan(const uint32_t* counts, const DepthSorted* gather, uint32_t* offsets,
                        uint32_t n, unsigned long long* status, uint32_t* tile_counter,
                        uint32_t epoch, uint32_t* total_out, uint32_t* err, LaunchStream s) {
  if (n == 0) {
    scan_empty_kernel<<<1, 1, 0, s>>>(offsets, total_out);
    return cudaGetLastError();
  }
  const uint32_t tiles = (n + kTile - 1) / kTile;
  launch_after(scan_kernel<Scan::counts>, tiles, kThreads, 0, s, counts,
               gather ? *gather : DepthSorted{}, ScanExtra{}, offsets, n, status, tile_counter,
               epoch, total_out, err);
  return cudaGetLastError();
}

cudaError_t launch_scan_cells(const uint32_t* counts, const uint32_t* rect8,
                              const gs3d_projected_splat* proj, const DepthSorted& gather,
                              uint32_t* offsets, uint32_t n, unsigned long long* status,
                              uint32_t* tile_counter, uint32_t epoch, uint32_t* total_out,
                              unsigned long long* ref_total, uint32_t* err, LaunchStream s) {
  if (n == 0) {
    scan_empty_kernel<<<1, 1, 0, s>>>(offsets, total_out);
    return cudaGetLastError();
  }
  const uint32_t tiles = (n + kTile - 1) / kTile;
  const ScanExtra ex{rect8, proj, ref_total};
  if (rect8 != nullptr)
    launch_after(scan_kernel<Scan::cells8>, tiles, kThreads, 0, s, counts, gather, ex, offsets, n,
                 status, tile_counter, epoch, total_out, err);
  else
    launch_after(scan_kernel<Scan::cells16>, tiles, kThreads, 0, s, counts, gather, ex, offsets, n,
                 status, tile_counter, epoch, total_out, err);
  return cudaGetLastError();
}

cudaError_t launch_scan_tiles(const uint32_t* tile_counts, uint32_t* tile_offsets, uint32_t n,
                              const unsigned long long* ref_total, unsigned long long* status,
                              uint32_t* tile_counter, uint32_t epoch, uint32_t* total_out,
                              uint32_t* err, LaunchStream s) {
  const uint32_t tiles = (n + kTile - 1) / kTile;
  const ScanExtra ex{nullptr, nullptr, const_cast<unsigned long long*>(ref_total)};
  launch_after(scan_kernel<Scan::tiles>, tiles, kThreads, 0, s, tile_counts, DepthSorted{}, ex,
               tile_offsets, n, status, tile_counter, epoch, total_out, err);
  return cudaGetLastError();
}

}  // namespace gs3d
