// binning.cu - the fused rebin's second half of the (tile | depth) order: from
// the splats of each cell, in depth order, to the sorted refs and the tile
// ranges.
//
// The reference sorts every (splat, tile) ref (radix_scatter.wgsl) and then
// finds the tile boundaries (identify_tile_ranges.wgsl).  Sorting the refs
// themselves writes each of them once per digit pass, and a splat of tens of
// tiles is carried through as tens of refs.  Here a view's tile grid is cut into
// cells of 8x8 tiles.  The emit writes one entry per (splat, cell), in depth
// order, with the splat's rectangle inside the cell (12 bits); a stable sort by
// cell leaves every cell's splats contiguous and in depth order; and the refs
// are then expanded straight to their final places, written once:
//
//   cell_table   first entry of every cell, cell of every chunk of entries
//   chunk_count  refs per (chunk of 1024 entries, tile of the cell)
//   chunk_scan   per (cell, tile): exclusive prefix over the cell's chunks, and
//                the tile's total
//   (scan.cu)    tile totals -> tile_offsets, in the reference's convention
//   chunk_place  keys and values at tile offset + chunk prefix + rank
//
// A rank needs no counting: the 32 entries of a group make a 32 x 64 bit matrix
// (entry x tile of the cell), which its lanes transpose by five shuffles per
// word; a lane then holds, for two tiles, which entries cover them, in order.
//
// Bound: the counts and the placement by instruction issue (54% and 72% busy;
// 170 instructions per 32 refs placed where a splat covers one tile or two), not
// by HBM (12 bytes a ref written once).  Scan to tile ranges, ref sort -> this:
// 3M splats (16x16 tiles) 623 -> 270 us, 8 views of 3M (64x32) 1743 -> 1250, 3M
// heavy-tailed splats at 4K (32x32) 3317 -> 510.
#include <algorithm>

#include "gs3d_internal.cuh"

namespace gs3d {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kGroups = kChunkEntries / kThreads;  // groups of 32 entries per warp
static_assert(kGroups * kThreads == kChunkEntries, "whole groups");
// Refs placed through shared memory at a time.  A chunk of no more is put in
// tile order by a tile a lane; in a chunk of more, whose windows hold the refs
// of a few tiles each, a tile a lane left most lanes idle (143 instructions per
// 32 refs), so there a warp places a tile's refs together, an entry a lane.
// refs + ranges of 3M heavy-tailed splats at 4K (40M refs) 666 -> 394 us, a 3M
// frame 152 -> 141, 8 views of 3M 519 -> 503; windows of 4096 and of 16384
// were slower (12 views: 428 and 443 us, 416 with this one).
constexpr uint32_t kWindow = 10240;

// A warp's transpose of a 32x32 bit matrix: lane i holds row i and gets column i.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, uint32_t lane) {
  constexpr uint32_t m[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int j = 16 >> s;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) == 0 ? (x & m[s]) | ((y & m[s]) << j) : ((y & ~m[s]) >> j) | (x & ~m[s]);
  }
  return x;
}

// The 64-bit cover of an entry's rectangle: bit 8 y + x for tile (x, y) of the cell.
__device__ __forceinline__ uint2 entry_cover(uint32_t hi) {
  const uint32_t x0 = hi & 7u, y0 = (hi >> 3) & 7u, x1 = (hi >> 6) & 7u, y1 = (hi >> 9) & 7u;
  const uint32_t row = ((0xffu >> (7u - (x1 - x0))) << x0) * 0x01010101u;
  const unsigned long long rows = (~0ull >> (8u * (7u - (y1 - y0)))) << (8u * y0);
  return make_uint2(row & (uint32_t)rows, row & (uint32_t)(rows >> 32));
}

// First sorted entry whose cell is m or above, by one warp: 32 probes a step.
__device__ __forceinline__ uint32_t first_of_cell(const uint2* __restrict__ entries, uint32_t n,
                                                  uint32_t m, uint32_t lane) {
  uint32_t lo = 0, hi = n;  // the answer lies in [lo, hi]
  while (hi - lo > 0) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t i = lo + lane * step;
    const bool below = i < hi && (__ldg(&entries[i].x) >> kCellShift) < m;
    const uint32_t b = __popc(__ballot_sync(0xffffffffu, below));  // probes below come first
    if (b == 0) return lo;
    hi = min(hi, lo + b * step);
    lo = lo + (b - 1) * step + 1;
  }
  return lo;
}

__global__ void __launch_bounds__(kThreads)
    cell_table_kernel(const uint2* __restrict__ entries, const uint32_t* __restrict__ entry_total,
                      const unsigned long long* __restrict__ ref_total, uint32_t capacity,
                      uint32_t num_cells, uint32_t* __restrict__ cell_start,
                      uint32_t* __restrict__ chunk_cell) {
  after_predecessor(entries, entry_total, ref_total);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t m = (blockIdx.x * kThreads + threadIdx.x) >> 5;
  if (m >= num_cells) return;
  const uint32_t n = *ref_total > capacity ? 0u : *entry_total;
  const uint32_t a = m == 0 ? 0u : first_of_cell(entries, n, m, lane);
  const uint32_t b = m + 1 == num_cells ? n : first_of_cell(entries, n, m + 1, lane);
  if (lane == 0) {
    cell_start[m] = a;
    if (m + 1 == num_cells) cell_start[num_cells] = n;
  }
  // chunk slots of the cell: chunk_slot(a, m) on, those past its chunks unused
  const uint32_t first = chunk_slot(a, m), end = chunk_slot(b, m + 1);
  const uint32_t chunks = (b - a + kChunkEntries - 1) / kChunkEntries;
  for (uint32_t k = lane; first + k < end; k += 32)
    chunk_cell[first + k] = k < chunks ? m : kNoCell;
}

// One warp's groups of a chunk: entries and, per group, the transposed covers
// of this lane's two tiles (lane and lane + 32).
struct Covers {
  uint32_t w[kGroups][2];
};
template <bool KEEP>
__device__ __forceinline__ Covers chunk_covers(const uint2* __restrict__ entries,
                                               const uint32_t* __restrict__ ids, uint32_t first,
                                               uint32_t end, uint2* s_entry) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint2 e[kGroups];
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    const uint32_t loc = (warp * kGroups + g) * 32 + lane, i = first + loc;
    e[g] = i < end ? __ldg(entries + i) : make_uint2(0u, 0u);
    if (KEEP && i < end) s_entry[loc] = make_uint2(e[g].y, __ldg(ids + i));
  }
  Covers c;
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    const uint32_t i = first + (warp * kGroups + g) * 32 + lane;
    const uint2 m = i < end ? entry_cover(e[g].x) : make_uint2(0u, 0u);
    c.w[g][0] = transpose32(m.x, lane);
    c.w[g][1] = transpose32(m.y, lane);
  }
  return c;
}

// Refs of every chunk per tile of its cell.  Resident blocks over the chunk
// slots.
__global__ void __launch_bounds__(kThreads)
    chunk_count_kernel(const uint2* __restrict__ entries, const uint32_t* __restrict__ cell_start,
                       const uint32_t* __restrict__ chunk_cell, uint32_t num_cells,
                       uint32_t* __restrict__ counts) {
  __shared__ uint32_t s_cnt[2][kCellTiles];
  after_predecessor(entries, cell_start, chunk_cell);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t slots = chunk_slot(__ldg(cell_start + num_cells), num_cells);
  if (threadIdx.x < 2 * kCellTiles) (&s_cnt[0][0])[threadIdx.x] = 0u;
  __syncthreads();
  int p = 0;
  for (uint32_t k = blockIdx.x; k < slots; k += gridDim.x) {
    const uint32_t m = __ldg(chunk_cell + k);
    if (m == kNoCell) continue;
    const uint32_t a = __ldg(cell_start + m), end = __ldg(cell_start + m + 1);
    const uint32_t first = a + (k - chunk_slot(a, m)) * kChunkEntries;
    const Covers c = chunk_covers<false>(entries, nullptr, first,
                                         min(end, first + kChunkEntries), nullptr);
    uint32_t n0 = 0, n1 = 0;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      n0 += __popc(c.w[g][0]);
      n1 += __popc(c.w[g][1]);
    }
    if (n0) atomicAdd(&s_cnt[p][lane], n0);
    if (n1) atomicAdd(&s_cnt[p][lane + 32], n1);
    __syncthreads();
    if (threadIdx.x < kCellTiles) {
      counts[(size_t)k * kCellTiles + threadIdx.x] = s_cnt[p][threadIdx.x];
      s_cnt[p][threadIdx.x] = 0u;  // next added to two chunks on, past the next barrier
    }
    p ^= 1;
  }
}

// One block per cell: thread (segment, tile) sums its share of the chunks, the
// segments' sums are scanned, and the counts become exclusive prefixes over the
// cell's chunks.
constexpr int kScanThreads = 1024;
constexpr int kSegments = kScanThreads / (int)kCellTiles;
__global__ void __launch_bounds__(kScanThreads)
    chunk_scan_kernel(const ViewDesc* __restrict__ views, uint32_t n_views,
                      const uint32_t* __restrict__ cell_start, uint32_t* __restrict__ counts,
                      uint32_t* __restrict__ tile_counts) {
  __shared__ uint32_t s_sum[kSegments][kCellTiles];
  after_predecessor(views, cell_start);
  const uint32_t m = blockIdx.x, t = threadIdx.x % kCellTiles, seg = threadIdx.x / kCellTiles;
  const uint32_t a = __ldg(cell_start + m), b = __ldg(cell_start + m + 1);
  const uint32_t chunks = (b - a + kChunkEntries - 1) / kChunkEntries;
  uint32_t* c = counts + (size_t)chunk_slot(a, m) * kCellTiles + t;
  const uint32_t per = (chunks + kSegments - 1) / kSegments;
  const uint32_t k0 = min(chunks, seg * per), k1 = min(chunks, k0 + per);
  uint32_t sum = 0;
#pragma unroll 4
  for (uint32_t k = k0; k < k1; ++k) sum += c[(size_t)k * kCellTiles];
  s_sum[seg][t] = sum;
  __syncthreads();
  uint32_t run = 0;
  for (uint32_t s = 0; s < seg; ++s) run += s_sum[s][t];
#pragma unroll 4
  for (uint32_t k = k0; k < k1; ++k) {
    const uint32_t v = c[(size_t)k * kCellTiles];
    c[(size_t)k * kCellTiles] = run;
    run += v;
  }
  if (seg == kSegments - 1) {
    const CellGeom g = cell_geom(views, n_views, m);
    const uint32_t x = t % kCellSide, y = t / kCellSide;
    if (x < g.w && y < g.h) tile_counts[g.tile0 + y * g.tiles_x + x] = run;
  }
}

// Places the refs of every chunk.  A window of them at a time is put in tile
// order in shared memory (2 bytes a ref: tile of the cell and entry of the
// chunk), then written out with unit stride, each tile's run contiguous (with
// the runs of 32 entries written straight to memory, 3M heavy-tailed splats at
// 4K took 1210 us).
__global__ void __launch_bounds__(kThreads)
    chunk_place_kernel(const ViewDesc* __restrict__ views, uint32_t n_views,
                       const uint2* __restrict__ entries, const uint32_t* __restrict__ ids,
                       const uint32_t* __restrict__ cell_start,
                       const uint32_t* __restrict__ chunk_cell, uint32_t num_cells,
                       const uint32_t* __restrict__ prefixes,
                       const uint32_t* __restrict__ tile_offsets,
                       const unsigned long long* __restrict__ ref_total, uint32_t capacity,
                       uint2* __restrict__ keys, uint32_t* __restrict__ values,
                       uint32_t* __restrict__ ticket, uint32_t* __restrict__ err) {
  __shared__ uint2 s_entry[kChunkEntries];  // depth bits, splat-view
  __shared__ uint16_t s_slot[kWindow];
  __shared__ uint32_t s_cnt[kWarps][kCellTiles];  // counts, then exclusive positions
  __shared__ uint2 s_tile[kCellTiles];  // destination - position in the chunk, global tile
  __shared__ uint32_t s_half, s_total, s_next;
  after_predecessor(cell_start, ref_total);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t slots = chunk_slot(__ldg(cell_start + num_cells), num_cells);
  if (*ref_total > capacity) return;  // latched by the emit
  const uint32_t total = (uint32_t)*ref_total;
  for (;;) {
    if (threadIdx.x == 0) s_next = atomicAdd(ticket, 1u);
    __syncthreads();  // also: the previous chunk's readers are done
    const uint32_t k = s_next;
    if (k >= slots) break;
    const uint32_t m = __ldg(chunk_cell + k);
    if (m == kNoCell) {
      __syncthreads();
      continue;
    }
    const uint32_t a = __ldg(cell_start + m), end = __ldg(cell_start + m + 1);
    const uint32_t first = a + (k - chunk_slot(a, m)) * kChunkEntries;
    Covers c = chunk_covers<true>(entries, ids, first, min(end, first + kChunkEntries), s_entry);
    uint32_t n0 = 0, n1 = 0;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      n0 += __popc(c.w[g][0]);
      n1 += __popc(c.w[g][1]);
    }
    s_cnt[warp][lane] = n0;
    s_cnt[warp][lane + 32] = n1;
    __syncthreads();
    // two warps, a tile a lane: positions of the warps' refs within the chunk
    uint32_t sum = 0, inc = 0;
    if (threadIdx.x < kCellTiles) {
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const uint32_t v = s_cnt[w][threadIdx.x];
        s_cnt[w][threadIdx.x] = sum;
        sum += v;
      }
      inc = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
      if (threadIdx.x == 31) s_half = inc;
    }
    __syncthreads();
    if (threadIdx.x < kCellTiles) {
      const uint32_t start = inc - sum + (threadIdx.x >= 32 ? s_half : 0u);
#pragma unroll
      for (int w = 0; w < kWarps; ++w) s_cnt[w][threadIdx.x] += start;
      if (threadIdx.x == kCellTiles - 1) s_total = start + sum;
      const CellGeom g = cell_geom(views, n_views, m);
      const uint32_t x = threadIdx.x % kCellSide, y = threadIdx.x / kCellSide;
      uint2 td = make_uint2(0u, 0u);
      if (x < g.w && y < g.h) {
        td.y = g.tile0 + y * g.tiles_x + x;
        td.x = __ldg(tile_offsets + td.y) +
               __ldg(prefixes + (size_t)k * kCellTiles + threadIdx.x) - start;
      }
      s_tile[threadIdx.x] = td;
    }
    __syncthreads();
    const uint32_t refs = s_total;
    const bool dense = refs > kWindow;
    uint32_t pos0 = s_cnt[warp][lane], pos1 = s_cnt[warp][lane + 32];
    for (uint32_t wb = 0; wb < refs; wb += kWindow) {
      const uint32_t we = min(refs, wb + kWindow);
      if (dense) {  // a tile of the window at a time, an entry a lane
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t pos = h ? pos1 : pos0, cnt = h ? n1 : n0;
          for (uint32_t tiles = __ballot_sync(0xffffffffu, cnt && pos < we && pos + cnt > wb);
               tiles != 0u; tiles &= tiles - 1u) {
            const int tl = __ffs(tiles) - 1;
            uint32_t at = __shfl_sync(0xffffffffu, pos, tl) - wb;  // may start before the window
            const uint32_t code = ((h * 32 + tl) << 10) | (warp * kGroups * 32 + lane);
#pragma unroll
            for (int g = 0; g < kGroups; ++g) {
              const uint32_t who = __shfl_sync(0xffffffffu, c.w[g][h], tl);
              const uint32_t to = at + __popc(who & lanemask_lt());
              if (((who >> lane) & 1u) && to < we - wb) s_slot[to] = (uint16_t)(code + g * 32);
              at += __popc(who);
            }
          }
        }
      } else {  // the window is the whole chunk: a tile a lane
        uint16_t *p0 = s_slot + pos0, *p1 = s_slot + pos1;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          const uint32_t code = (lane << 10) | ((warp * kGroups + g) * 32);
          for (uint32_t w = c.w[g][0]; w; w &= w - 1) *p0++ = (uint16_t)(code + __ffs(w) - 1);
          for (uint32_t w = c.w[g][1]; w; w &= w - 1)
            *p1++ = (uint16_t)(code + (32u << 10) + __ffs(w) - 1);
        }
      }
      __syncthreads();
      for (uint32_t j = wb + threadIdx.x; j < we; j += kThreads) {
        const uint32_t sl = s_slot[j - wb];
        const uint2 t = s_tile[sl >> 10], en = s_entry[sl & (kChunkEntries - 1)];
        const uint32_t dst = t.x + j;
        if (dst < total) {
          keys[dst] = make_uint2(t.y, en.x);
          values[dst] = en.y;
        } else {
          latch_error(err, DEVERR_RANGE);
        }
      }
      __syncthreads();
    }
  }
}

}  // namespace

size_t chunk_slots_max(uint32_t capacity, uint32_t num_cells) {
  return (size_t)capacity / kChunkEntries + num_cells + 2;
}

cudaError_t launch_bin_count(const ViewDesc* views, uint32_t n_views, uint32_t num_cells,
                             const uint2* entries, const uint32_t* entry_total,
                             const unsigned long long* ref_total, uint32_t capacity,
                             uint32_t* cell_start, uint32_t* chunk_cell, uint32_t* chunk_counts,
                             uint32_t* tile_counts, int sm_count, LaunchStream s) {
  launch_after(cell_table_kernel, (num_cells + kWarps - 1) / kWarps, kThreads, 0, s, entries,
               entry_total, ref_total, capacity, num_cells, cell_start, chunk_cell);
  launch_after(chunk_count_kernel, sm_count * 8, kThreads, 0, s, entries, cell_start, chunk_cell,
               num_cells, chunk_counts);
  launch_after(chunk_scan_kernel, num_cells, kScanThreads, 0, s, views, n_views, cell_start,
               chunk_counts, tile_counts);
  return cudaGetLastError();
}

cudaError_t launch_bin_place(const ViewDesc* views, uint32_t n_views, uint32_t num_cells,
                             const uint2* entries, const uint32_t* ids, const uint32_t* cell_start,
                             const uint32_t* chunk_cell, const uint32_t* chunk_counts,
                             const uint32_t* tile_offsets, const unsigned long long* ref_total,
                             uint32_t capacity, uint2* keys, uint32_t* values, uint32_t* ticket,
                             uint32_t* err, int sm_count, LaunchStream s) {
  launch_after(chunk_place_kernel, sm_count * 8, kThreads, 0, s, views, n_views, entries, ids,
               cell_start, chunk_cell, num_cells, chunk_counts, tile_offsets, ref_total, capacity,
               keys, values, ticket, err);
  return cudaGetLastError();
}

}  // namespace gs3d
