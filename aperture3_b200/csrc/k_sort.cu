// Particle ordering on the device.
//
// Per-step tile counting sort. The push/deposit kernel walks each tile's
// particles in the current (stable) tile order and records, per particle,
// the direction d in 0..8 of the tile it moved to (9 = gone) and per-tile
// direction counts. Because the input is grouped by tile and a particle
// only moves to one of its tile's eight neighbours, the stable counting
// sort by new tile reduces to:
//   k_tile_newcount / k_scan_counts (one launch up to 1024 tiles): for each
//                   destination tile, sum the counts from its (up to nine)
//                   source tiles and scan the sums to get tile offsets;
//   k_tile_groups   gives each (source, direction) group its offset in the
//                   destination tile, sources in ascending tile index (part
//                   of the scan's launch up to 113 tiles);
//   k_order_scatter for each source tile, rank particles within their
//                   direction group in order and write them to
//                   group offset + rank.
// The result equals a stable counting sort of the previous order by the new
// tile key (core/particle_base_impl.hpp:250-305 applied to tile keys).
//
// Full rebuild (after binding or external changes) and sort_by_cell
// (cuda/core/particle_base_impl.cu:435-487) use a stable LSD radix sort.
#include <cuda_runtime.h>

#include <type_traits>

#include "ap_device.cuh"
#include "ap_internal.h"

namespace apb {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScatterThreads = 256;

struct TileTopo {
  int ntx, nty, ntiles, per0, per1;
};

// Source tile of destination (ux, uy) for direction (dx, dy) in -1..1, or
// -1 when it falls outside a non-periodic edge.
__device__ __forceinline__ int source_tile(const TileTopo &T, int ux, int uy, int dx, int dy) {
  int sx = ux - dx, sy = uy - dy;
  if (sx < 0) {
    if (!T.per0) return -1;
    sx += T.ntx;
  } else if (sx >= T.ntx) {
    if (!T.per0) return -1;
    sx -= T.ntx;
  }
  if (sy < 0) {
    if (!T.per1) return -1;
    sy += T.nty;
  } else if (sy >= T.nty) {
    if (!T.per1) return -1;
    sy -= T.nty;
  }
  return sx + sy * T.ntx;
}

// New population of destination tile u: the counts its (up to nine) source
// tiles recorded for the direction that leads to it.
__device__ __forceinline__ uint32_t new_population(const TileTopo &T, const uint32_t *cnt, int u) {
  const int ux = u % T.ntx, uy = u / T.ntx;
  uint32_t nu = 0;
#pragma unroll
  for (int d = 0; d < 9; ++d) {
    const int s = source_tile(T, ux, uy, d % 3 - 1, d / 3 - 1);
    if (s >= 0) nu += cnt[s * 10 + d];
  }
  return nu;
}

// Position of the first entry of group (source tile s, direction d) in the
// new order: inside the destination tile the groups stand by ascending
// source tile, those of one source by ascending direction.
__device__ __forceinline__ uint32_t group_offset(const TileTopo &T, const uint32_t *cnt,
                                                 const uint32_t *new_start, int s, int d) {
  const int sx = s % T.ntx, sy = s / T.ntx;
  int ux = sx + d % 3 - 1, uy = sy + d / 3 - 1;
  if (ux < 0 || ux >= T.ntx) {
    if (!T.per0) return 0;  // an empty group
    ux += ux < 0 ? T.ntx : -T.ntx;
  }
  if (uy < 0 || uy >= T.nty) {
    if (!T.per1) return 0;
    uy += uy < 0 ? T.nty : -T.nty;
  }
  uint32_t off = new_start[ux + uy * T.ntx];
#pragma unroll
  for (int e = 0; e < 9; ++e) {
    const int o = source_tile(T, ux, uy, e % 3 - 1, e / 3 - 1);
    if (o >= 0 && (o < s || (o == s && e < d))) off += cnt[o * 10 + e];
  }
  return off;
}

// One thread per (tile, direction): 2 us on 4096 tiles, where one thread per
// tile, sorting its nine sources in local memory, took 7 us (6 us on 16
// tiles). Computing the offsets inside the scatter's blocks was slower: the
// chain of loads stands before every tile's walk (65 -> 100 us on 16384
// tiles of 1000 particles).
__global__ void k_tile_groups(TileTopo T, const uint32_t *__restrict__ cnt,
                              const uint32_t *__restrict__ new_start,
                              uint32_t *__restrict__ grp_off) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < T.ntiles * 9) grp_off[i] = group_offset(T, cnt, new_start, i / 9, i % 9);
}

__global__ void k_tile_newcount(TileTopo T, const uint32_t *__restrict__ cnt,
                                uint32_t *__restrict__ newcount) {
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < T.ntiles; u += gridDim.x * blockDim.x)
    newcount[u] = new_population(T, cnt, u);
}

// Stable placement of one source tile's entries [b, e) in the new order by
// two passes over them: the list is cut into one contiguous segment per
// warp; pass 1 counts the directions of each segment (each lane adds its
// entries into packed per-direction counters, summed over the warp at the
// end), one barrier turns the counts into per-warp offsets, and pass 2 walks
// the segment again 32 entries at a time, ranking lanes that share a
// direction (a ballot for the entries that stay in the tile, nearly all of
// them; __match_any_sync for the rest), so every entry lands at group offset
// + entries of that direction before it. Both passes issue the loads of four
// 32-entry steps before using them.
struct ScatterOut {
  const uint32_t *old_order;  // null: the particle at list position p sits in slot slot0 + p
  const uint8_t *dir;
  uint32_t *new_order;
  uint32_t capacity, slot0;
  DevStatus *status;
};

constexpr int kScatterWarps = kScatterThreads / 32;
constexpr int kScatterU = 4;  // 32-entry steps per batch of loads

// Places entries [w0, w1) of one warp in order; s_base[d] holds the position
// of the next entry of each direction.
__device__ __forceinline__ void scatter_walk(const ScatterOut &S, uint32_t w0, uint32_t w1,
                                             uint32_t *s_base) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t base4 = s_base[4];
  for (uint32_t q = w0; q < w1; q += 32 * kScatterU) {
    uint32_t d[kScatterU], src[kScatterU];
#pragma unroll
    for (int u = 0; u < kScatterU; ++u) {
      const uint32_t p = q + 32 * u + lane;
      d[u] = p < w1 ? S.dir[p] : 10u;
      src[u] = p < w1 ? (S.old_order ? S.old_order[p] : S.slot0 + p) : 0u;
    }
#pragma unroll
    for (int u = 0; u < kScatterU; ++u) {
      if (q + 32 * u >= w1) break;
      const uint32_t dk = d[u];
      const uint32_t stay = __ballot_sync(0xffffffffu, dk == 4u);
      const uint32_t other = __ballot_sync(0xffffffffu, dk < 9u && dk != 4u);
      uint32_t dst = 0xffffffffu;
      if (dk == 4u) dst = base4 + __popc(stay & lt);
      base4 += __popc(stay);
      if (other) {
        if ((other >> lane) & 1u) {
          const uint32_t peers = __match_any_sync(other, dk);
          const uint32_t bs = s_base[dk];
          dst = bs + __popc(peers & lt);
          __syncwarp(other);
          if ((peers & lt) == 0u) s_base[dk] = bs + __popc(peers);
        }
        __syncwarp();
      }
      if (dst != 0xffffffffu) {
        if (dst < S.capacity)
          S.new_order[dst] = src[u];
        else
          atomicAdd(&S.status->tile_faults, 1ull);
      }
    }
  }
}

__device__ __forceinline__ void scatter_two_pass(const ScatterOut &S, uint32_t b, uint32_t e,
                                                 uint32_t (*s_cnt)[10], uint32_t (*s_base)[10],
                                                 const uint32_t *s_off) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n = e - b;
  const uint32_t seg = ((n + kScatterWarps * 32 - 1) / (kScatterWarps * 32)) * 32;
  const uint32_t w0 = b + min(n, warp * seg), w1 = b + min(n, (warp + 1) * seg);
  // pass 1: direction counts of this warp's segment; packed counters of 16
  // bits, directions 0-3 in c0, 4-7 in c1, 8-9 in c2, summed over the warp
  // into lane f's mycnt every 256 batches (at most 32 x 4 x 256 = 32768
  // entries per counter in between)
  unsigned long long c0 = 0, c1 = 0, c2 = 0;
  uint32_t mycnt = 0;  // lane f < 10: count of direction f
  auto flush = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      c0 += __shfl_xor_sync(0xffffffffu, c0, o);
      c1 += __shfl_xor_sync(0xffffffffu, c1, o);
      c2 += __shfl_xor_sync(0xffffffffu, c2, o);
    }
    const unsigned long long w = lane < 4 ? c0 : (lane < 8 ? c1 : c2);
    if (lane < 10) mycnt += (uint32_t)((w >> (16 * (lane & 3))) & 0xffffull);
    c0 = c1 = c2 = 0;
  };
  int batches = 0;
  for (uint32_t q = w0; q < w1; q += 32 * kScatterU) {
    if (++batches == 256) {
      flush();
      batches = 0;
    }
    uint32_t d[kScatterU];
#pragma unroll
    for (int k = 0; k < kScatterU; ++k) {
      const uint32_t p = q + 32 * k + lane;
      d[k] = p < w1 ? S.dir[p] : 10u;
    }
#pragma unroll
    for (int k = 0; k < kScatterU; ++k) {
      const unsigned long long one = 1ull << (16 * (d[k] & 3u));
      if (d[k] < 4u)
        c0 += one;
      else if (d[k] < 8u)
        c1 += one;
      else if (d[k] < 10u)
        c2 += one;
    }
  }
  flush();
  if (lane < 10) s_cnt[warp][lane] = mycnt;
  __syncthreads();
  if (lane < 9) {
    uint32_t off = s_off[lane];
    for (int w = 0; w < warp; ++w) off += s_cnt[w][lane];
    s_base[warp][lane] = off;
  }
  __syncwarp();
  // pass 2: stable placement
  scatter_walk(S, w0, w1, s_base[warp]);
}

// One CTA per source tile. With the per-chunk direction counts the push /
// deposit kernel recorded (chunk k of source tile s is list entries [k CH,
// (k + 1) CH) of the tile, its counts at entry old_start[s] / CH + s + k of
// chunk_count) the placement takes one pass: the counts become the group
// offset of every (chunk, direction), and warp w places chunks w, w + 8, ...
// Without them, and for tiles of more than kMaxChunks chunks, two passes.
constexpr int kMaxChunks = 128;

__global__ void __launch_bounds__(kScatterThreads)
    k_order_scatter(int ntiles, int ch, const uint32_t *__restrict__ old_start,
                    const uint32_t *__restrict__ grp_off,
                    const uint32_t *__restrict__ chunk_count, ScatterOut S) {
  __shared__ uint32_t s_cb[kMaxChunks][9];  // group offset of each (chunk, direction)
  __shared__ uint32_t s_base[kScatterWarps][10];
  __shared__ uint32_t s_cnt[kScatterWarps][10];
  __shared__ uint32_t s_off[9];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int s = blockIdx.x; s < ntiles; s += gridDim.x) {
    const uint32_t b = old_start[s], e = old_start[s + 1];
    const uint32_t n = e - b;
    const int nch = (int)((n + ch - 1) / ch);
    const uint32_t off = tid < 9 ? grp_off[s * 9 + tid] : 0u;
    if (chunk_count && nch <= kMaxChunks) {
      const size_t c0 = (size_t)(b / ch) + s;
      // the tile's chunk counts, loaded by all threads, then scanned per
      // direction in shared memory
      for (int i = tid; i < nch * 9; i += kScatterThreads)
        s_cb[i / 9][i % 9] = chunk_count[(c0 + i / 9) * 10 + i % 9];
      __syncthreads();
      if (tid < 9) {
        uint32_t run = off;
        for (int k = 0; k < nch; ++k) {
          const uint32_t v = s_cb[k][tid];
          s_cb[k][tid] = run;
          run += v;
        }
      }
      __syncthreads();
      for (int k = warp; k < nch; k += kScatterWarps) {
        if (lane < 9) s_base[warp][lane] = s_cb[k][lane];
        __syncwarp();
        const uint32_t w0 = b + (uint32_t)k * ch, w1 = min(e, w0 + ch);
        scatter_walk(S, w0, w1, s_base[warp]);
        __syncwarp();
      }
    } else {
      if (tid < 9) s_off[tid] = off;  // read after the barrier between the passes
      scatter_two_pass(S, b, e, s_cnt, s_base, s_off);
    }
    __syncthreads();
  }
}

// start[k] = first position of key k in the sorted keys[0, n), for
// k = 0..nbins (start[nbins] = position of the first key >= nbins).
// Four consecutive keys per thread and round (one 16-byte load of the aligned
// keys and the key before them): one key per thread and round was bound by the
// latency of its loads (26 us for 8.4 M keys, 33 MB).
__global__ void k_segment_starts(const uint32_t *__restrict__ keys, size_t n, uint32_t nbins,
                                 uint32_t *__restrict__ start) {
  for (size_t i0 = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) * 4; i0 <= n;
       i0 += (size_t)gridDim.x * blockDim.x * 4) {
    uint32_t k[4];
    if (i0 + 3 < n) {
      const uint4 q = *reinterpret_cast<const uint4 *>(keys + i0);
      k[0] = q.x;
      k[1] = q.y;
      k[2] = q.z;
      k[3] = q.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = i0 + u < n ? keys[i0 + u] : nbins;
    }
    uint32_t prev = i0 == 0 ? 0u : min(keys[i0 - 1], nbins) + 1u;  // first key not yet started
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t cur = min(k[u], nbins);
      if (i0 + u <= n)
        for (; prev <= cur; ++prev) start[prev] = (uint32_t)(i0 + u);
    }
  }
}

// Tile order of particles sorted by cell: the particles of tile t are, row
// by row, the contiguous runs [cell_start[first cell of the row], cell_start
// [one past the last cell]) -- which is the stable counting sort by tile of
// the cell-sorted array.
__global__ void k_tile_counts_from_cells(MeshK m, TilesK T, const uint32_t *__restrict__ cs,
                                         uint32_t *__restrict__ counts) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T.ntiles; t += gridDim.x * blockDim.x) {
    const int tx = t % T.ntx, ty = t / T.ntx;
    const int x0 = m.guard[0] + tx * T.tx;
    const int x1 = min(x0 + T.tx, m.dims[0] - m.guard[0]);
    const int y0 = m.guard[1] + ty * T.ty;
    const int y1 = min(y0 + T.ty, m.dims[1] - m.guard[1]);
    uint32_t n = 0;
    for (int y = y0; y < y1; ++y) n += cs[y * m.dims[0] + x1] - cs[y * m.dims[0] + x0];
    counts[t] = n;
  }
}

__global__ void k_tile_fill_from_cells(MeshK m, TilesK T, const uint32_t *__restrict__ cs,
                                       const uint32_t *__restrict__ tile_start,
                                       uint32_t *__restrict__ order, uint32_t slot0) {
  for (int t = blockIdx.x; t < T.ntiles; t += gridDim.x) {
    const int tx = t % T.ntx, ty = t / T.ntx;
    const int x0 = m.guard[0] + tx * T.tx;
    const int x1 = min(x0 + T.tx, m.dims[0] - m.guard[0]);
    const int y0 = m.guard[1] + ty * T.ty;
    const int y1 = min(y0 + T.ty, m.dims[1] - m.guard[1]);
    uint32_t out = tile_start[t];
    for (int y = y0; y < y1; ++y) {
      const uint32_t a = cs[y * m.dims[0] + x0], b = cs[y * m.dims[0] + x1];
      for (uint32_t i = a + threadIdx.x; i < b; i += blockDim.x) order[out + (i - a)] = slot0 + i;
      out += b - a;
    }
  }
}

// Keys for the full rebuild: tile of a bulk cell, ntiles otherwise; cells
// outside the bulk are emptied as the reference push does (ptc_updater.cu:
// 87-90).
// Keys of slots base + i, i < n (vals = the slots).
__global__ void k_tile_keys(MeshK m, TilesK T, uint32_t *cell, size_t base, size_t n,
                            uint32_t *keys, uint32_t *vals) {
  cell += base;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    uint32_t c = cell[i];
    uint32_t key = (uint32_t)T.ntiles;
    if (c != AP_MAX_CELL) {
      int c1 = (int)(c % (uint32_t)m.dims[0]);
      int c2 = (int)((c / (uint32_t)m.dims[0]) % (uint32_t)m.dims[1]);
      int c3 = (int)(c / ((uint32_t)m.dims[0] * (uint32_t)m.dims[1]));
      bool bulk = c1 >= m.guard[0] && c1 < m.dims[0] - m.guard[0] && c2 >= m.guard[1] &&
                  c2 < m.dims[1] - m.guard[1] && c3 >= m.guard[2] && c3 < m.dims[2] - m.guard[2];
      if (bulk) {
        int tx = (c1 - m.guard[0]) / T.tx;
        int ty = (m.dim > 1) ? (c2 - m.guard[1]) / T.ty : 0;
        key = (uint32_t)(tx + ty * T.ntx);
      } else {
        cell[i] = AP_MAX_CELL;
      }
    }
    keys[i] = key;
    vals[i] = (uint32_t)(base + i);
  }
}

// Exclusive scan of nbins tile populations into start[0..nbins] with one CTA,
// four consecutive tiles per thread and 4096 per round with a carry (coalesced
// 16-byte loads; one thread per contiguous run of counters took 22 us on
// 16384 tiles, bound by its strided loads); the largest population goes to
// n_max[0]. With kPop the populations are the new ones, computed here (up to
// 1024 tiles, one per thread); with kStarts they are the differences of a
// start array that stands already.
// The same pass lists the push / deposit's work items: a tile of n particles
// gives ceil(n / item_len) of them, their number in n_max[1], item_len in
// n_max[2], those past the list's end in n_max[3].
enum ScanSource { kCounts, kPop, kStarts };

struct ItemOut {
  uint2 *items;
  uint32_t cap, len;
};

__device__ __forceinline__ uint32_t warp_scan(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

template <ScanSource kSrc>
__global__ void __launch_bounds__(kScanThreads)
    k_scan_counts(TileTopo T, const uint32_t *__restrict__ counts, int nbins,
                  uint32_t *start, uint32_t *n_max, ItemOut I, uint32_t *__restrict__ grp_off) {
  constexpr int kPer = kSrc == kCounts ? 4 : 1;
  __shared__ uint32_t s_w[kScanThreads / 32], s_i[kScanThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t carry = 0, icarry = 0, mx = 0;
  for (int b0 = 0; b0 < nbins; b0 += kPer * kScanThreads) {
    const int b = b0 + tid * kPer;
    uint32_t v[kPer];
    if constexpr (kSrc == kPop) {
      v[0] = b < nbins ? new_population(T, counts, b) : 0u;
    } else if constexpr (kSrc == kStarts) {
      v[0] = b < nbins ? counts[b + 1] - counts[b] : 0u;
    } else if (b + 3 < nbins) {
      const uint4 q = *reinterpret_cast<const uint4 *>(counts + b);
      v[0] = q.x;
      v[1] = q.y;
      v[2] = q.z;
      v[3] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < kPer; ++k) v[k] = b + k < nbins ? counts[b + k] : 0u;
    }
    uint32_t own = 0, iown = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      own += v[k];
      iown += (v[k] + I.len - 1) / I.len;
      mx = max(mx, v[k]);
    }
    const uint32_t inc = warp_scan(own, lane), iinc = warp_scan(iown, lane);
    if (lane == 31) {
      s_w[warp] = inc;
      s_i[warp] = iinc;
    }
    __syncthreads();
    // every warp scans the warp sums
    const uint32_t ws = warp_scan(s_w[lane], lane), is = warp_scan(s_i[lane], lane);
    const uint32_t before = __shfl_sync(0xffffffffu, ws, max(warp - 1, 0));
    const uint32_t ibefore = __shfl_sync(0xffffffffu, is, max(warp - 1, 0));
    uint32_t run = carry + (warp ? before : 0u) + inc - own;
    uint32_t item = icarry + (warp ? ibefore : 0u) + iinc - iown;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      if (kSrc != kStarts && b + k < nbins) start[b + k] = run;
      run += v[k];
      for (uint32_t p = 0; p < v[k]; p += I.len, ++item)
        if (item < I.cap) I.items[item] = make_uint2((uint32_t)(b + k), p);
    }
    carry += __shfl_sync(0xffffffffu, ws, 31);
    icarry += __shfl_sync(0xffffffffu, is, 31);
    __syncthreads();
  }
  if (kSrc != kStarts && tid == 0) start[nbins] = carry;
  if (kSrc == kPop && grp_off && tid < nbins * 9)  // the barrier above: start stands
    grp_off[tid] = group_offset(T, counts, start, tid / 9, tid % 9);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) s_w[warp] = mx;
  __syncthreads();
  if (warp == 0) {
    mx = __reduce_max_sync(0xffffffffu, s_w[lane]);
    if (lane == 0) {
      n_max[0] = mx;
      n_max[1] = min(icarry, I.cap);
      n_max[2] = I.len;
      n_max[3] = icarry - min(icarry, I.cap);
    }
  }
}
static_assert(kScanThreads == 1024, "one warp scans the 32 warp sums");

// dst[i] = src[perm[i]], four consecutive entries per thread: the permutation
// and the result move 16 bytes at a time and four gathers are in flight. The first
// `head` entries, up to dst's 16-byte boundary, go one by one; with a head the
// permutation's words are read singly.
template <typename T>
__global__ void k_gather(const T *__restrict__ src, const uint32_t *__restrict__ perm, size_t n,
                         T *__restrict__ dst, int head) {
  const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t stride = (size_t)gridDim.x * blockDim.x * 4;
  if (t < (size_t)head && t < n) dst[t] = src[perm[t]];
  for (size_t i = head + t * 4; i < n; i += stride) {
    if (i + 3 < n) {
      uint4 q;
      if (head == 0)
        q = *reinterpret_cast<const uint4 *>(perm + i);
      else
        q = make_uint4(perm[i], perm[i + 1], perm[i + 2], perm[i + 3]);
      const T a = src[q.x], b = src[q.y], c = src[q.z], d = src[q.w];
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<uint4 *>(dst + i) = make_uint4(a, b, c, d);
      } else {
        *reinterpret_cast<ulonglong2 *>(dst + i) = make_ulonglong2(a, b);
        *reinterpret_cast<ulonglong2 *>(dst + i + 2) = make_ulonglong2(c, d);
      }
    } else {
      for (size_t j = i; j < n; ++j) dst[j] = src[perm[j]];
    }
  }
}

// The cells of a sorted store from the sort's keys (16 bytes at a time where
// the cell array allows it).
__global__ void k_cells_of_keys(const uint32_t *__restrict__ keys, size_t n, uint32_t empty,
                                uint32_t *__restrict__ cell, bool vec) {
  const size_t stride = (size_t)gridDim.x * blockDim.x * 4;
  for (size_t i = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) * 4; i < n; i += stride) {
    if (i + 3 < n) {
      uint4 q = *reinterpret_cast<const uint4 *>(keys + i);
      q.x = q.x == empty ? AP_MAX_CELL : q.x;
      q.y = q.y == empty ? AP_MAX_CELL : q.y;
      q.z = q.z == empty ? AP_MAX_CELL : q.z;
      q.w = q.w == empty ? AP_MAX_CELL : q.w;
      if (vec) {
        *reinterpret_cast<uint4 *>(cell + i) = q;
      } else {
        cell[i] = q.x;
        cell[i + 1] = q.y;
        cell[i + 2] = q.z;
        cell[i + 3] = q.w;
      }
    } else {
      for (size_t j = i; j < n; ++j) cell[j] = keys[j] == empty ? AP_MAX_CELL : keys[j];
    }
  }
}

int bits_for(uint32_t maxkey) {
  int b = 1;
  while (b < 32 && (maxkey >> b) != 0) ++b;
  return b;
}

int grid_for(Ctx &c, size_t n, int threads) {
  size_t g = (n + threads - 1) / threads;
  size_t cap = (size_t)c.num_sms * 16;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

// One member gathered by the sort's permutation (4- and 8-byte members move as
// bits).
cudaError_t gather_member(Ctx &c, const void *src, const uint32_t *perm, size_t n, int bytes,
                          void *dst) {
  const int off = (int)(reinterpret_cast<uintptr_t>(dst) & 15u);
  const int head = off ? (16 - off) / bytes : 0;  // an 8-byte member starts at 0 or 8
  // a member that fits the 126 MB L2 takes 16 blocks per SM (8.4 M 4-byte
  // entries: 32 us one per thread, 19 us so); a larger one four, which keeps
  // the sources in flight of a store in tile order close together (all eleven
  // members of 67 M: 2.98 ms one per thread, 3.2 ms with 16 blocks)
  const int blocks = n * (size_t)bytes <= (size_t)128 << 20 ? 16 : 4;
  int g = grid_for(c, (n + 3) / 4, 256);
  if (g > c.num_sms * blocks) g = c.num_sms * blocks;
  auto run = [&](auto *s, auto *d) {
    using T = std::remove_pointer_t<decltype(d)>;
    k_gather<T><<<g, 256, 0, c.stream>>>(s, perm, n, d, head);
  };
  if (bytes == 8)
    run(static_cast<const uint64_t *>(src), static_cast<uint64_t *>(dst));
  else
    run(static_cast<const uint32_t *>(src), static_cast<uint32_t *>(dst));
  c.launches++;
  return cudaGetLastError();
}

void launch_cells_of_keys(Ctx &c, const uint32_t *keys, size_t n, uint32_t empty, uint32_t *cell) {
  const bool vec = (reinterpret_cast<uintptr_t>(cell) & 15u) == 0;
  k_cells_of_keys<<<grid_for(c, (n + 3) / 4, 256), 256, 0, c.stream>>>(keys, n, empty, cell, vec);
  c.launches++;
}

// Stable radix sort of (keys[0], vals[0]) -> result pointers (k_radix.cu).
cudaError_t radix_pairs(Ctx &c, size_t n, int end_bit, uint32_t **keys_out,
                        uint32_t **vals_out) {
  return radix_sort_pairs(c, n, end_bit, keys_out, vals_out);
}

}  // namespace

namespace {

TileTopo topo_of(const Ctx &c) {
  return TileTopo{c.tiles.ntx, c.tiles.nty, c.tiles.ntiles, c.params.periodic[0],
                  c.params.periodic[1]};
}

// Work items of the next push: about three per resident CTA of the variants
// with four CTAs per SM, so that neither a grid of few tiles nor a few crowded
// tiles leave the rest of the chip idle at the end; variants with two or three
// get the same lengths, four to six items per CTA. A tile of at most one item's
// length stays whole.
// An item costs its field tile, a cleared and a flushed current tile, about
// 2 us beside the 3 - 6 us of a 256-particle chunk.
ItemOut item_out(Ctx &c) {
  const uint32_t ch = (uint32_t)chunk_of(c);
  const size_t n = c.item_total > 0 ? c.item_total : c.number - c.store_base;
  const size_t slots = (size_t)c.num_sms * 4 * 3;
  const size_t chunks = (n / ch + slots - 1) / slots;
  c.item_len = ch * (uint32_t)(chunks < 1 ? 1 : chunks);
  return ItemOut{c.items, (uint32_t)c.items_cap, c.item_len};
}

}  // namespace

cudaError_t launch_tile_scan(Ctx &c, const uint32_t *dir_count, uint32_t *new_start,
                             uint32_t *grp_off) {
  const TileTopo T = topo_of(c);
  const int nt = c.tiles.ntiles;
  const ItemOut I = item_out(c);
  const bool groups = nt * 9 <= kScanThreads;  // in the scan's block
  if (nt <= kScanThreads) {
    k_scan_counts<kPop><<<1, kScanThreads, 0, c.stream>>>(T, dir_count, nt, new_start, c.n_max, I,
                                                          groups ? grp_off : nullptr);
    c.launches++;
  } else {
    k_tile_newcount<<<(nt + 127) / 128, 128, 0, c.stream>>>(T, dir_count, c.newcount);
    k_scan_counts<kCounts><<<1, kScanThreads, 0, c.stream>>>(T, c.newcount, nt, new_start,
                                                             c.n_max, I, nullptr);
    c.launches += 2;
  }
  if (!groups) {
    k_tile_groups<<<(nt * 9 + 255) / 256, 256, 0, c.stream>>>(T, dir_count, new_start, grp_off);
    c.launches++;
  }
  return cudaGetLastError();
}

cudaError_t launch_order_scatter(Ctx &c, const uint32_t *old_start, const uint32_t *old_order,
                                 const uint8_t *dir, const uint32_t *grp_off,
                                 uint32_t *new_order, uint32_t slot0) {
  const int grid = c.tiles.ntiles < c.num_sms * 8 ? c.tiles.ntiles : c.num_sms * 8;
  const ScatterOut S{old_order, dir, new_order, (uint32_t)c.order_cap, slot0, c.status};
  k_order_scatter<<<grid, kScatterThreads, 0, c.stream>>>(
      c.tiles.ntiles, chunk_of(c), old_start, grp_off,
      c.chunk_count_ok ? c.chunk_count : nullptr, S);
  c.launches++;
  return cudaGetLastError();
}

// Scratch for the radix sorts: two key and two value buffers of n entries,
// the per-CTA digit counts, and an 8-byte-per-slot gather buffer.
int ensure_scratch(Ctx &c, size_t n) {
  if (n <= c.scratch_cap && c.keys[0]) return AP_OK;
  for (int i = 0; i < 2; ++i) {
    cudaFree(c.keys[i]);
    cudaFree(c.vals[i]);
    c.keys[i] = c.vals[i] = nullptr;
  }
  cudaFree(c.rx_counts);
  cudaFree(c.gather_tmp);
  c.rx_counts = nullptr;
  c.gather_tmp = nullptr;
  size_t cap = n < 1024 ? 1024 : n;
  for (int i = 0; i < 2; ++i) {
    if (cudaMalloc(&c.keys[i], cap * sizeof(uint32_t)) != cudaSuccess) return AP_ERR_NOMEM;
    if (cudaMalloc(&c.vals[i], cap * sizeof(uint32_t)) != cudaSuccess) return AP_ERR_NOMEM;
  }
  if (cudaMalloc(&c.rx_counts, radix_count_words(c.num_sms) * sizeof(uint32_t)) != cudaSuccess)
    return AP_ERR_NOMEM;
  if (cudaMalloc(&c.gather_tmp, cap * sizeof(uint64_t)) != cudaSuccess) return AP_ERR_NOMEM;
  c.scratch_cap = cap;
  return AP_OK;
}

// After a compaction: the slots after the live ones (none, or a few that left
// the grid) are empty.
__global__ void k_compact_tail(const uint32_t *live, uint32_t *cell, size_t n) {
  for (size_t i = *live + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    cell[i] = AP_MAX_CELL;
}

namespace {

ap_particles store_layout(void *buf, size_t cap) {
  unsigned char *b = static_cast<unsigned char *>(buf);
  ap_particles s;
  s.id = reinterpret_cast<uint64_t *>(b);
  s.x1 = reinterpret_cast<float *>(b + 8 * cap);
  s.x2 = s.x1 + cap;
  s.x3 = s.x2 + cap;
  s.p1 = s.x3 + cap;
  s.p2 = s.p1 + cap;
  s.p3 = s.p2 + cap;
  s.E = s.p3 + cap;
  s.weight = s.E + cap;
  s.cell = reinterpret_cast<uint32_t *>(s.weight + cap);
  s.flag = s.cell + cap;
  return s;
}

}  // namespace

// The scratch store (48 B per slot, allocated on first use).
static cudaError_t compact_store_scratch(Ctx &c, PtcK *out, uint64_t **out_id) {
  const size_t n = c.capacity > c.number ? c.capacity : c.number;
  if (!c.compact_buf || c.compact_cap < n) {
    cudaFree(c.compact_buf);
    c.compact_buf = nullptr;
    cudaError_t e = cudaMalloc(&c.compact_buf, n * 48);
    if (e != cudaSuccess) return e;
    c.compact_cap = n;
  }
  const ap_particles s = store_layout(c.compact_buf, c.compact_cap);
  *out = PtcK{s.x1, s.x2, s.x3, s.p1, s.p2, s.p3, s.E, s.weight, s.cell, s.flag};
  *out_id = s.id;
  return cudaSuccess;
}

// Output of a compaction. When the caller's capacity leaves a free region
// as large as the occupied one ([store_base, number) holds every particle;
// the other half of the capacity is empty), the push writes the tile-ordered
// copy straight into it and the old region becomes empty slots; otherwise
// into the scratch store, copied back afterwards.
cudaError_t compact_store(Ctx &c, PtcK *out, uint64_t **out_id) {
  const size_t half = c.capacity / 2;
  const size_t used = c.number - c.store_base;
  if (c.store_base == 0 && c.number <= half) {
    c.compact_direct = true;
    c.compact_dst = half;
  } else if (c.store_base >= half && used <= c.store_base) {
    c.compact_direct = true;
    c.compact_dst = 0;
  } else {
    c.compact_direct = false;
    c.compact_dst = 0;
  }
  if (c.compact_direct) {
    const size_t d = c.compact_dst;
    *out = PtcK{c.ptc.x1 + d, c.ptc.x2 + d, c.ptc.x3 + d, c.ptc.p1 + d,  c.ptc.p2 + d,
                c.ptc.p3 + d, c.ptc.E + d,  c.ptc.weight + d, c.ptc.cell + d, c.ptc.flag + d};
    *out_id = c.ptc.id + d;
    return cudaSuccess;
  }
  return compact_store_scratch(c, out, out_id);
}

// After the order update of a compacting push: `live` (device) slots were
// written from compact_dst on. Direct output: the old region becomes empty
// and the new high-water mark is compact_dst + (number - store_base);
// scratch output: copied back to slots [0, number). Either way the slots
// between the written ones and the high-water mark become empty.
cudaError_t compact_finish(Ctx &c, const uint32_t *live) {
  const size_t n = c.number - c.store_base;
  if (n == 0) return cudaSuccess;
  cudaError_t e;
  if (c.compact_direct) {
    e = cudaMemsetAsync(c.ptc.cell + c.store_base, 0xff, n * sizeof(uint32_t), c.stream);
    if (e != cudaSuccess) return e;
  } else {
    const ap_particles s = store_layout(c.compact_buf, c.compact_cap);
    const struct {
      void *dst;
      const void *src;
      size_t bytes;
    } back[11] = {{c.ptc.x1, s.x1, 4}, {c.ptc.x2, s.x2, 4},         {c.ptc.x3, s.x3, 4},
                  {c.ptc.p1, s.p1, 4}, {c.ptc.p2, s.p2, 4},         {c.ptc.p3, s.p3, 4},
                  {c.ptc.E, s.E, 4},   {c.ptc.weight, s.weight, 4}, {c.ptc.cell, s.cell, 4},
                  {c.ptc.id, s.id, 8}, {c.ptc.flag, s.flag, 4}};
    for (const auto &m : back) {
      e = cudaMemcpyAsync(m.dst, m.src, n * m.bytes, cudaMemcpyDeviceToDevice, c.stream);
      if (e != cudaSuccess) return e;
    }
    if (c.store_base > 0) {
      e = cudaMemsetAsync(c.ptc.cell + n, 0xff, (c.number - n) * sizeof(uint32_t), c.stream);
      if (e != cudaSuccess) return e;
    }
  }
  k_compact_tail<<<grid_for(c, n, 256), 256, 0, c.stream>>>(live, c.ptc.cell + c.compact_dst, n);
  c.launches++;
  c.number = c.compact_dst + n;
  c.store_base = c.compact_dst;
  return cudaGetLastError();
}

// Builds the tile order from scratch: stable sort of slots
// [store_base, number) by tile key, then tile offsets from a histogram.
cudaError_t rebuild_tile_order(Ctx &c) {
  const size_t n = c.number - c.store_base;
  const uint32_t nt = (uint32_t)c.tiles.ntiles;
  uint32_t *start = c.tile_start[c.cur];
  cudaError_t e;
  if (n > 0) {
    k_tile_keys<<<grid_for(c, n, 256), 256, 0, c.stream>>>(c.mk, c.tiles, c.ptc.cell,
                                                          c.store_base, n, c.keys[0],
                                                          c.vals[0]);
    c.launches++;
    uint32_t *ko, *vo;
    e = radix_pairs(c, n, bits_for(nt), &ko, &vo);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(c.order[c.cur], vo, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                        c.stream);
    if (e != cudaSuccess) return e;
    k_segment_starts<<<grid_for(c, n / 4 + 1, 256), 256, 0, c.stream>>>(ko, n, nt, start);
    c.launches++;
  } else {
    e = cudaMemsetAsync(start, 0, sizeof(uint32_t) * (nt + 1), c.stream);
    if (e != cudaSuccess) return e;
  }
  const ItemOut I = item_out(c);
  k_scan_counts<kStarts><<<1, kScanThreads, 0, c.stream>>>(topo_of(c), start, (int)nt, nullptr,
                                                           c.n_max, I, nullptr);
  c.launches++;
  c.order_valid = true;
  return cudaGetLastError();
}

namespace {


// Tile-order derived from the cell starts of a store sorted into slots
// [slot0, slot0 + live).
cudaError_t tile_order_from_cells(Ctx &c, uint32_t slot0) {
  const int nt = c.tiles.ntiles;
  k_tile_counts_from_cells<<<(nt + 255) / 256, 256, 0, c.stream>>>(c.mk, c.tiles, c.cell_start,
                                                                   c.dir_count);
  k_scan_counts<kCounts><<<1, kScanThreads, 0, c.stream>>>(topo_of(c), c.dir_count, nt,
                                                           c.tile_start[c.cur], c.n_max,
                                                           item_out(c), nullptr);
  k_tile_fill_from_cells<<<nt < c.num_sms * 8 ? nt : c.num_sms * 8, 256, 0, c.stream>>>(
      c.mk, c.tiles, c.cell_start, c.tile_start[c.cur], c.order[c.cur], slot0);
  c.launches += 3;
  c.order_valid = true;
  return cudaGetLastError();
}

}  // namespace

cudaError_t sort_by_cell(Ctx &c, size_t *new_number) {
  // a 1D context with a device-side count (pair injection) sorts over its
  // capacity and writes the new count on the device; a 2D store after a
  // compaction into the upper half sorts slots [store_base, number)
  c.order_valid = false;
  const bool device_count = c.pstate && c.mk.dim == 1;
  const size_t base = device_count ? 0 : c.store_base;
  const size_t n = (device_count ? c.capacity : c.number) - base;
  *new_number = 0;
  if (n == 0) {
    c.store_base = 0;
    return cudaSuccess;
  }
  const uint32_t ncells =
      (uint32_t)c.mesh.dims[0] * (uint32_t)c.mesh.dims[1] * (uint32_t)c.mesh.dims[2];
  uint32_t *ko, *vo;
  cudaError_t e = radix_sort_cells(c, c.ptc.cell, base, n, ncells,
                                   device_count ? &c.pstate->number : nullptr, bits_for(ncells),
                                   &ko, &vo);
  if (e != cudaSuccess) return e;
  // With compaction on and a free half of the capacity, each member is
  // gathered straight into that half (the store then occupies
  // [out0, out0 + live)); otherwise through the gather buffer and back to
  // slots [0, live) (cuda/core/particle_base_impl.cu:466-487). One member at
  // a time: the random reads of one array stay in L2, those of eleven at once
  // do not.
  const size_t half = c.capacity / 2;
  size_t out0 = 0;
  bool direct = false;
  if (!device_count && c.compact_interval > 0) {
    if (c.store_base == 0 && c.number <= half) {
      direct = true;
      out0 = half;
    } else if (c.store_base >= half && n <= c.store_base) {
      direct = true;
      out0 = 0;
    }
  }
  const struct {
    void *p;
    int bytes;
  } member[10] = {{c.ptc.x1, 4}, {c.ptc.x2, 4}, {c.ptc.x3, 4},     {c.ptc.p1, 4}, {c.ptc.p2, 4},
                  {c.ptc.p3, 4}, {c.ptc.E, 4},  {c.ptc.weight, 4}, {c.ptc.id, 8}, {c.ptc.flag, 4}};
  for (const auto &m : member) {
    unsigned char *p = static_cast<unsigned char *>(m.p);
    if (direct) {
      e = gather_member(c, p, vo, n, m.bytes, p + out0 * m.bytes);
    } else {
      e = gather_member(c, p, vo, n, m.bytes, c.gather_tmp);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(p, c.gather_tmp, n * m.bytes, cudaMemcpyDeviceToDevice, c.stream);
    }
    if (e != cudaSuccess) return e;
  }
  // the cells are the sort's keys: no gather, and no copy back
  launch_cells_of_keys(c, ko, n, ncells, c.ptc.cell + (direct ? out0 : 0));
  if (direct && out0 > 0) {  // the old particles sat below the new range: empty them
    e = cudaMemsetAsync(c.ptc.cell, 0xff, c.number * sizeof(uint32_t), c.stream);
    if (e != cudaSuccess) return e;
  }
  // cell_start over the sorted keys; cell_start[ncells] is the number of
  // non-empty slots (upper_bound of MAX_CELL - 1, particle_base_impl.cu:454-458)
  if (!c.cell_start) {
    e = cudaMalloc(&c.cell_start, sizeof(uint32_t) * ((size_t)ncells + 1));
    if (e != cudaSuccess) return e;
  }
  k_segment_starts<<<grid_for(c, n / 4 + 1, 256), 256, 0, c.stream>>>(ko, n, ncells, c.cell_start);
  c.launches++;
  if (device_count) {
    c.number_stale = true;
    return cudaMemcpyAsync(&c.pstate->number, c.cell_start + ncells, sizeof(uint32_t),
                           cudaMemcpyDeviceToDevice, c.stream);
  }
  uint32_t live = 0;
  e = cudaMemcpyAsync(&live, c.cell_start + ncells, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                      c.stream);
  if (e != cudaSuccess) return e;
  if (c.mk.dim == 2) {
    // the tile order of the cell-sorted particles, without another sort
    e = tile_order_from_cells(c, (uint32_t)out0);
    if (e != cudaSuccess) return e;
  }
  e = cudaStreamSynchronize(c.stream);
  if (e != cudaSuccess) return e;
  c.store_base = out0;
  *new_number = out0 + live;
  return cudaSuccess;
}

// photons.sort_by_cell (sim_data_impl.hpp:81; particle_base_impl.cu:435-487
// for photon_data): the same stable sort of the photon slots [0, number),
// each of the twelve members gathered through the scratch buffer, and the
// empty slots trimmed.
cudaError_t sort_photons(Ctx &c, size_t *new_number) {
  const size_t n = c.ph_number;
  *new_number = 0;
  if (n == 0) return cudaSuccess;
  if (ensure_scratch(c, n) != AP_OK) return cudaErrorMemoryAllocation;
  const uint32_t ncells =
      (uint32_t)c.mesh.dims[0] * (uint32_t)c.mesh.dims[1] * (uint32_t)c.mesh.dims[2];
  uint32_t *ko, *vo;
  cudaError_t e = radix_sort_cells(c, c.ph.cell, 0, n, ncells, nullptr, bits_for(ncells), &ko, &vo);
  if (e != cudaSuccess) return e;
  const struct {
    void *p;
    int bytes;
  } member[11] = {{c.ph.x1, 4}, {c.ph.x2, 4}, {c.ph.x3, 4},     {c.ph.p1, 4},
                  {c.ph.p2, 4}, {c.ph.p3, 4}, {c.ph.E, 4},      {c.ph.weight, 4},
                  {c.ph.path_left, 4},        {c.ph.id, 8},     {c.ph.flag, 4}};
  for (const auto &m : member) {
    e = gather_member(c, m.p, vo, n, m.bytes, c.gather_tmp);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(m.p, c.gather_tmp, n * m.bytes, cudaMemcpyDeviceToDevice, c.stream);
    if (e != cudaSuccess) return e;
  }
  launch_cells_of_keys(c, ko, n, ncells, c.ph.cell);
  if (!c.cell_start) {
    e = cudaMalloc(&c.cell_start, sizeof(uint32_t) * ((size_t)ncells + 1));
    if (e != cudaSuccess) return e;
  }
  k_segment_starts<<<grid_for(c, n / 4 + 1, 256), 256, 0, c.stream>>>(ko, n, ncells, c.cell_start);
  c.launches++;
  uint32_t live = 0;
  e = cudaMemcpyAsync(&live, c.cell_start + ncells, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                      c.stream);
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(c.stream);
  if (e != cudaSuccess) return e;
  *new_number = live;
  return cudaSuccess;
}

}  // namespace apb
