// Fused Vay push + Esirkepov deposition + move for Cartesian 1D and 2D.
//
// Replaces Kernels::ptc_push_cart_{1,2}d and deposit_current_cart_{1,2}d
// (src/cuda/algorithms/ptc_updater.cu:21-141, 220-386), which the
// reference runs as two grid-stride launches with global float atomics.
//
// 2D design: the particles are kept in a stable tile order (one list of
// slot indices per tile of TX x TY cells, maintained by a counting sort each
// step). A persistent CTA takes work items from a queue, an item being a
// tile's list or a part of a long one; for each item it
//   1. brings the E/B tile plus a one-cell halo into shared memory with six
//      TMA 2D tiled loads (no multicast) completing on an mbarrier, and lays
//      it out as one record per cell (wide loads in the gather),
//   2. zeroes a shared-memory J (and Rho) tile with a two-cell halo,
//   3. walks the item's list in chunks of CH particles, the next chunk's
//      records in flight (cp.async) while this one is worked on: each warp
//      pushes and deposits 32 particles that sit CH/32 places apart in the
//      list (in a cell-sorted list that puts the lanes of a warp in
//      different cells, so their current updates do not collide), and a
//      coalesced store writes the chunk back,
//   4. flushes the J tile once into 64-bit accumulators in global memory; a
//      finalize pass folds the periodic guards and rounds each cell once to
//      FP32, and
//   5. records, per particle, the direction of its new tile (0..8, 9 = gone)
//      plus per-direction counts, which the order update consumes.
//
// Current and charge are accumulated exactly in fixed point: each FP32
// contribution (in 2D Cartesian runs the reference's up to the rounding of
// its products, whose factors are grouped per row and column; elsewhere the
// reference's value) becomes X = rint(v * 2^S), added as a
// high word X >> L (int32) and a low word X mod 2^L (uint32) with native
// 32-bit shared atomics. S and L are chosen from the largest tile population
// n so that neither word can overflow over n contributions; the sums are
// exact, so the result does not depend on the order of the atomics.
#include <cuda.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "ap_device.cuh"
#include "ap_internal.h"

namespace apb {

namespace {

constexpr int kThreads2D = 256;
constexpr uint32_t kDirGone = 9;
constexpr uint32_t kMbarSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\t"
      "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}

// Bounded wait on an mbarrier phase; returns false when the limit is hit.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          uint32_t limit = kMbarSpinLimit) {
  uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void tma_load_2d(float *dst, const CUtensorMap *map, int x, int y,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 4-byte asynchronous global -> shared copy (no register round trip).
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *gmem_src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(smem_dst)),
               "l"(gmem_src)
               : "memory");
}

__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Waits until at most N of this thread's committed groups are in flight.
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Bits needed to represent n (ceil(log2(n + 1))).
__device__ __forceinline__ int bits_of(uint32_t n) { return 32 - __clz(n); }

// Fixed-point format for sums of at most 2^lg contributions of magnitude at
// most qw: |X| < 2^(B-1), hi = X >> L with L = 32 - lg. With B = 63 - 2 lg,
// |sum hi| < 2^30 and sum lo < 2^32 over 2^lg contributions.
__device__ __forceinline__ FixedFmt fixed_format(int lg, int B, float qw) {
  FixedFmt f;
  f.L = 32 - lg;
  int S = B - 2;
  if (qw > 0.0f) S -= ilogbf(qw);
  f.S = max(-100, min(100, S));
  return f;
}

struct Acc32 {
  int *hi;
  unsigned *lo;
};

__device__ __forceinline__ void add_fixed(const Acc32 &a, int o, float v, float scale, int L) {
  const long long X = __float2ll_rn(v * scale);  // exact scaling by a power of two
  atomicAdd(a.hi + o, (int)(X >> L));
  atomicAdd(a.lo + o, (unsigned)X & ((1u << L) - 1u));
}

// The same for a contribution already scaled by 2^S. Scaling by a power of
// two commutes with rounding, so for a product a * b the value
// (a * 2^S) * b equals (a * b) * 2^S bit for bit whenever the result is a
// normal float; a result below the normal range rounds to X = 0 either way.
// The low word takes all 32 low bits of X (mod 2^32): with H the sum of the
// high words, the exact total is H * 2^L plus a remainder in [0, 2^32), which
// the low sum gives mod 2^32 (fixed_total), so the low bits need no mask.
__device__ __forceinline__ void add_fixed_scaled(const Acc32 &a, int o, float vs, int L) {
  const long long X = __float2ll_rn(vs);
  atomicAdd(a.hi + o, (int)(X >> L));
  atomicAdd(a.lo + o, (unsigned)X);
}

// The exact sum behind the two words of add_fixed_scaled: sum X = H * 2^L +
// sum (X mod 2^L), the last sum below 2^32 for at most 2^lg contributions
// (L = 32 - lg).
__device__ __forceinline__ long long fixed_total(int H, unsigned lo, int L) {
  const long long high = (long long)H * (1ll << L);
  return high + (long long)(lo - (unsigned)high);
}

// Chunks of at most 256 particles are double-buffered: the loads of the
// next chunk run while the current one is pushed and deposited.
template <int CH>
constexpr bool pipelined() {
  return CH <= 256;
}

template <int TX, int TY, int CH>
struct TileGeom {
  static constexpr int BX = TX + 8;   // field box width: x start rounded down to 4 floats
  static constexpr int BY = TY + 2;   // one halo row on each side
  static constexpr int FSZ = ((BX * BY + 31) / 32) * 32;  // 128-byte aligned stride
  static constexpr size_t raw_bytes() { return 4 * 6 * FSZ; }  // the six loaded components
  static constexpr int RX = TX + 1;   // field records of nodes x0 - 1 .. x0 + TX - 1 of a row
  static constexpr size_t rec_bytes() { return (48 * RX * BY + 127) / 128 * 128; }
  static constexpr int JX = TX + 4;   // J tile: two halo cells on each side
  static constexpr int JY = TY + 4;
  static constexpr int JSZ = JX * JY;
  static constexpr int SP = CH + CH / 32;  // staged chunk, one pad word per 32
  static constexpr int HDR = 128;     // mbarrier, tile id, abort flag, counters
  static constexpr size_t stage_bytes() { return 10 * 4 * SP + (SP + 3) / 4 * 4; }
  static constexpr int NBUF = pipelined<CH>() ? 2 : 1;
  // double-buffered chunks: the order indices of the next two chunks
  static constexpr size_t order_bytes() { return NBUF == 2 ? 2 * 4 * CH : 0; }
  // the components land in the last staged-chunk buffer, which the first
  // chunk of an item does not use when there are two
  static constexpr size_t stage0_bytes() { return NBUF == 2 ? (stage_bytes() + 127) / 128 * 128 : 0; }
  static constexpr size_t stage1_bytes() {
    return stage_bytes() > raw_bytes() ? stage_bytes() : raw_bytes();
  }
  static constexpr size_t smem_bytes(int nrho, bool ls = false) {
    return HDR + rec_bytes() + stage0_bytes() + stage1_bytes() + 8 * (3 + nrho) * JSZ +
           (ls ? 4 * JSZ : 0) + order_bytes();
  }
  // The limit belongs to the kernel on its device, not to a context or a
  // launch: every caller sets the same one, which holds any number of species
  // (of the 227 KB a block may have, less the batch's parameters).
  template <class Kernel>
  static cudaError_t allow_smem(Kernel *kern) {
    constexpr size_t most = smem_bytes(AP_MAX_SPECIES, true);
    static_assert(most + sizeof(PushDepositParams) <= 227 * 1024, "shared memory of a block");
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
  }
};

// Lane l of a warp works on element l * CH / 32 + k: with one pad word per 32
// elements the 32 lanes of a chunk of 256 (8 apart) fall into 32 banks, and so
// do 32 consecutive elements of the coalesced loads and stores.
__device__ __forceinline__ int spos(int e) { return e + (e >> 5); }

// Write-back modes of a staged particle.
constexpr uint8_t kWritePos = 1;  // x1, x2, x3, cell
constexpr uint8_t kWriteMom = 2;  // p1, p2, p3, E
constexpr uint8_t kWriteFlag = 4; // flag (log-spherical outflow)
// Direction and mode of an element left to the second walk of its chunk.
constexpr uint8_t kLeft = 0xff;

// Shared-memory copy of one run's parameters (batched launches only).
template <bool kMulti>
__device__ __forceinline__ uint32_t *param_smem() {
  if constexpr (kMulti) {
    __shared__ __align__(16) uint32_t buf[sizeof(PushDepositParams) / 4];
    return buf;
  } else {
    return nullptr;
  }
}

// The fused push + deposit over the tiles of one run (kMulti false: the
// parameters P0 and tensor maps maps0 live in the kernel's parameter
// space) or of a batch of runs (kMulti true: runs[r] in global memory,
// run r owning items [base[r], base[r + 1]) of one queue; each CTA copies
// the parameters of the run whose item it takes into shared memory, so
// the per-particle code reads them from there and not through global
// loads that the particle stores could alias).
template <int TX, int TY, int CH, bool kTMA, bool kRho, bool kLS, bool kMulti>
__device__ __forceinline__ void push_deposit_tiles(const PushDepositParams &P0,
                                                   const CUtensorMap *maps0,
                                                   const RunDesc *__restrict__ runs,
                                                   const uint32_t *__restrict__ base, int nruns,
                                                   uint32_t *queue) {
  using G = TileGeom<TX, TY, CH>;
  constexpr int SP = G::SP;
  constexpr int PER_THREAD = CH / kThreads2D;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *mbar = reinterpret_cast<uint64_t *>(smem);
  int *s_tile = reinterpret_cast<int *>(smem + 8);
  int *s_abort = reinterpret_cast<int *>(smem + 12);
  uint32_t *s_cnt = reinterpret_cast<uint32_t *>(smem + 16);
  // field records of the tile's nodes (i, j): pairs of nodes i, i + 1, so that
  // a particle reads the four nodes of a component as two aligned vectors:
  // sEB[0] = (E1, E1+, B2, B2+), sEB[1] = (E2, E2+, B1, B1+) (the two
  // components of one record share their stagger), sZ[0] = (E3, E3+),
  // sZ[1] = (B3, B3+)
  constexpr int kNodes = G::RX * G::BY;
  float4 *sEB = reinterpret_cast<float4 *>(smem + G::HDR);
  float2 *sZ = reinterpret_cast<float2 *>(sEB + 2 * kNodes);
  unsigned char *s_stage = smem + G::HDR + G::rec_bytes();
  float *sRaw = reinterpret_cast<float *>(s_stage + G::stage0_bytes());
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    if (kTMA) mbar_init(mbar, 1);
    *s_abort = 0;
  }
  __syncthreads();

  uint32_t *s_pbuf = param_smem<kMulti>();
  uint32_t phase = 0;
  for (;;) {
    if (tid == 0) *s_tile = (int)atomicAdd(queue, 1u);
    if (tid < 10) s_cnt[tid] = 0;
    __syncthreads();
    const int g = *s_tile;
    const CUtensorMap *mp = maps0;
    const uint32_t *n_items = P0.n_items;
    const uint2 *items = P0.items;
    int k = g;  // work item of the run
    if constexpr (kMulti) {
      if ((uint32_t)g >= base[nruns]) break;
      int lo = 0, hi = nruns - 1;  // largest r with base[r] <= g
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= (uint32_t)g) lo = mid;
        else hi = mid - 1;
      }
      const uint32_t *src = reinterpret_cast<const uint32_t *>(&runs[lo].P);
      for (int i = tid; i < (int)(sizeof(PushDepositParams) / 4); i += kThreads2D)
        s_pbuf[i] = src[i];
      __syncthreads();
      mp = runs[lo].maps.m;
      k = g - (int)base[lo];
      n_items = reinterpret_cast<const PushDepositParams *>(s_pbuf)->n_items;
      items = reinterpret_cast<const PushDepositParams *>(s_pbuf)->items;
    } else {
      if ((uint32_t)k >= *n_items) break;
    }
    const uint2 item = items[k];
    const int t = (int)item.x;  // its tile, and the first and last list entry
    const int p0 = (int)item.y;
    const uint32_t item_len = n_items[1];
    const PushDepositParams &P =
        kMulti ? *reinterpret_cast<const PushDepositParams *>(s_pbuf) : P0;

    // shared-memory layout of this run (the charge tile depends on its
    // number of species)
    const int ncomp = 3 + (kRho ? P.num_species : 0);
    int *sJhi = reinterpret_cast<int *>(s_stage + G::stage0_bytes() + G::stage1_bytes());
    unsigned *sJlo = reinterpret_cast<unsigned *>(sJhi + ncomp * G::JSZ);
    // log-spherical: cell volumes over the J tile window
    float *s_dv = reinterpret_cast<float *>(sJlo + ncomp * G::JSZ);
    uint32_t *s_ord = reinterpret_cast<uint32_t *>(s_dv + (kLS ? G::JSZ : 0));
    const int dims0 = P.m.dims[0], dims1 = P.m.dims[1];
    const int g0 = P.m.guard[0], g1 = P.m.guard[1];
    const bool exact_grid = dims0 <= kExactCells && dims1 <= kExactCells;
    const int nacc = ncomp * G::JSZ;

    // fixed-point format of this update, from the largest tile population
    const int lg = max(4, bits_of(*P.n_max));
    const FixedFmt fx = fixed_format(lg, 63 - 2 * lg, P.qmax * *P.wmax);
    const float fscale = ldexpf(1.0f, fx.S);
    if (k == 0 && tid == 0) {
      *P.fx_used = fx;
      if (n_items[2]) atomicAdd(&P.status->tile_faults, (unsigned long long)n_items[2]);
    }

    const int tix = t % P.t.ntx, tiy = t / P.t.ntx;
    const int x0 = g0 + tix * TX, y0 = g1 + tiy * TY;
    const int xs = (x0 - 1) & ~3, ys = y0 - 1;
    const int jx0 = x0 - 2, jy0 = y0 - 2;

    // the tile's particle list; with double-buffered chunks the order
    // indices run two chunks ahead (slot (chunk index) & 1 of s_ord), so
    // the gathers of the next chunk never wait for them
    const uint32_t base = P.tile_start[t];
    const int n_tile = (int)(P.tile_start[t + 1] - base);
    const int n_t = min(n_tile, p0 + (int)item_len);  // end of the item
    auto prefetch_order = [&](int c0) {
      uint32_t *dst = s_ord + ((c0 / CH) & 1) * CH;
      const int nch = min(CH, n_t - c0);
      for (int e = tid; e < nch; e += kThreads2D) cp_async4(dst + e, P.order + base + c0 + e);
      cp_async_commit();
    };
    if (G::NBUF == 2) {
      if (p0 < n_t) prefetch_order(p0);
      if (p0 + CH < n_t) prefetch_order(p0 + CH);
    }

    // 3a. coalesced asynchronous load of the chunk at c0 into buffer b
    auto issue = [&](int c0, int b) {
      float *sb = reinterpret_cast<float *>(s_stage + b * G::stage0_bytes());
      const int nch = min(CH, n_t - c0);
#pragma unroll
      for (int k = 0; k < PER_THREAD; ++k) {
        const int e = tid + k * kThreads2D;
        if (e < nch) {
          const int s = spos(e);
          const uint32_t idx =
              G::NBUF == 2 ? s_ord[((c0 / CH) & 1) * CH + e] : P.order[base + c0 + e];
          reinterpret_cast<uint32_t *>(sb + 9 * SP)[s] = idx;
          cp_async4(sb + 7 * SP + s, P.p.cell + idx);
          cp_async4(sb + 8 * SP + s, P.p.flag + idx);
          cp_async4(sb + s, P.p.x1 + idx);
          cp_async4(sb + SP + s, P.p.x2 + idx);
          cp_async4(sb + 2 * SP + s, P.p.x3 + idx);
          cp_async4(sb + 3 * SP + s, P.p.p1 + idx);
          cp_async4(sb + 4 * SP + s, P.p.p2 + idx);
          cp_async4(sb + 5 * SP + s, P.p.p3 + idx);
          cp_async4(sb + 6 * SP + s, P.p.w + idx);
        }
      }
      cp_async_commit();
    };
    // 1. field tile: the copies run while the current tile is zeroed and the
    // first chunk's loads are issued
    if (kTMA && tid == 0) {
      fence_proxy_async_smem();
      mbar_expect_tx(mbar, 6u * G::BX * G::BY * 4u);
#pragma unroll
      for (int k = 0; k < 6; ++k) tma_load_2d(sRaw + k * G::FSZ, mp + k, xs, ys, mbar);
    }
    // 2. zero the current (and charge) tile
    for (int i = tid; i < nacc; i += kThreads2D) {
      sJhi[i] = 0;
      sJlo[i] = 0u;
    }
    if constexpr (kLS) {
      for (int i = tid; i < G::JSZ; i += kThreads2D) {
        const int gx = jx0 + i % G::JX, gy = jy0 + i / G::JX;
        s_dv[i] = (gx < dims0 && gy < dims1) ? P.dV.ptr[(size_t)gy * P.dV.pitch + gx] : 1.0f;
      }
    }
    if (G::NBUF == 2) {
      cp_async_wait_group<0>();
      __syncthreads();  // the order indices of the first chunks
      if (p0 < n_t) issue(p0, 0);
    }
    if (kTMA) {
      if (!mbar_wait(mbar, phase)) atomicExch(s_abort, 1);
    }
    for (int i = tid; i < kNodes; i += kThreads2D) {
      const int j = i / G::RX, col = i - j * G::RX;
      float f[6][2];
#pragma unroll
      for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          if constexpr (kTMA) {
            f[k][d] = sRaw[k * G::FSZ + j * G::BX + (x0 - 1 - xs) + col + d];
          } else {
            const int xx = x0 - 1 + col + d, yy = ys + j;
            f[k][d] = xx < dims0 && yy < dims1 ? P.F[k].ptr[(size_t)yy * P.F[k].pitch + xx] : 0.0f;
          }
        }
      sEB[i] = make_float4(f[0][0], f[0][1], f[4][0], f[4][1]);
      sEB[kNodes + i] = make_float4(f[1][0], f[1][1], f[3][0], f[3][1]);
      sZ[i] = make_float2(f[2][0], f[2][1]);
      sZ[kNodes + i] = make_float2(f[5][0], f[5][1]);
    }
    cp_async_wait_group<0>();  // the first chunk
    __syncthreads();
    if (*s_abort) {
      if (tid == 0) {
        atomicAdd(&P.status->timeouts, 1ull);
        mbar_wait(mbar, phase);  // give copies in flight one more bounded wait
      }
      break;
    }

    // 3. particles of this item, CH at a time
    int buf = 0;
    uint32_t cnt_prev = 0;  // threads < 10: the tile's direction count so far
    for (int c0 = p0; c0 < n_t; c0 += CH) {
      const int nch = min(CH, n_t - c0);
      if (G::NBUF == 2) {
        // this chunk landed at the end of the previous one; start the next
        // chunk's gathers and the order indices of the one after
        if (c0 + CH < n_t) issue(c0 + CH, buf ^ 1);
        if (c0 + 2 * CH < n_t) prefetch_order(c0 + 2 * CH);
      } else {
        issue(c0, 0);
        cp_async_wait_group<0>();
        __syncthreads();
      }
      float *stc = reinterpret_cast<float *>(s_stage + buf * G::stage0_bytes());
      float *s_x1 = stc, *s_x2 = stc + SP, *s_x3 = stc + 2 * SP;
      float *s_p1 = stc + 3 * SP, *s_p2 = stc + 4 * SP, *s_p3 = stc + 5 * SP;
      float *s_w = stc + 6 * SP;  // weight in, gamma out
      uint32_t *s_cell = reinterpret_cast<uint32_t *>(stc + 7 * SP);
      uint32_t *s_flag = reinterpret_cast<uint32_t *>(stc + 8 * SP);
      uint32_t *s_idx = reinterpret_cast<uint32_t *>(stc + 9 * SP);
      uint8_t *s_dm = reinterpret_cast<uint8_t *>(stc + 10 * SP);  // direction, mode << 4
      // 3b. push + deposit of one element. kAny: with the expressions for any
      // offset; without, for offsets in [0, 1] on grids of at most kExactCells
      // a side.
      auto particle = [&](auto any, const int e) {
        constexpr bool kAny = decltype(any)::value;
        const int s = spos(e);
        const uint32_t c = s_cell[s];
        const uint32_t flag = s_flag[s];
        const float x1 = s_x1[s], x2 = s_x2[s], x3 = s_x3[s];
        float p1 = s_p1[s], p2 = s_p2[s], p3 = s_p3[s];
        const float w = s_w[s];
        const int c2 = (int)__umul64hi((unsigned long long)c, P.m.div0);
        const int c1 = (int)c - c2 * dims0;
        uint32_t dir = 4;
        uint8_t mode = 0;
        const int lx = c1 - x0, ly = c2 - y0;  // within the tile
        const bool in_tile = c != AP_MAX_CELL && (unsigned)lx < (unsigned)TX &&
                             (unsigned)ly < (unsigned)TY;
        if (!in_tile) {
          atomicAdd(&P.status->tile_faults, 1ull);
          dir = kDirGone;
        } else if (p1 != p1 || p2 != p2 || p3 != p3) {
          // The reference traps here (ptc_updater.cu:102-109); the particle is
          // left untouched and reported instead.
          atomicAdd(&P.status->nan_momenta, 1ull);
        } else {
          const int sp = ptc_type(flag);
          float gamma = sqrtf(1.0f + p1 * p1 + p2 * p2 + p3 * p3);
          const bool em = !(flag & kFlagIgnoreEM);
          float v1, v2, v3;
          // log-spherical: r at the particle (user_push_2d_logsph.cuh:36)
          float r_push = 0.0f;
          if constexpr (kLS) r_push = expf(mesh_pos(P.m.lower[0], P.m.delta[0], c1, g0, x1));
          if (em) {
            const float qm = P.qm[sp];
            const Weights1D Wx = kLS ? weights_1d(x1, c1)
                                 : kAny ? weights_any(x1, c1) : weights_inside(x1, c1);
            const Weights1D Wy = kLS ? weights_1d(x2, c2)
                                 : kAny ? weights_any(x2, c2) : weights_inside(x2, c2);
            // each component: its four nodes in the reference's order, times
            // the x weight, then the y weight, added up from zero
            float fe[6];
            auto comp = [&](float2 r0, float2 r1, const float wx[2], const float wy[2]) {
              const float2 w = make_float2(wx[0], wx[1]);
              const float2 a = __fmul2_rn(__fmul2_rn(r0, w), make_float2(wy[0], wy[0]));
              const float2 b = __fmul2_rn(__fmul2_rn(r1, w), make_float2(wy[1], wy[1]));
              float acc = 0.0f;
              acc += a.x;
              acc += a.y;
              acc += b.x;
              acc += b.y;
              return acc * qm;
            };
            const int i0 = Wx.base0 - (x0 - 1), i1 = Wx.base1 - (x0 - 1);
            const int j0 = (Wy.base0 - ys) * G::RX, j1 = (Wy.base1 - ys) * G::RX;
            {
              const float4 r0 = sEB[j1 + i0], r1 = sEB[j1 + G::RX + i0];
              fe[0] = comp(make_float2(r0.x, r0.y), make_float2(r1.x, r1.y), Wx.w0, Wy.w1);
              fe[4] = comp(make_float2(r0.z, r0.w), make_float2(r1.z, r1.w), Wx.w0, Wy.w1);
            }
            {
              const float4 r0 = sEB[kNodes + j0 + i1], r1 = sEB[kNodes + j0 + G::RX + i1];
              fe[1] = comp(make_float2(r0.x, r0.y), make_float2(r1.x, r1.y), Wx.w1, Wy.w0);
              fe[3] = comp(make_float2(r0.z, r0.w), make_float2(r1.z, r1.w), Wx.w1, Wy.w0);
            }
            fe[2] = comp(sZ[j1 + i1], sZ[j1 + G::RX + i1], Wx.w1, Wy.w1);
            fe[5] = comp(sZ[kNodes + j0 + i0], sZ[kNodes + j0 + G::RX + i0], Wx.w0, Wy.w0);
            if constexpr (!kLS) {
              vay_push_v(p1, p2, p3, gamma, fe[0], fe[1], fe[2], fe[3], fe[4], fe[5], v1, v2, v3);
            } else {
              vay_push(p1, p2, p3, gamma, fe[0], fe[1], fe[2], fe[3], fe[4], fe[5]);
              // gravity (gravity.cuh:12-26), applied with strength
              // dev_params.gravity on every push, then sync_kill_perp
              // when radiative cooling is on and the particle is no ion.
              p1 -= P.dt * P.ls_gravity * P.mass[sp] / (r_push * r_push * fabsf(P.charge[sp]));
              gamma = sqrtf(1.0f + p1 * p1 + p2 * p2 + p3 * p3);
              if (gamma != gamma) atomicAdd(&P.status->nan_momenta, 1ull);
              if (P.ls_rad_on && sp != 2)
                sync_kill_perp(p1, p2, p3, gamma, fe[3], fe[4], fe[5], qm, P.ls_rad_coef,
                               P.ls_B0);
            }
          } else {
            gamma = P.p.E[s_idx[s]];  // the deposit reads the stored gamma
          }
          if (kLS || !em) {
            v1 = p1 / gamma;
            v2 = p2 / gamma;
            v3 = p3 / gamma;
          }
          float nx1, nx2, nx3;
          int dc1, dc2;
          if constexpr (!kLS) {
            // deposit_current_cart_2d (ptc_updater.cu:295-386)
            nx1 = x1 + (v1 * P.dt) * P.m.inv_delta[0];
            nx2 = x2 + (v2 * P.dt) * P.m.inv_delta[1];
            dc1 = (int)floorf(nx1);
            dc2 = (int)floorf(nx2);
            nx1 -= (float)dc1;
            nx2 -= (float)dc2;
            nx3 = x3 + v3 * P.dt;
          } else {
            // deposit_and_move_2d_log_sph (ptc_updater_logsph.cu:163-233):
            // move in Cartesian space, return to (ln r, theta, phi), rotate
            // the velocity into the new local basis, reflect at the axis.
            const float r1 = mesh_pos(P.m.lower[0], P.m.delta[0], c1, g0, x1);
            const float exp_r1 = expf(r1);
            const float r2 = mesh_pos(P.m.lower[1], P.m.delta[1], c2, g1, x2);
            const float2 sc2 = sin_cos_ool(r2), sc3 = sin_cos_ool(x3);
            v3 = v3 - beta_phi_s(P.ls_compactness, P.ls_omega, exp_r1, sc2.x);
            float x = exp_r1 * sc2.x * sc3.y;
            float y = exp_r1 * sc2.x * sc3.x;
            float z = exp_r1 * sc2.y;
            logsph2cart_sc(v1, v2, v3, sc2.y, sc2.x, sc3.y, sc3.x);
            x += 1.0f * v1 * P.dt;  // alpha_gr(r) = 1
            y += 1.0f * v2 * P.dt;
            z += 1.0f * v3 * P.dt;
            float r1p = sqrtf(x * x + y * y + z * z);
            const float r2p = acosf(z / r1p);
            const float exp_r1p = r1p;
            r1p = logf(r1p);
            const float r3p = atan2f(y, x);
            const float2 sp2 = sin_cos_ool(r2p), sp3 = sin_cos_ool(r3p);
            cart2logsph_sc(v1, v2, v3, sp2.y, sp2.x, sp3.y, sp3.x);
            p1 = v1 * gamma;
            p2 = v2 * gamma;
            p3 = (v3 + beta_phi_s(P.ls_compactness, P.ls_omega, exp_r1p, sp2.x)) * gamma;
            nx1 = x1 + (r1p - r1) / P.m.delta[0];
            nx2 = x2 + (r2p - r2) / P.m.delta[1];
            dc1 = (int)floorf(nx1);
            dc2 = (int)floorf(nx2);
            nx1 -= (float)dc1;
            nx2 -= (float)dc2;
            if (mesh_pos(P.m.lower[1], P.m.delta[1], c2 + dc2, g1, nx2) < 0.0f) {
              dc2 += 1;
              nx2 = 1.0f - nx2;
              p2 = -p2;
              p3 = -p3;
            }
            if ((double)mesh_pos(P.m.lower[1], P.m.delta[1], c2 + dc2, g1, nx2) >=
                3.14159265358979323846) {
              dc2 -= 1;
              nx2 = 1.0f - nx2;
              p2 = -p2;
              p3 = -p3;
            }
            nx3 = r3p;
          }
          const bool far = dc1 > 1 || dc1 < -1 || dc2 > 1 || dc2 < -1;

          if (!far && !(flag & kFlagIgnoreCurrent)) {
            if constexpr (!kLS) {
              // Esirkepov over the reference's ranges i in [i0, i1], j in [j0, j1]
              // (2 or 3 nodes per dim). Every lane walks the same 3 x 3 window
              // starting at (ib, jb) so the warp does not diverge; the third
              // node of a 2-node range is predicated off. The decomposition is
              // separable: with DX the cumulative sum of sx1 - sx0 along a row
              // and YM the mean of sy0 and sy1, J1 of the face after node a in
              // row b is -q w DX[a] YM[b]; J2 likewise; J3 is a sum of two
              // products. The face after the last node of a range is not
              // deposited: its cumulative sum covers the whole support (sum of
              // new weights minus sum of old weights), zero up to rounding.
              const float weight = -P.charge[sp] * w;
              // the factors carry 2^S (exact), so that a product is the scaled
              // contribution
              const float wsc = weight * fscale;
              const bool x3n = dc1 != 0, y3n = dc2 != 0;
              const int ib = (dc1 == -1 ? -2 : -1), jb = (dc2 == -1 ? -2 : -1);
              const Acc32 J1{sJhi, sJlo}, J2{sJhi + G::JSZ, sJlo + G::JSZ},
                  J3{sJhi + 2 * G::JSZ, sJlo + 2 * G::JSZ};
              const Acc32 R{sJhi + (3 + sp) * G::JSZ, sJlo + (3 + sp) * G::JSZ};
              const bool rho = kRho && P.do_rho && sp < P.num_species;
              const int o = (ly + jb + 2) * G::JX + (lx + ib + 2);
              if constexpr (!kAny) {
                // old weights 1 - x, x on the nodes -1, 0; new ones 1 - nx, nx
                // on -1 + dc, dc; the window starts at -2 for dc = -1, else -1
                float sx0[3], sx1[3], sy0[3], sy1[3];
                auto node_weights = [](float x, float nx, int dc, float s0[3], float s1[3]) {
                  const bool m = dc < 0, p = dc > 0;
                  const float r = 1.0f - x, nr = 1.0f - nx;
                  s0[0] = m ? 0.0f : r;
                  s0[1] = m ? r : x;
                  s0[2] = m ? x : 0.0f;
                  s1[0] = p ? 0.0f : nr;
                  s1[1] = p ? nr : nx;
                  s1[2] = p ? nx : 0.0f;
                };
                node_weights(x1, nx1, dc1, sx0, sx1);
                node_weights(x2, nx2, dc2, sy0, sy1);
                {
                  const float h = 0.5f * wsc;
                  // the cumulative sums from either end (the weights add up to 1)
                  const float d0 = sx1[0] - sx0[0], d1 = sx0[2] - sx1[2];
                  const float e0 = sy1[0] - sy0[0], e1 = sy0[2] - sy1[2];
                  const float dx[2] = {h * d0, h * d1}, dy[2] = {h * e0, h * e1};
#pragma unroll
                  for (int b = 0; b < 3; ++b) {
                    const float ym = sy0[b] + sy1[b], xm = sx0[b] + sx1[b];
                    const bool yv = b < 2 || y3n, xv = b < 2 || x3n;
                    if (yv) add_fixed_scaled(J1, o + b * G::JX + 1, dx[0] * ym, fx.L);
                    if (yv && x3n) add_fixed_scaled(J1, o + b * G::JX + 2, dx[1] * ym, fx.L);
                    if (xv) add_fixed_scaled(J2, o + G::JX + b, dy[0] * xm, fx.L);
                    if (xv && y3n) add_fixed_scaled(J2, o + 2 * G::JX + b, dy[1] * xm, fx.L);
                  }
                }
                const float k3 = -wsc * v3 * 0.1666667f;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                  const float c1w = k3 * (2.0f * sx1[a] + sx0[a]);
                  const float c0w = k3 * (sx1[a] + 2.0f * sx0[a]);
                  const float rw = -wsc * sx1[a];
#pragma unroll
                  for (int b = 0; b < 3; ++b) {
                    if ((a < 2 || x3n) && (b < 2 || y3n)) {
                      const int s3 = o + b * G::JX + a;
                      const float val = __fmaf_rn(c1w, sy1[b], c0w * sy0[b]);
                      add_fixed_scaled(J3, s3, val, fx.L);
                      if (rho) add_fixed_scaled(R, s3, rw * sy1[b], fx.L);
                    }
                  }
                }
              } else {
                // an offset outside [0, 1] (a particle its caller placed so, or
                // a NaN): the weights are the clamped ones of any offset, they
                // need not add up to 1, and every face of the range counts.
                // Once per particle: the move leaves offsets in [0, 1].
                const int nib = x3n ? 3 : 2, njb = y3n ? 3 : 2;
#pragma unroll 1
                for (int b = 0; b < njb; ++b) {
                  const float sy0 = cic(-x2 + (jb + b) + 1);
                  const float sy1 = cic(-nx2 + (jb + b + 1 - dc2));
                  float djx = 0.0f;
#pragma unroll 1
                  for (int a = 0; a < nib; ++a) {
                    const float sx0 = cic(-x1 + (ib + a) + 1);
                    const float sx1 = cic(-nx1 + (ib + a + 1 - dc1));
                    const int s3 = o + b * G::JX + a;
                    djx += movement2d(sy0, sy1, sx0, sx1);
                    add_fixed_scaled(J1, s3 + 1, wsc * djx, fx.L);
                    add_fixed_scaled(J3, s3, -wsc * v3 * center2d(sx0, sx1, sy0, sy1), fx.L);
                    if (rho) add_fixed_scaled(R, s3, -wsc * (sx1 * sy1), fx.L);
                  }
                }
#pragma unroll 1
                for (int a = 0; a < nib; ++a) {
                  const float sx0 = cic(-x1 + (ib + a) + 1);
                  const float sx1 = cic(-nx1 + (ib + a + 1 - dc1));
                  float djy = 0.0f;
#pragma unroll 1
                  for (int b = 0; b < njb; ++b) {
                    const float sy0 = cic(-x2 + (jb + b) + 1);
                    const float sy1 = cic(-nx2 + (jb + b + 1 - dc2));
                    djy += movement2d(sx0, sx1, sy0, sy1);
                    add_fixed_scaled(J2, o + (b + 1) * G::JX + a, wsc * djy, fx.L);
                  }
                }
              }
            } else {
              // Esirkepov over the reference's ranges i in [i0, i1], j in [j0, j1]
              // (2 or 3 nodes per dim). Every lane walks the same 3 x 3 window
              // starting at (ib, jb) so the warp does not diverge; the third
              // node of a 2-node range is predicated off. Cumulative sums run
              // in the reference's order, so each contribution keeps its value.
              // The third column of J1 and the third row of J2 are only ever the
              // last node of a 3-node range, where the cumulative sum covers the
              // whole support (sum of new weights minus sum of old weights,
              // zero up to rounding); the reference adds that rounding residue,
              // these sites are skipped.
              const float weight = -P.charge[sp] * w;
              // the deposit's factors pre-scaled by 2^S (exact): weight, and
              // -weight * v3 as the reference forms it before the site loop
              const float wsc = weight * fscale;
              const float w3s = -wsc * v3;
              const int ib = (dc1 == -1 ? -2 : -1), nib = (dc1 == 0 ? 2 : 3);
              const int jb = (dc2 == -1 ? -2 : -1), njb = (dc2 == 0 ? 2 : 3);
              float sx0[3], sx1[3];
#pragma unroll
              for (int a = 0; a < 3; ++a) {
                const int i = ib + a;
                sx0[a] = cic(-x1 + i + 1);
                sx1[a] = cic(-nx1 + (i + 1 - dc1));
              }
              float djy[3] = {0.0f, 0.0f, 0.0f};
              const Acc32 J1{sJhi, sJlo}, J2{sJhi + G::JSZ, sJlo + G::JSZ},
                  J3{sJhi + 2 * G::JSZ, sJlo + 2 * G::JSZ};
              const Acc32 R{sJhi + (3 + sp) * G::JSZ, sJlo + (3 + sp) * G::JSZ};
              const bool rho = kRho && P.do_rho && sp < P.num_species;
              const int obase = (c2 + jb - jy0) * G::JX + (c1 + ib - jx0);
#pragma unroll
              for (int b = 0; b < 3; ++b) {
                const int j = jb + b;
                const bool jv = b < njb;
                const float sy0 = cic(-x2 + j + 1);
                const float sy1 = cic(-nx2 + (j + 1 - dc2));
                float djx = 0.0f;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                  if (jv && a < nib) {
                    const int o = obase + b * G::JX + a;
                    djx += movement2d(sy0, sy1, sx0[a], sx1[a]);
                    if (a < 2) add_fixed_scaled(J1, o + 1, wsc * djx, fx.L);
                    djy[a] += movement2d(sx0[a], sx1[a], sy0, sy1);
                    if (b < 2) add_fixed_scaled(J2, o + G::JX, wsc * djy[a], fx.L);
                    const float val2 = center2d(sx0[a], sx1[a], sy0, sy1);
                    add_fixed_scaled(J3, o, w3s * val2 / s_dv[o], fx.L);
                    if (rho) {
                      const float s1 = sx1[a] * sy1;
                      add_fixed_scaled(R, o, -wsc * s1, fx.L);
                    }
                  }
                }
              }
            }
          }
          // move + wrap through periodic sides (send_particles semantics)
          int c1n = c1 + dc1, c2n = c2 + dc2;
          // past the upper end of the bulk: the next tile, also from a tile
          // that the end cuts short
          const bool over1 = c1n >= dims0 - g0, over2 = c2n >= dims1 - g1;
          bool keep = !far;
          keep = keep && wrap_coord(c1n, g0, dims0, P.m.red[0], P.periodic[0]);
          keep = keep && wrap_coord(c2n, g1, dims1, P.m.red[1], P.periodic[1]);
          uint32_t ncell = AP_MAX_CELL;
          if (keep) {
            ncell = (uint32_t)(c1n + c2n * dims0);
            const int dtx = lx + dc1 < 0 ? 0 : (lx + dc1 >= TX || over1 ? 2 : 1);
            const int dty = ly + dc2 < 0 ? 0 : (ly + dc2 >= TY || over2 ? 6 : 3);
            dir = (uint32_t)(dty + dtx);
            if constexpr (kLS) {
              // ptc_outflow (ptc_updater_logsph.cu:440-455)
              if (!(flag & kFlagIgnoreEM) && c1n > P.ls_outflow_c1) {
                s_flag[s] = flag | kFlagIgnoreEM;
                mode |= kWriteFlag;
              }
            }
          } else {
            dir = kDirGone;
            if (far)
              atomicAdd(&P.status->moved_far, 1ull);
            else
              atomicAdd(&P.status->lost, 1ull);
          }
          s_x1[s] = nx1;
          s_x2[s] = nx2;
          s_x3[s] = nx3;
          s_cell[s] = ncell;
          mode |= kWritePos;
          if (em || kLS) {
            s_p1[s] = p1;
            s_p2[s] = p2;
            s_p3[s] = p3;
            s_w[s] = gamma;
            mode |= kWriteMom;
          }
        }
        s_dm[s] = (uint8_t)(dir | (uint32_t)mode << 4);
        // direction counts: one add per warp for the particles that stay in
        // the tile (nearly all), one per particle for the rest
        const unsigned act = __activemask();
        const unsigned stay = __ballot_sync(act, dir == 4u);
        if (lane == __ffs(act) - 1) atomicAdd(&s_cnt[4], (uint32_t)__popc(stay));
        if (dir != 4u) atomicAdd(&s_cnt[dir], 1u);
      };
      // lane l of warp w takes element l*CH/32 + w*PER_THREAD + k. Offsets
      // outside [0, 1] (particles their caller placed so, once: the move leaves
      // offsets inside) are left to a second walk: in branches of the first one
      // their expressions cost every particle (512^2 x 32: 441 us per update
      // without them, 445 with those of the deposit in a branch, 450 with those
      // of the weights too, 444 so).
      bool rest = false;
      for (int k = 0; k < PER_THREAD; ++k) {
        const int e = lane * (CH / 32) + warp * PER_THREAD + k;
        if (e >= nch) continue;
        if (kLS || (exact_grid && offsets_inside(s_x1[spos(e)], s_x2[spos(e)]))) {
          particle(std::false_type{}, e);
        } else {
          s_dm[spos(e)] = kLeft;
          rest = true;
        }
      }
      if constexpr (kLS) {
        __syncthreads();
      } else if (__syncthreads_or(rest)) {
        for (int k = 0; k < PER_THREAD; ++k) {
          const int e = lane * (CH / 32) + warp * PER_THREAD + k;
          if (e < nch && s_dm[spos(e)] == kLeft) particle(std::true_type{}, e);
        }
        __syncthreads();
      }
      // direction counts of this chunk, for the one-pass order update
      if (P.chunk_count && tid < 10) {
        const uint32_t v = s_cnt[tid];
        P.chunk_count[((size_t)(base / CH + t) + c0 / CH) * 10 + tid] = v - cnt_prev;
        cnt_prev = v;
      }
      // 3c. coalesced write-back of the chunk
#pragma unroll
      for (int k = 0; k < PER_THREAD; ++k) {
        const int e = tid + k * kThreads2D;
        if (e < nch) {
          const int s = spos(e);
          const uint32_t dm = s_dm[s], mode = dm >> 4;
          const uint32_t idx = s_idx[s];
          if (P.cout.x1) {
            // compaction: every member to its tile-list position
            const size_t q = base + c0 + e;
            P.cout.x1[q] = s_x1[s];
            P.cout.x2[q] = s_x2[s];
            P.cout.x3[q] = s_x3[s];
            P.cout.p1[q] = s_p1[s];
            P.cout.p2[q] = s_p2[s];
            P.cout.p3[q] = s_p3[s];
            P.cout.E[q] = (mode & kWriteMom) ? s_w[s] : P.p.E[idx];
            P.cout.w[q] = P.p.w[idx];
            P.cout.cell[q] = s_cell[s];
            P.cout.flag[q] = s_flag[s];
            P.cout_id[q] = P.id[idx];
            P.dir[base + c0 + e] = (uint8_t)(dm & 15u);
            continue;
          }
          if (mode & kWritePos) {
            P.p.x1[idx] = s_x1[s];
            P.p.x2[idx] = s_x2[s];
            P.p.x3[idx] = s_x3[s];
            P.p.cell[idx] = s_cell[s];
          }
          if (mode & kWriteMom) {
            P.p.p1[idx] = s_p1[s];
            P.p.p2[idx] = s_p2[s];
            P.p.p3[idx] = s_p3[s];
            P.p.E[idx] = s_w[s];
          }
          if (kLS && (mode & kWriteFlag)) P.p.flag[idx] = s_flag[s];
          P.dir[base + c0 + e] = (uint8_t)(dm & 15u);
        }
      }
      if (G::NBUF == 2) cp_async_wait_group<0>();  // the next chunk and order indices
      __syncthreads();
      if (G::NBUF == 2) buf ^= 1;
    }

    // 4. flush the current (and charge) tile once
    for (int i = tid; i < nacc; i += kThreads2D) {
      const long long v = fixed_total(sJhi[i], sJlo[i], fx.L);
      if (v == 0) continue;
      const int comp = i / G::JSZ, rem = i % G::JSZ;
      const int gx = jx0 + rem % G::JX, gy = jy0 + rem / G::JX;
      if (gx >= dims0 || gy >= dims1) continue;
      atomicAdd(P.acc + comp * P.acc_comp + (size_t)gy * P.acc_pitch + gx,
                (unsigned long long)v);
    }
    // the tile's other items add to the same counts, which start at 0
    if (tid < 10 && s_cnt[tid]) atomicAdd(&P.dir_count[t * 10 + tid], s_cnt[tid]);
    phase ^= 1u;
  }
}

template <int TX, int TY, int CH, int MINB, bool kTMA, bool kRho, bool kLS>
__global__ void __launch_bounds__(kThreads2D, MINB)
    k_push_deposit_2d(const __grid_constant__ PushDepositParams P,
                      const __grid_constant__ FieldMaps maps) {
  push_deposit_tiles<TX, TY, CH, kTMA, kRho, kLS, false>(P, maps.m, nullptr, nullptr, 0, P.queue);
}

// Many independent Cartesian runs in one persistent launch: CTAs take work
// items (a tile's list of one run, or a part of it) from one queue over all
// runs' items.
template <int TX, int TY, int CH, int MINB, bool kTMA, bool kRho>
__global__ void __launch_bounds__(kThreads2D, MINB)
    k_push_deposit_2d_batch(const RunDesc *__restrict__ runs, const uint32_t *__restrict__ base,
                            int nruns, uint32_t *queue) {
  push_deposit_tiles<TX, TY, CH, kTMA, kRho, false, true>(runs[0].P, nullptr, runs, base, nruns,
                                                           queue);
}

// ---------------------------------------------------------------------------
// Self-test of the bounded wait: an mbarrier that announces bytes no copy
// will bring is waited on with the field-tile wait above; the give-up is
// recorded as a timeout in the status word. No asynchronous copy is
// issued, so nothing is left in flight when the kernel returns.
__global__ void k_selftest_wait(DevStatus *status, uint32_t limit) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_expect_tx(&bar, 64u);
    if (!mbar_wait(&bar, 0u, limit)) atomicAdd(&status->timeouts, 1ull);
  }
}

// 1D: the whole line is small, so each CTA takes a contiguous chunk of
// particle slots, finds the cell range it touches, and deposits into a
// shared-memory window over that range (or straight to the global
// accumulators when the window would not fit). Fields are read through the
// read-only cache.

constexpr int kThreads1D = 256;
constexpr int kItems1D = 8;
constexpr int kChunk1D = kThreads1D * kItems1D;  // 2048 particles
constexpr int kWin1D = 6000;                     // cell-components per window

__device__ __forceinline__ float interp_1d_global(const FieldArr &f, const Weights1D &W,
                                                  int stag) {
  const int b = stag ? W.base1 : W.base0;
  const float w0 = stag ? W.w1[0] : W.w0[0];
  const float w1 = stag ? W.w1[1] : W.w0[1];
  float acc = 0.0f;
  acc += __ldg(f.ptr + b) * w0;
  acc += __ldg(f.ptr + b + 1) * w1;
  return acc;
}

// Warp-collective deposit of a warp's particles into the 1D window. In a
// cell-sorted run neighbouring lanes hold particles of the same cell, so their
// atomics would all hit one address: when the lanes touch at most kAgg1D
// distinct first nodes, each node's fixed-point words are summed across the
// lanes that share it (integer sums, so the result is the same bits) and one
// lane adds them; a few active lanes, and nodes of many cells, add directly.
constexpr int kAgg1D = 4;

// The lanes that share a first node: found once per particle for its two or
// three nodes.
struct Groups1D {
  unsigned leaders;  // lowest lane of each group
  bool few;          // at most kAgg1D groups
};

__device__ __forceinline__ Groups1D groups_1d(bool act, int o) {
  const int lane = threadIdx.x & 31;
  const unsigned key = act ? (unsigned)o : (0x80000000u | (unsigned)lane);
  const unsigned peers = __match_any_sync(0xffffffffu, key);
  Groups1D g;
  g.leaders = __ballot_sync(0xffffffffu, act && lane == __ffs(peers) - 1);
  g.few = __popc(g.leaders) <= kAgg1D;
  return g;
}

// One node (every lane of the warp calls it): `act` lanes contribute a1 to J1
// at window offset o + 1 and a2, a3 to J2, J3 at o; g groups the offsets.
__device__ __forceinline__ void deposit_1d_node(const Groups1D &g, bool act, int o, float a1,
                                                float a2, float a3, int *hi, unsigned *lo,
                                                int win_comp, float scale, int L) {
  const unsigned am = __ballot_sync(0xffffffffu, act);
  if (am == 0u) return;
  const int lane = threadIdx.x & 31;
  const unsigned mask = (1u << L) - 1u;
  unsigned h[3], l[3];
  const float a[3] = {a1, a2, a3};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const long long X = act ? __float2ll_rn(a[c] * scale) : 0ll;  // exact scaling
    h[c] = (unsigned)(int)(X >> L);
    l[c] = (unsigned)X & mask;
  }
  const int dst[3] = {o + 1, win_comp + o, 2 * win_comp + o};
  if (g.few && __popc(am) > kAgg1D) {
    for (unsigned m = g.leaders; m != 0u; m &= m - 1u) {
      const int ld = __ffs(m) - 1;
      const int ko = __shfl_sync(0xffffffffu, o, ld);  // every lane takes part
      const bool in = act && o == ko;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const unsigned sh = __reduce_add_sync(0xffffffffu, in ? h[c] : 0u);
        const unsigned sl = __reduce_add_sync(0xffffffffu, in ? l[c] : 0u);
        if (lane == ld) {
          atomicAdd(hi + dst[c], (int)sh);
          atomicAdd(lo + dst[c], sl);
        }
      }
    }
  } else if (act) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      atomicAdd(hi + dst[c], (int)h[c]);
      atomicAdd(lo + dst[c], l[c]);
    }
  }
}

// One chunk of kThreads1D * kItems particle slots of a 1D run: push, deposit
// into a shared-memory window over the cells the chunk touches (or straight
// into the global accumulators when the window would not fit), move.
template <bool kRho, int kItems = kItems1D>
__device__ __forceinline__ void push_deposit_1d_chunk(const PushDepositParams &P, size_t ch,
                                                      int *sWhi, unsigned *sWlo, int &s_lo,
                                                      int &s_hi) {
  const int tid = threadIdx.x;
  const int n0 = P.m.dims[0], g0 = P.m.guard[0];
  const int ncomp = 3 + (kRho ? P.num_species : 0);
  const int win_comp = kWin1D / ncomp;
  // A window sums at most kChunk1D contributions per cell; the global
  // accumulators at most `number`.
  const int lgw = bits_of(kChunk1D);
  const size_t number = P.d_number ? (size_t)*P.d_number : P.number;
  const int lgn = bits_of((uint32_t)min(number, (size_t)0x7fffffff));
  const FixedFmt fx = fixed_format(lgw, min(63 - 2 * lgw, 62 - lgn), P.qmax * *P.wmax);
  const float fscale = ldexpf(1.0f, fx.S);
  if (ch == 0 && tid == 0) *P.fx_used = fx;
  const size_t first = ch * (size_t)(kThreads1D * kItems);
  if (tid == 0) {
    s_lo = INT_MAX;
    s_hi = INT_MIN;
  }
  __syncthreads();
  uint32_t cells[kItems];
  int lo = INT_MAX, hi = INT_MIN;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    const size_t idx = first + (size_t)k * kThreads1D + tid;
    cells[k] = idx < number ? P.p.cell[idx] : AP_MAX_CELL;
    if (cells[k] != AP_MAX_CELL) {
      lo = min(lo, (int)cells[k]);
      hi = max(hi, (int)cells[k]);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((tid & 31) == 0 && lo <= hi) {
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
  }
  __syncthreads();
  const int wlo = s_lo - 2;
  const int wlen = s_hi - s_lo + 5;
  const bool use_smem = (s_lo <= s_hi) && wlen <= win_comp;
  if (use_smem)
    for (int i = tid; i < ncomp * wlen; i += kThreads1D) {
      const int si = (i / wlen) * win_comp + i % wlen;
      sWhi[si] = 0;
      sWlo[si] = 0u;
    }
  __syncthreads();

  // The members of item k + 1 are loaded while item k is pushed and
  // deposited (the items of one thread are distinct slots).
  struct Item1D {
    uint32_t flag;
    float x1, x2, x3, p1, p2, p3, w;
  };
  auto load_item = [&](int k, Item1D &it) {
    const uint32_t c = cells[k];
    if (c == AP_MAX_CELL || (int)c < g0 || (int)c >= n0 - g0) return;
    const size_t idx = first + (size_t)k * kThreads1D + tid;
    it.flag = P.p.flag[idx];
    it.x1 = P.p.x1[idx];
    it.x2 = P.p.x2[idx];
    it.x3 = P.p.x3[idx];
    it.p1 = P.p.p1[idx];
    it.p2 = P.p.p2[idx];
    it.p3 = P.p.p3[idx];
    it.w = P.p.w[idx];
  };
  Item1D cur{}, nxt{};
  load_item(0, cur);
#pragma unroll 1
  for (int k = 0; k < kItems; ++k) {
    if (k + 1 < kItems) load_item(k + 1, nxt);
    // deposit inputs of this item; the deposit runs after the item, with
    // every lane of the warp present
    bool dep = false;
    float d_x1 = 0.0f, d_nx1 = 0.0f, d_w = 0.0f, d_v2 = 0.0f, d_v3 = 0.0f;
    int d_c1 = 0, d_dc1 = 0, d_sp = 0;
    do {  // one item; `break` skips to the next
    const size_t idx = first + (size_t)k * kThreads1D + tid;
    uint32_t c = cells[k];
    if (c == AP_MAX_CELL) break;
    if ((int)c < g0 || (int)c >= n0 - g0) {  // ptc_updater.cu:30-33
      P.p.cell[idx] = AP_MAX_CELL;
      break;
    }
    const uint32_t flag = cur.flag;
    float x1 = cur.x1;
    float p1 = cur.p1, p2 = cur.p2, p3 = cur.p3;
    if (p1 != p1 || p2 != p2 || p3 != p3) {
      atomicAdd(&P.status->nan_momenta, 1ull);
      break;
    }
    const int sp = ptc_type(flag);
    const int c1 = (int)c;
    float gamma = sqrtf(1.0f + p1 * p1 + p2 * p2 + p3 * p3);
    const bool em = !(flag & kFlagIgnoreEM);
    float v1, v2, v3;
    if (em) {
      // ptc_push_cart_1d (ptc_updater.cu:21-76): only the x stagger bit
      // matters in 1D.
      const float qm = P.qm[sp];
      const Weights1D W = weights_1d(x1, c1);
      float fe[6];
#pragma unroll
      for (int q = 0; q < 6; ++q) fe[q] = interp_1d_global(P.F[q], W, stag_x(q)) * qm;
      vay_push_v(p1, p2, p3, gamma, fe[0], fe[1], fe[2], fe[3], fe[4], fe[5], v1, v2, v3);
      P.p.p1[idx] = p1;
      P.p.p2[idx] = p2;
      P.p.p3[idx] = p3;
      P.p.E[idx] = gamma;
    } else {
      gamma = P.p.E[idx];
      v1 = p1 / gamma;
      v2 = p2 / gamma;
      v3 = p3 / gamma;
    }
    // deposit_current_cart_1d (ptc_updater.cu:220-293)
    const float w = cur.w;
    const float x2 = cur.x2, x3 = cur.x3;
    float nx1 = x1 + (v1 * P.dt) / P.m.delta[0];
    const int dc1 = (int)floorf(nx1);
    nx1 -= (float)dc1;
    const bool far = dc1 > 1 || dc1 < -1;
    P.p.x1[idx] = nx1;
    P.p.x2[idx] = x2 + v2 * P.dt;
    P.p.x3[idx] = x3 + v3 * P.dt;
    if (!far && !(flag & kFlagIgnoreCurrent)) {
      dep = true;
      d_x1 = x1;
      d_nx1 = nx1;
      d_w = P.charge[sp] * w;
      d_v2 = v2;
      d_v3 = v3;
      d_c1 = c1;
      d_dc1 = dc1;
      d_sp = sp;
    }
    int cn = c1 + dc1;
    bool keep = !far && wrap_coord(cn, g0, n0, P.m.red[0], P.periodic[0]);
    if (!keep) atomicAdd(far ? &P.status->moved_far : &P.status->lost, 1ull);
    P.p.cell[idx] = keep ? (uint32_t)cn : AP_MAX_CELL;
    } while (false);
    {
      const float weight = d_w;
      // the reference's node range [i0, i1] has 2 or 3 nodes; every lane
      // walks three node slots i0, i0 + 1, i0 + 2 (the third active only for
      // a cell crossing), in the reference's order
      const int i0 = (d_dc1 == -1 ? -2 : -1), i1 = (d_dc1 == 1 ? 1 : 0);
      float djx = 0.0f;
      const Groups1D groups = groups_1d(dep, i0 + d_c1 - wlo);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int i = i0 + j;
        const bool act = dep && i <= i1;
        float sx1 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
        const int off = i + d_c1;
        if (act) {
          const float sx0 = cic(-d_x1 + i + 1);
          sx1 = cic(-d_nx1 + (i + 1 - d_dc1));
          djx += sx1 - sx0;
          a1 = -weight * djx;
          const float val1 = 0.5f * (sx0 + sx1);
          a2 = weight * d_v2 * val1;
          a3 = weight * d_v3 * val1;
        }
        if (use_smem) {
          deposit_1d_node(groups, act, off - wlo, a1, a2, a3, sWhi, sWlo, win_comp, fscale,
                          fx.L);
          if (act && kRho && P.do_rho && d_sp < P.num_species) {
            const Acc32 W{sWhi, sWlo};
            add_fixed(W, (3 + d_sp) * win_comp + off - wlo, weight * sx1, fscale, fx.L);
          }
        } else if (act) {
          auto gadd = [&](int k2, int x, float v) {
            atomicAdd(P.acc + k2 * P.acc_comp + x,
                      (unsigned long long)__float2ll_rn(v * fscale));
          };
          gadd(0, off + 1, a1);
          gadd(1, off, a2);
          gadd(2, off, a3);
          if (kRho && P.do_rho && d_sp < P.num_species) gadd(3 + d_sp, off, weight * sx1);
        }
      }
    }
    cur = nxt;
  }
  __syncthreads();
  if (use_smem) {
    for (int i = tid; i < ncomp * wlen; i += kThreads1D) {
      const int comp = i / wlen, o = i % wlen;
      const int si = comp * win_comp + o;
      const long long v = (long long)sWhi[si] * (1ll << fx.L) + (long long)sWlo[si];
      if (v == 0) continue;
      const int gx = wlo + o;
      if (gx < 0 || gx >= n0) continue;
      atomicAdd(P.acc + comp * P.acc_comp + gx, (unsigned long long)v);
    }
  }
  __syncthreads();
}

template <bool kRho, int kItems>
__global__ void __launch_bounds__(kThreads1D)
    k_push_deposit_1d(const __grid_constant__ PushDepositParams P) {
  __shared__ int sWhi[kWin1D];
  __shared__ unsigned sWlo[kWin1D];
  __shared__ int s_lo, s_hi;
  constexpr size_t kChunk = kThreads1D * kItems;
  const size_t nchunks = (P.number + kChunk - 1) / kChunk;
  for (size_t ch = blockIdx.x; ch < nchunks; ch += gridDim.x)
    push_deposit_1d_chunk<kRho, kItems>(P, ch, sWhi, sWlo, s_lo, s_hi);
}

// Many independent 1D runs in one launch: work item g is chunk
// g - base[r] of run r; the CTA copies that run's parameters into shared
// memory before the chunk.
template <bool kRho>
__global__ void __launch_bounds__(kThreads1D)
    k_push_deposit_1d_batch(const RunDesc *__restrict__ runs, const uint32_t *__restrict__ base,
                            int nruns) {
  __shared__ int sWhi[kWin1D];
  __shared__ unsigned sWlo[kWin1D];
  __shared__ int s_lo, s_hi;
  __shared__ __align__(16) uint32_t s_pbuf[sizeof(PushDepositParams) / 4];
  const uint32_t total = base[nruns];
  const PushDepositParams &P = *reinterpret_cast<const PushDepositParams *>(s_pbuf);
  for (uint32_t g = blockIdx.x; g < total; g += gridDim.x) {
    int lo = 0, hi = nruns - 1;  // largest r with base[r] <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (base[mid] <= g) lo = mid;
      else hi = mid - 1;
    }
    __syncthreads();  // the previous chunk is done with s_pbuf
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&runs[lo].P);
    for (int i = threadIdx.x; i < (int)(sizeof(PushDepositParams) / 4); i += kThreads1D)
      s_pbuf[i] = src[i];
    __syncthreads();
    push_deposit_1d_chunk<kRho>(P, g - base[lo], sWhi, sWlo, s_lo, s_hi);
  }
}

template <int TX, int TY, int CH, int MINB, bool kLS = false>
cudaError_t launch_2d_tiles(Ctx &c, const PushDepositParams &P) {
  using G = TileGeom<TX, TY, CH>;
  const int nrho = P.do_rho ? P.num_species : 0;
  const size_t smem = G::smem_bytes(nrho, kLS);  // the queue was cleared with the status
  auto run = [&](auto kern) -> cudaError_t {
    // blocks per SM of the variant, asked for when the context's variant changes
    if (c.pd_kern != reinterpret_cast<const void *>(kern) || c.pd_smem != smem) {
      cudaError_t err = G::allow_smem(kern);
      if (err != cudaSuccess) return err;
      int per_sm = 0;
      err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads2D, smem);
      if (err != cudaSuccess) return err;
      if (per_sm < 1) return cudaErrorInvalidConfiguration;
      c.pd_kern = reinterpret_cast<const void *>(kern);
      c.pd_smem = smem;
      c.pd_per_sm = per_sm;
    }
    size_t grid = (size_t)c.num_sms * c.pd_per_sm;
    const size_t items = P.t.ntiles + (c.number - c.store_base) / c.item_len;  // at most
    if (grid > items) grid = items;
    if (grid < 1) grid = 1;
    kern<<<(int)grid, kThreads2D, smem, c.stream>>>(P, c.maps);
    c.launches++;
    return cudaGetLastError();
  };
  if (c.use_tma) {
    return P.do_rho ? run(k_push_deposit_2d<TX, TY, CH, MINB, true, true, kLS>)
                    : run(k_push_deposit_2d<TX, TY, CH, MINB, true, false, kLS>);
  }
  return P.do_rho ? run(k_push_deposit_2d<TX, TY, CH, MINB, false, true, kLS>)
                  : run(k_push_deposit_2d<TX, TY, CH, MINB, false, false, kLS>);
}

// Staged chunks of 256 particles, double-buffered, with four CTAs per SM
// (default: 64 registers, no spills; the order indices run two chunks ahead
// and the gathers one chunk ahead, so no global load is waited on inside a
// tile; measured 3 % faster than 512 single-buffered on the 1024^2 box),
// 512 single-buffered with four, 1024 with three, 2048 with two.
template <int TX, int TY>
cudaError_t launch_2d_chunk(Ctx &c, const PushDepositParams &P) {
  // log-spherical: the pipelined 256-particle chunk with three CTAs per SM
  // (64 registers, no spills; the transcendental move makes it the slower
  // kernel, so a third CTA per SM pays: 0.355 ms against 0.476 ms for
  // single-buffered 1024-particle chunks on the pulsar grid)
  if (c.coord == 1) return launch_2d_tiles<TX, TY, 256, 3, true>(c, P);
  switch (chunk_of(c)) {
    case 2048: return launch_2d_tiles<TX, TY, 2048, 2>(c, P);
    case 1024: return launch_2d_tiles<TX, TY, 1024, 3>(c, P);
    case 512: return launch_2d_tiles<TX, TY, 512, 4>(c, P);
    default: return launch_2d_tiles<TX, TY, 256, 4>(c, P);
  }
}

// Largest |weight| over slots [0, n) (non-negative floats order like their
// bit patterns).
__global__ void k_weight_max(const float *w, const uint32_t *cell, size_t n, float *out) {
  float mx = 0.0f;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    if (cell[i] != AP_MAX_CELL) mx = fmaxf(mx, fabsf(w[i]));
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0)
    atomicMax(reinterpret_cast<unsigned int *>(out), __float_as_uint(mx));
}

}  // namespace

// Recomputes the largest particle weight (after the caller changed particles).
cudaError_t launch_fixed_scale(Ctx &c) {
  cudaError_t e = cudaMemsetAsync(c.wmax, 0, sizeof(float), c.stream);
  if (e != cudaSuccess) return e;
  if (c.number > 0) {
    size_t g = (c.number + 255) / 256;
    if (g > (size_t)c.num_sms * 8) g = (size_t)c.num_sms * 8;
    k_weight_max<<<(int)g, 256, 0, c.stream>>>(c.ptc.weight, c.ptc.cell, c.number, c.wmax);
    c.launches++;
  }
  c.scale_valid = true;
  return cudaGetLastError();
}

namespace {

template <int TX, int TY>
size_t cta_bytes(int chunk, int nrho) {
  const size_t dyn = chunk == 2048   ? TileGeom<TX, TY, 2048>::smem_bytes(nrho)
                     : chunk == 1024 ? TileGeom<TX, TY, 1024>::smem_bytes(nrho)
                     : chunk == 512  ? TileGeom<TX, TY, 512>::smem_bytes(nrho)
                                     : TileGeom<TX, TY, 256>::smem_bytes(nrho);
  return dyn + sizeof(PushDepositParams);  // a batch's copy of the parameters
}

}  // namespace

// The configured chunk while the current and charge tiles of all species leave
// room for a second CTA on the SM (228 KB, 1 KB reserved per CTA), else the
// next shorter one that does (512 for 256, whose two buffers take more). Alone
// on its SM a CTA has nothing to hide its barriers behind: 512^2 cells x 32
// particles with charges, us per update, one CTA and by this rule (and before
// the field records, which take the room, two CTAs): 16x16/2048 with 2 species
// 985, 574 (764); 16x8/2048 with 8 species 1049, 604 (797); 32x16/1024 with 6
// 1007, 722 (788); 32x16/256 with 8 927, 726 (764); 32x16/2048 with 2 966, 674
// (1056, one CTA then too). Three CTAs in place of four, and two in place of
// three, cost less than the records give: 16x16/256 with 3 species 523 (600),
// 32x16/256 with 2 611 (712), 16x16/1024 with 3 636 (672).
int chunk_of(const Ctx &c) {
  if (c.coord == 1) return kMinChunk;
  const int want = c.params.chunk == 512 || c.params.chunk == 1024 || c.params.chunk == 2048
                       ? c.params.chunk : kMinChunk;
  const int tx = c.tiles.tx, ty = c.tiles.ty, ns = c.params.num_species;
  const int tries[3] = {want, 1024, 512};
  for (int ch : tries) {
    if (ch > want && ch != 512) continue;
    const size_t bytes = tx == 32 ? cta_bytes<32, 16>(ch, ns)
                         : ty == 16 ? cta_bytes<16, 16>(ch, ns)
                         : tx == 16 ? cta_bytes<16, 8>(ch, ns)
                         : tx == 8 ? cta_bytes<8, 8>(ch, ns) : cta_bytes<4, 4>(ch, ns);
    if (2 * (bytes + 1024) <= 228 * 1024) return ch;
  }
  return want;
}

cudaError_t launch_push_deposit_2d(Ctx &c, const PushDepositParams &P) {
  const int tx = P.t.tx, ty = P.t.ty;
  if (tx == 16 && ty == 16) return launch_2d_chunk<16, 16>(c, P);
  if (tx == 32 && ty == 16) return launch_2d_chunk<32, 16>(c, P);
  if (tx == 8 && ty == 8) return launch_2d_chunk<8, 8>(c, P);
  if (tx == 16 && ty == 8) return launch_2d_chunk<16, 8>(c, P);
  if (tx == 4 && ty == 4) return launch_2d_chunk<4, 4>(c, P);
  return cudaErrorInvalidValue;
}

namespace {

// First item of each run in the batch's queue, from the runs' item counts (one
// warp); the queue starts at 0.
__global__ void k_batch_bases(const RunDesc *__restrict__ runs, int nruns, uint32_t *base,
                              uint32_t *queue) {
  const int lane = threadIdx.x;
  uint32_t carry = 0;
  for (int r0 = 0; r0 < nruns; r0 += 32) {
    const int r = r0 + lane;
    const uint32_t own = r < nruns ? *runs[r].P.n_items : 0u;
    uint32_t inc = own;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (r < nruns) base[r] = carry + inc - own;
    carry += __shfl_sync(0xffffffffu, inc, 31);
  }
  if (lane == 0) {
    base[nruns] = carry;
    *queue = 0u;
  }
}

template <int TX, int TY, int CH, int MINB>
cudaError_t launch_batch_tiles(cudaStream_t stream, int num_sms, bool tma, bool do_rho,
                               int max_species, const RunDesc *runs, uint32_t *base,
                               int nruns, uint32_t total, uint32_t *queue) {
  using G = TileGeom<TX, TY, CH>;
  const size_t smem = G::smem_bytes(do_rho ? max_species : 0);
  k_batch_bases<<<1, 32, 0, stream>>>(runs, nruns, base, queue);
  auto run = [&](auto kern) -> cudaError_t {
    cudaError_t err = G::allow_smem(kern);
    if (err != cudaSuccess) return err;
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads2D, smem);
    if (err != cudaSuccess) return err;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    uint32_t grid = (uint32_t)num_sms * per_sm;
    if (grid > total) grid = total;
    if (grid < 1) grid = 1;
    kern<<<grid, kThreads2D, smem, stream>>>(runs, base, nruns, queue);
    return cudaGetLastError();
  };
  if (tma)
    return do_rho ? run(k_push_deposit_2d_batch<TX, TY, CH, MINB, true, true>)
                  : run(k_push_deposit_2d_batch<TX, TY, CH, MINB, true, false>);
  return do_rho ? run(k_push_deposit_2d_batch<TX, TY, CH, MINB, false, true>)
                : run(k_push_deposit_2d_batch<TX, TY, CH, MINB, false, false>);
}

template <int TX, int TY>
cudaError_t launch_batch_chunk(cudaStream_t stream, int num_sms, int chunk, bool tma,
                               bool do_rho, int max_species, const RunDesc *runs,
                               uint32_t *base, int nruns, uint32_t total,
                               uint32_t *queue) {
  if (chunk == 2048)
    return launch_batch_tiles<TX, TY, 2048, 2>(stream, num_sms, tma, do_rho, max_species, runs,
                                               base, nruns, total, queue);
  if (chunk == 1024)
    return launch_batch_tiles<TX, TY, 1024, 3>(stream, num_sms, tma, do_rho, max_species, runs,
                                               base, nruns, total, queue);
  if (chunk == 512)
    return launch_batch_tiles<TX, TY, 512, 4>(stream, num_sms, tma, do_rho, max_species, runs,
                                              base, nruns, total, queue);
  return launch_batch_tiles<TX, TY, 256, 4>(stream, num_sms, tma, do_rho, max_species, runs,
                                            base, nruns, total, queue);
}

}  // namespace

cudaError_t launch_push_deposit_2d_batch(cudaStream_t stream, int num_sms, int tx, int ty,
                                         int chunk, bool tma, bool do_rho, int max_species,
                                         const RunDesc *runs, uint32_t *base, int nruns,
                                         uint32_t total, uint32_t *queue) {
  if (total == 0) return cudaSuccess;
#define AP_BATCH_SHAPE(X, Y)                                                                 \
  if (tx == X && ty == Y)                                                                    \
    return launch_batch_chunk<X, Y>(stream, num_sms, chunk, tma, do_rho, max_species, runs, \
                                    base, nruns, total, queue);
  AP_BATCH_SHAPE(16, 16)
  AP_BATCH_SHAPE(32, 16)
  AP_BATCH_SHAPE(8, 8)
  AP_BATCH_SHAPE(16, 8)
  AP_BATCH_SHAPE(4, 4)
#undef AP_BATCH_SHAPE
  return cudaErrorInvalidValue;
}

cudaError_t launch_push_deposit_1d_batch(cudaStream_t stream, int num_sms, bool do_rho,
                                         const RunDesc *runs, const uint32_t *base, int nruns,
                                         uint32_t total_chunks) {
  if (total_chunks == 0) return cudaSuccess;
  const uint32_t grid = total_chunks < (uint32_t)num_sms * 8 ? total_chunks : (uint32_t)num_sms * 8;
  if (do_rho)
    k_push_deposit_1d_batch<true><<<grid, kThreads1D, 0, stream>>>(runs, base, nruns);
  else
    k_push_deposit_1d_batch<false><<<grid, kThreads1D, 0, stream>>>(runs, base, nruns);
  return cudaGetLastError();
}

cudaError_t launch_selftest_wait(Ctx &c, uint32_t limit) {
  k_selftest_wait<<<1, 32, 0, c.stream>>>(c.status, limit);
  c.launches++;
  return cudaGetLastError();
}

namespace {

template <int kItems>
cudaError_t launch_1d_items(Ctx &c, const PushDepositParams &P) {
  const size_t chunk = (size_t)kThreads1D * kItems;
  const size_t nchunks = (P.number + chunk - 1) / chunk;
  if (nchunks == 0) return cudaSuccess;
  const int grid = (int)(nchunks < (size_t)c.num_sms * 8 ? nchunks : (size_t)c.num_sms * 8);
  if (P.do_rho)
    k_push_deposit_1d<true, kItems><<<grid, kThreads1D, 0, c.stream>>>(P);
  else
    k_push_deposit_1d<false, kItems><<<grid, kThreads1D, 0, c.stream>>>(P);
  c.launches++;
  return cudaGetLastError();
}

}  // namespace

// A chunk's slots per thread run one after the other, so few particles are cut
// into shorter chunks until there are about four blocks per SM (the 48 KB
// windows allow four).
cudaError_t launch_push_deposit_1d(Ctx &c, const PushDepositParams &P) {
  const size_t per = P.number / ((size_t)c.num_sms * 4 * kThreads1D);
  if (per >= 4) return launch_1d_items<kItems1D>(c, P);
  if (per >= 2) return launch_1d_items<4>(c, P);
  if (per >= 1) return launch_1d_items<2>(c, P);
  return launch_1d_items<1>(c, P);
}

}  // namespace apb
