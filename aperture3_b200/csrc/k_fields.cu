// Yee FDTD update, divergences, current filter and guard-cell exchange on
// one rank (src/cuda/algorithms/field_solver.cu, ptc_updater.cu:501-560,
// cuda/sim_environment.cpp:9-127).
//
// The reference updates the bulk and then copies interior strips into the
// guard cells with one MPI self-exchange per direction. Here each thread
// that updates a bulk cell near a periodic side also writes that cell's
// periodic images in the guard layers, which leaves every guard cell of a
// periodic dim holding its bulk image -- the state send_guard_cells
// produces -- without a separate pass.
#include <cuda_runtime.h>

#include "ap_device.cuh"
#include "ap_internal.h"

namespace apb {

namespace {

struct Arr {
  float *p;
  int pitch;  // floats
  __device__ __forceinline__ float &operator()(int i, int j) const {
    return p[(size_t)j * pitch + i];
  }
};

__host__ Arr arr(const ap_array &a) { return Arr{a.ptr, (int)(a.pitch / sizeof(float))}; }

struct Geo {
  int n0, n1, g0, g1, r0, r1, per0, per1, dim;
  float id0, id1;
};

// Writes v at (i, j) and at its periodic guard images.
__device__ __forceinline__ void store_with_images(const Arr &a, const Geo &G, int i, int j,
                                                  float v) {
  a(i, j) = v;
  int ix[2] = {i, i}, jx[2] = {j, j};
  int ni = 1, nj = 1;
  if (G.per0) {
    if (i < 2 * G.g0) ix[ni++] = i + G.r0;
    else if (i >= G.n0 - 2 * G.g0) ix[ni++] = i - G.r0;
  }
  if (G.dim > 1 && G.per1) {
    if (j < 2 * G.g1) jx[nj++] = j + G.r1;
    else if (j >= G.n1 - 2 * G.g1) jx[nj++] = j - G.r1;
  }
  for (int b = 0; b < nj; ++b)
    for (int a2 = 0; a2 < ni; ++a2)
      if (a2 || b) a(ix[a2], jx[b]) = v;
}

// compute_e_update2d (field_solver.cu:45-84) / compute_e_update1d (:14-43)
// for bulk cell (n1, n2).
__device__ __forceinline__ void e_update_cell(const Geo &G, const Arr &e1, const Arr &e2,
                                              const Arr &e3, const Arr &b1, const Arr &b2,
                                              const Arr &b3, const Arr &b01, const Arr &b02,
                                              const Arr &b03, const Arr &j1, const Arr &j2,
                                              const Arr &j3, float dt, int n1, int n2) {
  if (G.dim > 1) {
    const float v1 = e1(n1, n2) + dt * ((b3(n1, n2 + 1) - b3(n1, n2) - b03(n1, n2 + 1) +
                                         b03(n1, n2)) * G.id1 - j1(n1, n2));
    const float v2 = e2(n1, n2) + dt * ((b3(n1, n2) - b3(n1 + 1, n2) - b03(n1, n2) +
                                         b03(n1 + 1, n2)) * G.id0 - j2(n1, n2));
    const float v3 =
        e3(n1, n2) + dt * ((b2(n1 + 1, n2) - b2(n1, n2) - b02(n1 + 1, n2) + b02(n1, n2)) *
                               G.id0 +
                           (b1(n1, n2) - b1(n1, n2 + 1) - b01(n1, n2) + b01(n1, n2 + 1)) *
                               G.id1 - j3(n1, n2));
    store_with_images(e1, G, n1, n2, v1);
    store_with_images(e2, G, n1, n2, v2);
    store_with_images(e3, G, n1, n2, v3);
  } else {
    const float v1 = e1(n1, 0) - dt * j1(n1, 0);
    const float v2 = e2(n1, 0) + dt * ((b3(n1, 0) - b3(n1 + 1, 0) - b03(n1, 0) +
                                        b03(n1 + 1, 0)) * G.id0 - j2(n1, 0));
    const float v3 = e3(n1, 0) + dt * ((b2(n1 + 1, 0) - b2(n1, 0) - b02(n1 + 1, 0) +
                                        b02(n1, 0)) * G.id0 - j3(n1, 0));
    store_with_images(e1, G, n1, 0, v1);
    store_with_images(e2, G, n1, 0, v2);
    store_with_images(e3, G, n1, 0, v3);
  }
}

__global__ void k_update_e(Geo G, Arr e1, Arr e2, Arr e3, Arr b1, Arr b2, Arr b3, Arr b01,
                           Arr b02, Arr b03, Arr j1, Arr j2, Arr j3, float dt) {
  const int n1 = G.g0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int n2 = (G.dim > 1 ? G.g1 : 0) + blockIdx.y * blockDim.y + threadIdx.y;
  if (n1 >= G.n0 - G.g0) return;
  if (G.dim > 1 && n2 >= G.n1 - G.g1) return;
  e_update_cell(G, e1, e2, e3, b1, b2, b3, b01, b02, b03, j1, j2, j3, dt, n1, n2);
}

// compute_b_update2d (field_solver.cu:160-193) / compute_b_update1d (:133-158)
// for bulk cell (n1, n2).
__device__ __forceinline__ void b_update_cell(const Geo &G, const Arr &e1, const Arr &e2,
                                              const Arr &e3, const Arr &e01, const Arr &e02,
                                              const Arr &e03, const Arr &b1, const Arr &b2,
                                              const Arr &b3, float dt, int n1, int n2) {
  if (G.dim > 1) {
    const float v1 = b1(n1, n2) - dt * (e3(n1, n2) - e3(n1, n2 - 1) - e03(n1, n2) +
                                        e03(n1, n2 - 1)) * G.id1;
    const float v2 = b2(n1, n2) - dt * (e3(n1 - 1, n2) - e3(n1, n2) - e03(n1 - 1, n2) +
                                        e03(n1, n2)) * G.id0;
    const float v3 =
        b3(n1, n2) - dt * ((e2(n1, n2) - e2(n1 - 1, n2) - e02(n1, n2) + e02(n1 - 1, n2)) *
                               G.id0 +
                           (e1(n1, n2 - 1) - e1(n1, n2) - e01(n1, n2 - 1) + e01(n1, n2)) *
                               G.id1);
    store_with_images(b1, G, n1, n2, v1);
    store_with_images(b2, G, n1, n2, v2);
    store_with_images(b3, G, n1, n2, v3);
  } else {
    // b1 is not updated in 1D; its guards are still refreshed by the
    // reference's exchange, which is a no-op when they already hold images.
    const float v2 = b2(n1, 0) - dt * (e3(n1 - 1, 0) - e3(n1, 0) - e03(n1 - 1, 0) +
                                       e03(n1, 0)) * G.id0;
    const float v3 = b3(n1, 0) - dt * (e2(n1, 0) - e2(n1 - 1, 0) - e02(n1, 0) +
                                       e02(n1 - 1, 0)) * G.id0;
    store_with_images(b1, G, n1, 0, b1(n1, 0));
    store_with_images(b2, G, n1, 0, v2);
    store_with_images(b3, G, n1, 0, v3);
  }
}

__global__ void k_update_b(Geo G, Arr e1, Arr e2, Arr e3, Arr e01, Arr e02, Arr e03, Arr b1,
                           Arr b2, Arr b3, float dt) {
  const int n1 = G.g0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int n2 = (G.dim > 1 ? G.g1 : 0) + blockIdx.y * blockDim.y + threadIdx.y;
  if (n1 >= G.n0 - G.g0) return;
  if (G.dim > 1 && n2 >= G.n1 - G.g1) return;
  b_update_cell(G, e1, e2, e3, e01, e02, e03, b1, b2, b3, dt, n1, n2);
}

// compute_divs_2d (field_solver.cu:261-288) / compute_divs_1d (:237-259) for
// bulk cell (n1, n2).
__device__ __forceinline__ void divs_cell(const Geo &G, const Arr &e1, const Arr &e2,
                                          const Arr &b1, const Arr &b2, const Arr &e01,
                                          const Arr &e02, const Arr &b01, const Arr &b02,
                                          const Arr &divE, const Arr &divB, int n1, int n2) {
  if (G.dim > 1) {
    divE(n1, n2) = (e1(n1 + 1, n2) - e01(n1 + 1, n2) - e1(n1, n2) + e01(n1, n2)) * G.id0 +
                   (e2(n1, n2 + 1) - e02(n1, n2 + 1) - e2(n1, n2) + e02(n1, n2)) * G.id1;
    divB(n1, n2) = (b1(n1, n2) - b01(n1, n2) - b1(n1 - 1, n2) + b01(n1 - 1, n2)) * G.id0 +
                   (b2(n1, n2) - b02(n1, n2) - b2(n1, n2 - 1) + b02(n1, n2 - 1)) * G.id1;
  } else {
    divE(n1, 0) = (e1(n1 + 1, 0) - e01(n1 + 1, 0) - e1(n1, 0) + e01(n1, 0)) * G.id0;
    divB(n1, 0) = (b1(n1, 0) - b01(n1, 0) - b1(n1 - 1, 0) + b01(n1 - 1, 0)) * G.id0;
  }
}

__global__ void k_divs(Geo G, Arr e1, Arr e2, Arr b1, Arr b2, Arr e01, Arr e02, Arr b01,
                       Arr b02, Arr divE, Arr divB) {
  const int n1 = G.g0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int n2 = (G.dim > 1 ? G.g1 : 0) + blockIdx.y * blockDim.y + threadIdx.y;
  if (n1 >= G.n0 - G.g0) return;
  if (G.dim > 1 && n2 >= G.n1 - G.g1) return;
  divs_cell(G, e1, e2, b1, b2, e01, e02, b01, b02, divE, divB, n1, n2);
}

// update_fields of a small grid (the optional half step of E, then B, E and
// the divergences) in one launch: one cluster of eight CTAs, a cluster barrier
// between the stages in place of a launch. Small CTAs, so that they find room
// beside another run's push. The line lies at two cells per thread: three
// launches take 12.3 us up to 65536 cells (latency), the cluster 6.2 us for 1024
// cells, 9.1 (1D) and 10.3 (64^2) for 4096, 12.3 for 72^2, 14.3 for 8192 and 22.5
// for 16384.
constexpr int kSmallThreads = 256;
constexpr int kSmallCtas = 8;
constexpr int kSmallCells = 2 * kSmallThreads * kSmallCtas;

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

struct FieldSet {
  Arr e1, e2, e3, b1, b2, b3, e01, e02, e03, b01, b02, b03, j1, j2, j3, divE, divB;
};

__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(kSmallThreads)
    k_fields_small(Geo G, const __grid_constant__ FieldSet F, float dt, float dt_half, int divs) {
  const int first = blockIdx.x * kSmallThreads + threadIdx.x;
  const int n = G.r0 * (G.dim > 1 ? G.r1 : 1);
  const int y0 = G.dim > 1 ? G.g1 : 0;
  auto each = [&](auto &&f) {
    for (int t = first; t < n; t += kSmallThreads * kSmallCtas) {
      const int y = t / G.r0;
      f(G.g0 + t - y * G.r0, y0 + y);
    }
  };
  auto e_step = [&](float h) {
    each([&](int x, int y) {
      e_update_cell(G, F.e1, F.e2, F.e3, F.b1, F.b2, F.b3, F.b01, F.b02, F.b03, F.j1, F.j2, F.j3,
                    h, x, y);
    });
    cluster_barrier();
  };
  if (dt_half != 0.0f) e_step(dt_half);
  each([&](int x, int y) {
    b_update_cell(G, F.e1, F.e2, F.e3, F.e01, F.e02, F.e03, F.b1, F.b2, F.b3, dt, x, y);
  });
  cluster_barrier();
  e_step(dt);
  if (divs)
    each([&](int x, int y) {
      divs_cell(G, F.e1, F.e2, F.b1, F.b2, F.e01, F.e02, F.b01, F.b02, F.divE, F.divB, x, y);
    });
}

// Guard strips of one dim: mode 0 copies interior strips into the opposite
// guards (send_array_guard_cells_single_dir), mode 1 adds guard strips into
// the opposite interior (send_add_array_guard_cells_single_dir). Both
// directions are handled in one launch; their strips are disjoint.
__global__ void k_guard_strips(Arr a, int n0, int n1, int g, int dim, int mode) {
  const int len = dim == 0 ? n1 : n0;  // extent along the other dim
  const int total = 2 * g * len;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    const int dir = t / (g * len);  // 0: dir -1, 1: dir +1
    const int rem = t % (g * len);
    const int layer = rem / len, o = rem % len;
    const int n = dim == 0 ? n0 : n1;
    int src, dst;
    if (mode == 0) {
      src = dir == 0 ? g + layer : n - 2 * g + layer;
      dst = dir == 0 ? n - g + layer : layer;
    } else {
      src = dir == 0 ? layer : n - g + layer;
      dst = dir == 0 ? n - 2 * g + layer : g + layer;
    }
    if (dim == 0) {
      if (mode == 0) a(dst, o) = a(src, o);
      else a(dst, o) += a(src, o);
    } else {
      if (mode == 0) a(o, dst) = a(o, src);
      else a(o, dst) += a(o, src);
    }
  }
}

// One smoothing pass over several arrays (the current and, on output steps,
// the charge densities) in two launches, blockIdx.z the array:
// k_filter, filter_current_cart_2d / _1d (ptc_updater.cu:501-560), the bulk
// only, into the scratch arrays; k_filter_store, the filtered bulk back and,
// with `images`, every periodic guard cell as send_guard_cells leaves it
// (dim 0 over all rows, then dim 1 over all columns): the value of its image,
// which in a guard row of a non-periodic dim is that row's own, unfiltered,
// value. Per array this was four launches (filter, copy, two guard strips), 20
// for a current with two charge densities: 36 us of small kernels and their
// launches on a 193^2 grid, which two launches replace.
struct SmoothArrs {
  Arr a[3 + AP_MAX_SPECIES];
};

__global__ void k_filter(Geo G, const __grid_constant__ SmoothArrs A, float *tmp, int tpitch,
                         size_t tcomp, int bl0, int bu0, int bl1, int bu1) {
  const int a = G.g0 + blockIdx.x * blockDim.x + threadIdx.x;
  const int b = (G.dim > 1 ? G.g1 : 0) + blockIdx.y * blockDim.y + threadIdx.y;
  const Arr j = A.a[blockIdx.z];
  const Arr t{tmp + blockIdx.z * tcomp, tpitch};
  if (a >= G.n0 - G.g0) return;
  const int xp = (bu0 && a == G.n0 - G.g0 - 1) ? 0 : 1;
  const int xm = (bl0 && a == G.g0) ? 0 : 1;
  if (G.dim > 1) {
    if (b >= G.n1 - G.g1) return;
    const int yp = (bu1 && b == G.n1 - G.g1 - 1) ? 0 : 1;
    const int ym = (bl1 && b == G.g1) ? 0 : 1;
    float v = 0.25f * j(a, b);
    v += 0.125f * j(a + xp, b);
    v += 0.125f * j(a - xm, b);
    v += 0.125f * j(a, b + yp);
    v += 0.125f * j(a, b - ym);
    v += 0.0625f * j(a + xp, b + yp);
    v += 0.0625f * j(a - xm, b + yp);
    v += 0.0625f * j(a + xp, b - ym);
    v += 0.0625f * j(a - xm, b - ym);
    t(a, b) = v;
  } else {
    float v = 0.5f * j(a, 0);
    v += 0.25f * j(a + xp, 0);
    v += 0.25f * j(a - xm, 0);
    t(a, 0) = v;
  }
}

__global__ void k_filter_store(Geo G, const float *__restrict__ tmp, int tpitch, size_t tcomp,
                               const __grid_constant__ SmoothArrs A, int images) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int rows = G.dim > 1 ? G.n1 : 1;
  if (x >= G.n0 || y >= rows) return;
  const Arr a = A.a[blockIdx.z];
  int xs = x, ys = y;  // the cell whose value this one takes
  if (images && G.per0) {
    if (x < G.g0) xs = x + G.r0;
    else if (x >= G.n0 - G.g0) xs = x - G.r0;
  }
  if (images && G.dim > 1 && G.per1) {
    if (y < G.g1) ys = y + G.r1;
    else if (y >= G.n1 - G.g1) ys = y - G.r1;
  }
  const bool bulk = xs >= G.g0 && xs < G.n0 - G.g0 &&
                    (G.dim == 1 || (ys >= G.g1 && ys < G.n1 - G.g1));
  if (bulk)
    a(x, y) = tmp[blockIdx.z * tcomp + (size_t)ys * tpitch + xs];
  else if (xs != x || ys != y)
    a(x, y) = a(xs, ys);
}

// Folds the periodic guard layers of the fixed-point accumulators into the
// bulk and rounds once to FP32. For one rank, send_add_guard_cells
// (cuda/sim_environment.cpp:71-127) adds the lower guard strip of a dim into
// the upper interior strip and the upper guard strip into the lower interior
// strip, dim 0 (all rows) before dim 1 (all columns), leaving the guard
// values in place; per cell that is the gather below. The integer sums are
// exact, so the order of the adds does not matter; the only rounding is the
// final conversion (int64 -> double is exact below 2^53, then one rounding
// to FP32).
__device__ __forceinline__ unsigned long long finalize_sum(const Geo &G,
                                                           const unsigned long long *a,
                                                           int acc_pitch, int x, int y) {
  int xi = -1, yi = -1;
  if (G.per0) {
    if (x >= G.g0 && x < 2 * G.g0) xi = x + G.r0;
    else if (x >= G.n0 - 2 * G.g0 && x < G.n0 - G.g0) xi = x - G.r0;
  }
  if (G.dim > 1 && G.per1) {
    if (y >= G.g1 && y < 2 * G.g1) yi = y + G.r1;
    else if (y >= G.n1 - 2 * G.g1 && y < G.n1 - G.g1) yi = y - G.r1;
  }
  unsigned long long v = a[(size_t)y * acc_pitch + x];
  if (xi >= 0) v += a[(size_t)y * acc_pitch + xi];
  if (yi >= 0) {
    v += a[(size_t)yi * acc_pitch + x];
    if (xi >= 0) v += a[(size_t)yi * acc_pitch + xi];
  }
  return v;
}

// 2^-S for the formats' |S| <= 100.
__device__ __forceinline__ double pow2_neg(int S) {
  return __longlong_as_double((long long)(1023 - S) << 52);
}

struct FinalArrs {
  Arr a[3 + AP_MAX_SPECIES];
};

// blockIdx.z the component; a thread rounds kFinalRows rows of one column, all
// loads before the first store (one cell per thread and round took 59 us for
// three components of 2048^2 cells, 151 MB).
constexpr int kFinalRows = 4;

__global__ void k_finalize(Geo G, const unsigned long long *__restrict__ acc, int acc_pitch,
                           size_t acc_comp, const FixedFmt *fmt,
                           const __grid_constant__ FinalArrs O) {
  const int rows = G.dim > 1 ? G.n1 : 1;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y0 = blockIdx.y * blockDim.y * kFinalRows + threadIdx.y;
  if (x >= G.n0) return;
  const Arr out = O.a[blockIdx.z];
  const unsigned long long *a = acc + blockIdx.z * acc_comp;
  const double inv = pow2_neg(fmt->S);
  unsigned long long v[kFinalRows];
#pragma unroll
  for (int k = 0; k < kFinalRows; ++k) {
    const int y = y0 + k * blockDim.y;
    v[k] = y < rows ? finalize_sum(G, a, acc_pitch, x, y) : 0ull;
  }
#pragma unroll
  for (int k = 0; k < kFinalRows; ++k) {
    const int y = y0 + k * blockDim.y;
    if (y < rows) out(x, y) = (float)((double)(long long)v[k] * inv);
  }
}

Geo make_geo(const Ctx &c) {
  const ap_mesh &m = c.mesh;
  Geo G;
  G.n0 = m.dims[0];
  G.n1 = m.dims[1];
  G.g0 = m.guard[0];
  G.g1 = m.guard[1];
  G.r0 = m.dims[0] - 2 * m.guard[0];
  G.r1 = m.dims[1] - 2 * m.guard[1];
  G.per0 = c.params.periodic[0];
  G.per1 = c.params.periodic[1];
  G.dim = c.mk.dim;
  G.id0 = m.inv_delta[0];
  G.id1 = m.inv_delta[1];
  return G;
}

void bulk_launch_shape(const Geo &G, dim3 &grid, dim3 &block) {
  if (G.dim > 1) {
    block = dim3(32, 8);
    grid = dim3((G.r0 + 31) / 32, (G.r1 + 7) / 8);
  } else {
    block = dim3(256, 1);
    grid = dim3((G.r0 + 255) / 256, 1);
  }
}

}  // namespace

namespace {

// ---------------------------------------------------------------------------
// Batched 1D launches: work item g belongs to run r with base[r] <= g <
// base[r + 1]; the per-cell arithmetic is the single-run kernels'.

__device__ __forceinline__ int run_of(const uint32_t *base, int nruns, uint32_t g) {
  int lo = 0, hi = nruns - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ Arr farr(const FieldArr &a) { return Arr{a.ptr, a.pitch}; }

__device__ __forceinline__ Geo geo1(const Run1D &R) {
  Geo G;
  G.n0 = R.n0;
  G.n1 = 1;
  G.g0 = R.g0;
  G.g1 = 0;
  G.r0 = R.r0;
  G.r1 = 0;
  G.per0 = R.per0;
  G.per1 = 0;
  G.dim = 1;
  G.id0 = R.id0;
  G.id1 = 0.0f;
  return G;
}

__global__ void k_b1_zero(const Run1D *__restrict__ runs, const uint32_t *__restrict__ base,
                          int nruns) {
  const uint32_t total = base[nruns];
  for (uint32_t g = blockIdx.x; g < total; g += gridDim.x) {
    const int r = run_of(base, nruns, g);
    const Run1D &R = runs[r];
    const size_t w = (size_t)(g - base[r]) * 256 + threadIdx.x;
    if (w < (size_t)R.zero_comps * R.acc_comp) R.acc[w] = 0ull;
  }
}

__global__ void k_b1_finalize(const Run1D *__restrict__ runs, const uint32_t *__restrict__ base,
                              int nruns) {
  const uint32_t total = base[nruns];
  for (uint32_t g = blockIdx.x; g < total; g += gridDim.x) {
    const int r = run_of(base, nruns, g);
    const Run1D &R = runs[r];
    const int x = (int)(g - base[r]) * 256 + threadIdx.x;
    if (x >= R.n0) continue;
    const Geo G = geo1(R);
    const double inv = pow2_neg(R.fx->S);
    for (int comp = 0; comp < R.ncomp; ++comp) {
      const Arr out = farr(comp < 3 ? R.J[comp] : R.Rho[comp - 3]);
      const long long v = (long long)finalize_sum(G, R.acc + comp * R.acc_comp, R.n0, x, 0);
      out(x, 0) = (float)((double)v * inv);
    }
  }
}

__global__ void k_b1_fields(const Run1D *__restrict__ runs, const uint32_t *__restrict__ base,
                            int nruns, int which) {
  const uint32_t total = base[nruns];
  for (uint32_t g = blockIdx.x; g < total; g += gridDim.x) {
    const int r = run_of(base, nruns, g);
    const Run1D &R = runs[r];
    const int n1 = R.g0 + (int)(g - base[r]) * 256 + threadIdx.x;
    if (n1 >= R.n0 - R.g0) continue;
    const Geo G = geo1(R);
    if (which == 0 || which == 2) {
      const float dt = which == 0 ? R.dt_half : R.dt;
      if (which == 0 && !(dt > 0.0f)) continue;
      e_update_cell(G, farr(R.E[0]), farr(R.E[1]), farr(R.E[2]), farr(R.B[0]), farr(R.B[1]),
                    farr(R.B[2]), farr(R.Bb[0]), farr(R.Bb[1]), farr(R.Bb[2]), farr(R.J[0]),
                    farr(R.J[1]), farr(R.J[2]), dt, n1, 0);
    } else if (which == 1) {
      b_update_cell(G, farr(R.E[0]), farr(R.E[1]), farr(R.E[2]), farr(R.Eb[0]), farr(R.Eb[1]),
                    farr(R.Eb[2]), farr(R.B[0]), farr(R.B[1]), farr(R.B[2]), R.dt, n1, 0);
    } else if (R.has_divs) {
      divs_cell(G, farr(R.E[0]), farr(R.E[1]), farr(R.B[0]), farr(R.B[1]), farr(R.Eb[0]),
                farr(R.Eb[1]), farr(R.Bb[0]), farr(R.Bb[1]), farr(R.divE), farr(R.divB), n1, 0);
    }
  }
}

uint32_t grid_of(uint32_t total, int num_sms) {
  const uint32_t cap = (uint32_t)num_sms * 16;
  return total < cap ? total : cap;
}

}  // namespace

cudaError_t launch_b1_zero(cudaStream_t s, int num_sms, const Run1D *runs, const uint32_t *base,
                           int nruns, uint32_t total) {
  if (total == 0) return cudaSuccess;
  k_b1_zero<<<grid_of(total, num_sms), 256, 0, s>>>(runs, base, nruns);
  return cudaGetLastError();
}

cudaError_t launch_b1_finalize(cudaStream_t s, int num_sms, const Run1D *runs,
                               const uint32_t *base, int nruns, uint32_t total) {
  if (total == 0) return cudaSuccess;
  k_b1_finalize<<<grid_of(total, num_sms), 256, 0, s>>>(runs, base, nruns);
  return cudaGetLastError();
}

cudaError_t launch_b1_fields(cudaStream_t s, int num_sms, const Run1D *runs, const uint32_t *base,
                             int nruns, uint32_t total, int which) {
  if (total == 0) return cudaSuccess;
  k_b1_fields<<<grid_of(total, num_sms), 256, 0, s>>>(runs, base, nruns, which);
  return cudaGetLastError();
}

cudaError_t launch_update_e(Ctx &c, float dt) {
  const ap_fields &f = c.fields;
  Geo G = make_geo(c);
  dim3 grid, block;
  bulk_launch_shape(G, grid, block);
  k_update_e<<<grid, block, 0, c.stream>>>(G, arr(f.E[0]), arr(f.E[1]), arr(f.E[2]),
                                           arr(f.B[0]), arr(f.B[1]), arr(f.B[2]),
                                           arr(f.Bbg[0]), arr(f.Bbg[1]), arr(f.Bbg[2]),
                                           arr(f.J[0]), arr(f.J[1]), arr(f.J[2]), dt);
  c.launches++;
  return cudaGetLastError();
}

cudaError_t launch_update_b(Ctx &c, float dt) {
  const ap_fields &f = c.fields;
  Geo G = make_geo(c);
  dim3 grid, block;
  bulk_launch_shape(G, grid, block);
  k_update_b<<<grid, block, 0, c.stream>>>(G, arr(f.E[0]), arr(f.E[1]), arr(f.E[2]),
                                           arr(f.Ebg[0]), arr(f.Ebg[1]), arr(f.Ebg[2]),
                                           arr(f.B[0]), arr(f.B[1]), arr(f.B[2]), dt);
  c.launches++;
  return cudaGetLastError();
}

// field_solver::update_fields (field_solver.cu:334-358): B, E, divergences,
// at step 0 after a half step of E. Grids of up to kSmallCells bulk cells take
// one launch, larger ones a launch per stage.
cudaError_t launch_fields(Ctx &c, float dt, float dt_half) {
  const Geo G = make_geo(c);
  const ap_fields &f = c.fields;
  if ((size_t)G.r0 * (G.dim > 1 ? G.r1 : 1) <= (size_t)kSmallCells) {
    const bool divs = f.divE.ptr && f.divB.ptr;
    const FieldSet F{arr(f.E[0]),   arr(f.E[1]),   arr(f.E[2]),   arr(f.B[0]),   arr(f.B[1]),
                     arr(f.B[2]),   arr(f.Ebg[0]), arr(f.Ebg[1]), arr(f.Ebg[2]), arr(f.Bbg[0]),
                     arr(f.Bbg[1]), arr(f.Bbg[2]), arr(f.J[0]),   arr(f.J[1]),   arr(f.J[2]),
                     divs ? arr(f.divE) : Arr{nullptr, 0}, divs ? arr(f.divB) : Arr{nullptr, 0}};
    k_fields_small<<<kSmallCtas, kSmallThreads, 0, c.stream>>>(G, F, dt, dt_half, divs ? 1 : 0);
    c.launches++;
    return cudaGetLastError();
  }
  cudaError_t e = dt_half != 0.0f ? launch_update_e(c, dt_half) : cudaSuccess;
  if (e == cudaSuccess) e = launch_update_b(c, dt);
  if (e == cudaSuccess) e = launch_update_e(c, dt);
  return e == cudaSuccess ? launch_divs(c) : e;
}

cudaError_t launch_divs(Ctx &c) {
  const ap_fields &f = c.fields;
  if (!f.divE.ptr || !f.divB.ptr) return cudaSuccess;
  Geo G = make_geo(c);
  dim3 grid, block;
  bulk_launch_shape(G, grid, block);
  k_divs<<<grid, block, 0, c.stream>>>(G, arr(f.E[0]), arr(f.E[1]), arr(f.B[0]), arr(f.B[1]),
                                       arr(f.Ebg[0]), arr(f.Ebg[1]), arr(f.Bbg[0]),
                                       arr(f.Bbg[1]), arr(f.divE), arr(f.divB));
  c.launches++;
  return cudaGetLastError();
}

static cudaError_t guard_pass(Ctx &c, ap_array a, int mode) {
  const ap_mesh &m = c.mesh;
  const int nd = c.mk.dim;
  for (int d = 0; d < nd && d < 2; ++d) {
    if (!c.params.periodic[d]) continue;
    const int len = d == 0 ? m.dims[1] : m.dims[0];
    const int total = 2 * m.guard[d] * len;
    int grid = (total + 255) / 256;
    if (grid > 1024) grid = 1024;
    k_guard_strips<<<grid, 256, 0, c.stream>>>(arr(a), m.dims[0], m.dims[1], m.guard[d], d, mode);
    c.launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_copy_guards(Ctx &c, ap_array a) { return guard_pass(c, a, 0); }
cudaError_t launch_fold_guards(Ctx &c, ap_array a) { return guard_pass(c, a, 1); }

static cudaError_t smooth_pass(Ctx &c, const SmoothArrs &A, int narr, float *tmp, size_t tcomp,
                               const int bnd[4], bool images) {
  const Geo G = make_geo(c);
  dim3 grid, block;
  bulk_launch_shape(G, grid, block);
  grid.z = narr;
  k_filter<<<grid, block, 0, c.stream>>>(G, A, tmp, G.n0, tcomp, bnd[0], bnd[1], bnd[2], bnd[3]);
  const dim3 all((G.n0 + block.x - 1) / block.x,
                 G.dim > 1 ? (G.n1 + block.y - 1) / block.y : 1, narr);
  k_filter_store<<<all, block, 0, c.stream>>>(G, tmp, G.n0, tcomp, A, images ? 1 : 0);
  c.launches += 2;
  return cudaGetLastError();
}

// The filter of one array alone, its guards as they are.
cudaError_t launch_filter(Ctx &c, ap_array a, int bnd[4]) {
  SmoothArrs A{};
  A.a[0] = arr(a);
  return smooth_pass(c, A, 1, c.tmp_j, 0, bnd, false);
}

// One smoothing pass of an update: J and, with_rho, the charge densities,
// then their periodic guards. The scratch is the fixed-point accumulators'
// memory: between the finalize and the next update they hold nothing.
cudaError_t launch_smooth_current(Ctx &c, bool with_rho, const int bnd[4]) {
  SmoothArrs A{};
  int n = 0;
  for (int k = 0; k < 3; ++k) A.a[n++] = arr(c.fields.J[k]);
  if (with_rho)
    for (int s = 0; s < c.params.num_species; ++s) A.a[n++] = arr(c.fields.Rho[s]);
  return smooth_pass(c, A, n, reinterpret_cast<float *>(c.acc), 2 * c.acc_comp, bnd, true);
}

// ---------------------------------------------------------------------------
// The 1D labs' smoothing (gap: 1-2-1 over whole rows, ptc_updater_1dgap.cu:
// 196-213; GR: weighted by a flux-tube factor and divided by the cell's own,
// ptc_updater_1dgr.cu:388-404): all passes of several rows in one launch, one
// CTA per row, the row in shared memory between the passes (two buffers). The
// value past either end of a row counts as 0.
struct LineRow {
  const float *src;
  float *dst, *dst2;    // dst2: a second copy of the result, or null
  const float *k1;      // GR: the weights; null: the gap lab's filter
};
struct LineRows {
  LineRow r[2 + AP_MAX_SPECIES];
};
constexpr int kLineThreads = 512;

__global__ void __launch_bounds__(kLineThreads)
    k_line_smooth(const __grid_constant__ LineRows R, int n, int g, int bnd_lower, int bnd_upper,
                  int passes) {
  extern __shared__ float s_line[];
  const LineRow &row = R.r[blockIdx.x];
  float *a = s_line, *b = s_line + n;
  for (int i = threadIdx.x; i < n; i += kLineThreads) a[i] = row.src[i];
  __syncthreads();
  for (int it = 0; it < passes; ++it) {
    for (int i = threadIdx.x; i < n; i += kLineThreads) {
      const int ip = i + ((bnd_upper && i == n - g - 1) ? 0 : 1);
      const int im = i - ((bnd_lower && i == g) ? 0 : 1);
      const float jp = ip < n ? a[ip] : 0.0f, jm = im >= 0 ? a[im] : 0.0f;
      float t;
      if (row.k1) {
        const float kp = ip < n ? row.k1[ip] : 0.0f, km = im >= 0 ? row.k1[im] : 0.0f;
        t = 0.5f * a[i] * row.k1[i];
        t += 0.25f * jp * kp;
        t += 0.25f * jm * km;
        t /= row.k1[i];
      } else {
        t = 0.5f * a[i];
        t += 0.25f * jp;
        t += 0.25f * jm;
      }
      b[i] = t;
    }
    __syncthreads();
    float *t = a;
    a = b;
    b = t;
  }
  for (int i = threadIdx.x; i < n; i += kLineThreads) {
    row.dst[i] = a[i];
    if (row.dst2) row.dst2[i] = a[i];
  }
}

// Rows that fit shared memory twice: up to 28000 cells in one launch for all
// rows and passes. 8192 cells, one pass of E3, J1 and two charge densities:
// 9 launches of 1.6 us before, 2 here.
constexpr int kLineCells = 28000;
bool line_smooth_fits(const Ctx &c) { return c.mesh.dims[0] <= kLineCells; }

static cudaError_t launch_line_rows(Ctx &c, const LineRows &R, int rows, int passes) {
  const size_t smem = 2 * sizeof(float) * (size_t)c.mesh.dims[0];
  if (smem > 48 * 1024) {  // the longest row's, the same from every context and thread
    cudaError_t e = cudaFuncSetAttribute(k_line_smooth,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(2 * sizeof(float) * kLineCells));
    if (e != cudaSuccess) return e;
  }
  const int b = !c.params.periodic[0];
  k_line_smooth<<<rows, kLineThreads, smem, c.stream>>>(R, c.mesh.dims[0], c.mesh.guard[0], b, b,
                                                        passes);
  c.launches++;
  return cudaGetLastError();
}

// E3 = E1 smoothed `passes` times, the scratch E2 a copy of it when passes > 0.
cudaError_t launch_line_smooth_e(Ctx &c, const float *k1, int passes) {
  LineRows R{};
  R.r[0] = LineRow{c.fields.E[0].ptr, c.fields.E[2].ptr,
                   passes > 0 ? c.fields.E[1].ptr : nullptr, k1};
  return launch_line_rows(c, R, 1, passes);
}

// J1 (weights kj) and every charge density (weights kr) smoothed in place.
cudaError_t launch_line_smooth_current(Ctx &c, const float *kj, const float *kr, int passes) {
  if (passes <= 0) return cudaSuccess;
  LineRows R{};
  R.r[0] = LineRow{c.fields.J[0].ptr, c.fields.J[0].ptr, nullptr, kj};
  for (int s = 0; s < c.params.num_species; ++s)
    R.r[1 + s] = LineRow{c.fields.Rho[s].ptr, c.fields.Rho[s].ptr, nullptr, kr};
  return launch_line_rows(c, R, 1 + c.params.num_species, passes);
}

cudaError_t launch_finalize_current(Ctx &c, int ncomp) {
  Geo G = make_geo(c);
  FinalArrs O{};
  for (int k = 0; k < 3; ++k) O.a[k] = arr(c.fields.J[k]);
  for (int s = 0; s < c.params.num_species; ++s) O.a[3 + s] = arr(c.fields.Rho[s]);
  const dim3 block = G.dim > 1 ? dim3(32, 8) : dim3(256, 1);
  const int rows = (int)block.y * kFinalRows;
  const dim3 grid((G.n0 + block.x - 1) / block.x, G.dim > 1 ? (G.n1 + rows - 1) / rows : 1, ncomp);
  k_finalize<<<grid, block, 0, c.stream>>>(G, c.acc, c.mesh.dims[0], c.acc_comp, c.fx_used, O);
  c.launches++;
  return cudaGetLastError();
}

cudaError_t launch_zero(Ctx &c, ap_array a) {
  const ap_mesh &m = c.mesh;
  return cudaMemset2DAsync(a.ptr, a.pitch, 0, sizeof(float) * m.dims[0],
                           (size_t)m.dims[1] * m.dims[2], c.stream);
}

}  // namespace apb
