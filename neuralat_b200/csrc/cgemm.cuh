// Complex product Y += A X with more than eight right-hand sides (FP32), above
// 8192 unknowns.
//
// A tile of 64 rows x 64 (128 x 16) right-hand sides per CTA and 16 columns of A
// and rows of X per stage of a shared-memory ring filled by cp.async.  A thread
// owns 4 rows x 4 right-hand sides; a column costs its warp four shared-memory
// wavefronts and 32 packed FMAs a lane, so the FP32 pipe is the bound (against
// eight right-hand sides at a time, with X read from shared memory for 4 rows
// only, and A once per eight).  Measured on B200: 40 962 unknowns, 64 right-hand
// sides 35.6 -> 18.2 ms (47 TFLOP/s of 74), 48: 21.6 -> 15.6 ms, 16: 7.2 -> 4.9
// ms; 10 242 unknowns, 64: 1.82 -> 1.23 ms, 24: 0.71 -> 0.61 ms, 16: 0.43 -> 0.32
// ms.
//
// Sums: re(a) x and im(a) x over 16 columns each, these over 128 columns in
// registers, these over the CTA's columns (up to 1024, spread over the matrix so
// that a smooth integrand's oscillations cancel within the sums) in shared
// memory, these over the CTAs of a cluster in FP64 and rounded once, and one
// atomic per cluster, no more of them than with lane sums over 1024 columns.
// Against 64 bits, 10 242 unknowns and smooth fields, those lane sums and this:
// double layer 1.1e-7 and 0.9e-7, single layer 8.3e-8 and 6.6 to 7.4e-8 (with 32
// columns, the CTA's columns in one chain and one atomic per CTA 1.2e-7 and
// 9.1e-8).
#pragma once

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "async_copy.cuh"
#include "bem_common.cuh"

namespace bemb {
namespace {

constexpr int kCgCols = 16;    // columns of A per stage
constexpr int kCgFar = 128;    // columns per second-level sum
constexpr int kCgPitch = kCgCols * 8 + 16;  // bytes between A rows: 8 rows start in distinct bank groups
static_assert(kCgFar % kCgCols == 0 && kCgCols % 2 == 0, "");

template <int TM>
struct CgShape {
  static constexpr int kThreads = TM == 64 ? 256 : 128;
  static constexpr int kPerSm = 512 / kThreads;  // CTAs at 128 registers
  static constexpr int kRows = 16 * kThreads / TM;
  static constexpr int kStages = TM == 16 ? 2 : 4;
  static constexpr int kStageBytes = kRows * kCgPitch + kCgCols * TM * 8;
  static constexpr int kRing = kStages * kStageBytes;
  static constexpr int kSmem = kRing + 16 * kThreads * (int)sizeof(float2);  // and the threads' sums
};

__device__ __forceinline__ void cg_copy16(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cg_copy8(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}

// Columns [c, c + 16) of A and rows of X into one stage; past the matrix zeros.
template <int TM, bool PAIRS>
__device__ __forceinline__ void cg_load(unsigned char* stage, const float2* __restrict__ A, int n,
                                        const float2* __restrict__ X, int m, int s0, int r0, int c) {
  constexpr int kRows = CgShape<TM>::kRows;
  if (PAIRS) {
#pragma unroll
    for (int e = threadIdx.x; e < kRows * kCgCols / 2; e += CgShape<TM>::kThreads) {
      const int r = e / (kCgCols / 2), q = 2 * (e % (kCgCols / 2));
      const bool ok = r0 + r < n && c + q < n;
      cg_copy16(stage + r * kCgPitch + 8 * q, ok ? A + (size_t)(r0 + r) * n + c + q : A, ok);
    }
  } else {
#pragma unroll
    for (int e = threadIdx.x; e < kRows * kCgCols; e += CgShape<TM>::kThreads) {
      const int r = e / kCgCols, q = e % kCgCols;
      const bool ok = r0 + r < n && c + q < n;
      cg_copy8(stage + r * kCgPitch + 8 * q, ok ? A + (size_t)(r0 + r) * n + c + q : A, ok);
    }
  }
  unsigned char* xs = stage + kRows * kCgPitch;
#pragma unroll
  for (int e = threadIdx.x; e < kCgCols * TM; e += CgShape<TM>::kThreads) {
    const int q = e / TM, sl = e % TM;
    const bool ok = c + q < n && s0 + sl < m;
    cg_copy8(xs + 8 * e, ok ? X + (size_t)(c + q) * m + s0 + sl : X, ok);
  }
}

// Rows blockIdx.x * kRows ..., every gridDim.y-th tile of columns, right-hand
// sides first + blockIdx.z * TM ...
template <int TM, bool PAIRS>
__global__ void __launch_bounds__(CgShape<TM>::kThreads, CgShape<TM>::kPerSm)
    cgemm_kernel(const float2* __restrict__ A, int n, const float2* __restrict__ X, int m, int first,
                 float2* __restrict__ Y) {
  using Sh = CgShape<TM>;
  extern __shared__ __align__(16) unsigned char cg_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kSideWarps = TM / 16;
  const int row = (warp / kSideWarps) * 32 + (lane >> 2);               // rows row + 8 i of the tile
  const int side = (warp % kSideWarps) * 16 + 4 * (lane & 3);           // right-hand sides side + j
  const int r0 = blockIdx.x * Sh::kRows, s0 = first + blockIdx.z * TM;
  const int c0 = blockIdx.y * kCgCols, step = gridDim.y * kCgCols;  // tile t: columns c0 + t step ...
  const int tiles = (n - c0 + step - 1) / step;

  float2 acc[4][4], p[4][4], q[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = p[i][j] = q[i][j] = make_float2(0.f, 0.f);
  auto fold = [&]() {
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        acc[i][j].x += p[i][j].x - q[i][j].y;
        acc[i][j].y += p[i][j].y + q[i][j].x;
        p[i][j] = q[i][j] = make_float2(0.f, 0.f);
      }
  };

  // the thread's sums of the columns before
  float2* sums = reinterpret_cast<float2*>(cg_smem + Sh::kRing);
  bool fresh = true;
  auto move = [&]() {
#pragma unroll
    for (int e = 0; e < 16; e++) {
      float2 v = acc[e / 4][e % 4];
      float2& t = sums[e * Sh::kThreads + threadIdx.x];
      if (!fresh) v = f2_add(v, t);
      t = v;
      acc[e / 4][e % 4] = make_float2(0.f, 0.f);
    }
    fresh = false;
  };
#pragma unroll
  for (int t = 0; t < Sh::kStages - 1; t++) {
    if (t < tiles) cg_load<TM, PAIRS>(cg_smem + t * Sh::kStageBytes, A, n, X, m, s0, r0, c0 + t * step);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int t = 0; t < tiles; t++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(Sh::kStages - 2) : "memory");
    __syncthreads();  // stage t has landed for all, stage t - 1 has been read by all
    const int ahead = t + Sh::kStages - 1;
    if (ahead < tiles)
      cg_load<TM, PAIRS>(cg_smem + (ahead % Sh::kStages) * Sh::kStageBytes, A, n, X, m, s0, r0, c0 + ahead * step);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const unsigned char* stage = cg_smem + (t % Sh::kStages) * Sh::kStageBytes;
    const unsigned char* as = stage + row * kCgPitch;
    const unsigned char* xs = stage + Sh::kRows * kCgPitch + 8 * side;
#pragma unroll
    for (int c = 0; c < kCgCols; c += 2) {
      float4 a[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const float4*>(as + 8 * i * kCgPitch + 8 * c);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const float4 x01 = *reinterpret_cast<const float4*>(xs + (c + h) * TM * 8);
        const float4 x23 = *reinterpret_cast<const float4*>(xs + (c + h) * TM * 8 + 16);
        const float2 x[4] = {make_float2(x01.x, x01.y), make_float2(x01.z, x01.w), make_float2(x23.x, x23.y),
                             make_float2(x23.z, x23.w)};
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float2 re = f2(h ? a[i].z : a[i].x), im = f2(h ? a[i].w : a[i].y);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            p[i][j] = f2_fma(re, x[j], p[i][j]);
            q[i][j] = f2_fma(im, x[j], q[i][j]);
          }
        }
      }
    }
    fold();
    if ((t + 1) % (kCgFar / kCgCols) == 0) move();
  }
  auto add_out = [&](int i, int j, float2 v) {
    if (r0 + row + 8 * i < n && s0 + side + j < m) atomicAdd(&Y[(size_t)(r0 + row + 8 * i) * m + s0 + side + j], v);
  };
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int ctas = (int)cluster.num_blocks();
  move();
  // every CTA adds up a part of the cluster's sums
  cluster.sync();  // they are complete
  for (int e = (int)cluster.block_rank(); e < 16; e += ctas) {
    double re = 0.0, im = 0.0;
    for (int r = 0; r < ctas; r++) {
      const float2 v = *cluster.map_shared_rank(&sums[e * Sh::kThreads + threadIdx.x], r);
      re += (double)v.x;
      im += (double)v.y;
    }
    add_out(e / 4, e % 4, make_float2((float)re, (float)im));
  }
  cluster.sync();  // they have been read
}

template <int TM, bool PAIRS>
int cgemm_part(const float2* A, int n, const float2* X, int m, int first, int groups, float2* Y, int sms,
               cudaStream_t s) {
  using Sh = CgShape<TM>;
  static DeviceOnce once;
  if (const int rc = once.shared_memory(cgemm_kernel<TM, PAIRS>, Sh::kSmem)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(Sh::kThreads, 1, 1);
  cfg.dynamicSmemBytes = Sh::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  // CTAs that fit as clusters of 4 and of 8
  static std::atomic<int> fit[2];
  auto places = [&](int c) -> long long {
    std::atomic<int>& known = fit[c == 8];
    int k = known.load(std::memory_order_relaxed);
    if (k == 0) {
      at[0].val.clusterDim.y = (unsigned)c;
      cfg.gridDim = dim3(1, (unsigned)c, 1);
      if (cudaOccupancyMaxActiveClusters(&k, cgemm_kernel<TM, PAIRS>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
      }
      if (k < 1) k = -1;  // none
      known.store(k, std::memory_order_relaxed);
    }
    return k > 0 ? (long long)k * c : 0;
  };
  // Cut of the columns: least time for whole rounds of the CTAs that fit (a
  // CTA's start and end cost about 48 columns), at most 1024 columns per CTA, at
  // least 1024 per cluster.
  const long long rows = (n + Sh::kRows - 1) / Sh::kRows;
  int best = (n + 1023) / 1024, ctas = 1;
  long long cost = 0;
  for (int cuts = (best + 3) / 4 * 4; 128 * cuts <= n; cuts += 4)
    for (int c = 4; c <= 8; c *= 2) {
      if (cuts % c || 1024LL * cuts > (long long)c * n) continue;
      const long long fits = places(c);
      if (!fits) continue;
      const long long w = ((n + cuts - 1) / cuts + kCgCols - 1) / kCgCols * kCgCols;
      const long long time = (rows * groups * cuts + fits - 1) / fits * (w + 48);
      if (!cost || time < cost) {
        best = cuts;
        ctas = c;
        cost = time;
      }
    }
  at[0].val.clusterDim.y = (unsigned)ctas;
  cfg.gridDim = dim3((unsigned)rows, (unsigned)best, (unsigned)groups);
  BEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, cgemm_kernel<TM, PAIRS>, A, n, X, m, first, Y));
  count_launch();
  return BEM_OK;
}

// Y += A X.
template <bool PAIRS>
int cgemm_all(const float2* A, int n, const float2* X, int m, float2* Y, int sms, cudaStream_t s) {
  // a remainder of up to 48 right-hand sides goes 16 at a time: three reads of A
  // take less time than a tile of 64 (10 242 unknowns: 0.32 ms each, 1.2 ms)
  const int wide = m % 64 > 48 ? (m + 63) / 64 : m / 64, first = 64 * wide;
  if (wide) {
    const int rc = cgemm_part<64, PAIRS>(A, n, X, m, 0, wide, Y, sms, s);
    if (rc) return rc;
  }
  return m > first ? cgemm_part<16, PAIRS>(A, n, X, m, first, (m - first + 15) / 16, Y, sms, s) : BEM_OK;
}

// Where it is used.  Up to 8192 unknowns it would still take 0.80 to 0.86 of the
// time with 9 to 16 right-hand sides (2562 unknowns 42 and 34 us), but single
// layers times smooth fields come out up to 1.15 times as far off 64 bits (642
// to 5002 unknowns), and with 17 to 56 it is no faster.
inline bool cgemm_takes(int n, int m) { return m > 8 && n > 8192; }

int launch_cgemm(const float2* A, int n, const float2* X, int m, float2* Y, int sms, cudaStream_t s) {
  const bool pairs = (n & 1) == 0 && ((uintptr_t)A & 15) == 0;
  return pairs ? cgemm_all<true>(A, n, X, m, Y, sms, s) : cgemm_all<false>(A, n, X, m, Y, sms, s);
}

}  // namespace
}  // namespace bemb
