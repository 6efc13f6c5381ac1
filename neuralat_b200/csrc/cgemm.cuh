// Complex product Y += A X with more than eight right-hand sides (FP32).
//
// A tile of 64 rows x 64 (64 x 32, 128 x 16) right-hand sides per CTA and 16
// columns of A and rows of X per stage of a shared-memory ring filled by
// cp.async.  A thread owns 4 rows x 4 right-hand sides; a column costs its warp
// four shared-memory wavefronts and 32 packed FMAs a lane, so the FP32 pipe is
// the bound (against eight right-hand sides at a time, with X read from shared
// memory for 4 rows only, and A once per eight).  Measured on B200, 64
// right-hand sides: 40 962 unknowns 35.9 -> 17.4 ms (49 TFLOP/s of 74), 10 242
// unknowns 1.80 -> 1.12 ms, 2562 unknowns 118 -> 87 us; 16 right-hand sides:
// 40 962 unknowns 7.26 -> 4.57 ms (0.45 of the bandwidth, 0.63 of the FP32 rate).
//
// Sums: re(a) x and im(a) x over 32 columns each, these over the CTA's columns
// (up to 1024, spread over the matrix so that a smooth integrand's oscillations
// cancel within the sums), these by one atomic per CTA.  Error against 64 bits
// on random entries, 64 right-hand sides: 1.93e-7 (lane sums over 1024 columns
// added by atomics: 1.96e-7) for 40 962 unknowns, 1.36e-7 (1.53e-7) for 2562.
// Below kCgLeast unknowns those lane sums have under 16 columns and the smaller
// error, and both kernels take less time than their launch.
#pragma once

#include <algorithm>
#include <atomic>
#include <cmath>

#include "async_copy.cuh"
#include "bem_common.cuh"

namespace bemb {
namespace {

constexpr int kCgLeast = 512;  // unknowns, and
constexpr int kCgSides = 8;    // right-hand sides above which it is used
constexpr int kCgCols = 16;    // columns of A per stage
constexpr int kCgRun = 32;     // columns per first-level sum
constexpr int kCgPitch = kCgCols * 8 + 16;  // bytes between A rows: 8 rows start in distinct bank groups
static_assert(kCgRun % kCgCols == 0 && kCgCols % 2 == 0, "");

template <int TM>
struct CgShape {
  static constexpr int kThreads = TM == 64 ? 256 : 128;
  static constexpr int kPerSm = 512 / kThreads;  // CTAs at 128 registers
  static constexpr int kRows = 16 * kThreads / TM;
  static constexpr int kStages = TM == 16 ? 2 : 4;
  static constexpr int kStageBytes = kRows * kCgPitch + kCgCols * TM * 8;
  static constexpr int kSmem = kStages * kStageBytes;
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
    if ((t + 1) % (kCgRun / kCgCols) == 0) fold();
  }
  fold();
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (r0 + row + 8 * i < n && s0 + side + j < m)
        atomicAdd(&Y[(size_t)(r0 + row + 8 * i) * m + s0 + side + j], acc[i][j]);
}

template <int TM, bool PAIRS>
int cgemm_part(const float2* A, int n, const float2* X, int m, int first, int groups, float2* Y, int sms,
               cudaStream_t s) {
  using Sh = CgShape<TM>;
  static std::atomic<bool> attr{false};
  if (!attr.load(std::memory_order_acquire)) {
    BEM_CUDA_TRY(cudaFuncSetAttribute(cgemm_kernel<TM, PAIRS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::kSmem));
    attr.store(true, std::memory_order_release);
  }
  const long long rows = (n + Sh::kRows - 1) / Sh::kRows;
  // Cut of the columns: least time for whole rounds of the CTAs that fit (a
  // CTA's start and end cost about 48 columns), around sqrt(32 n) columns, where
  // the roundings of the CTA's sums and of the atomics are least together.
  const double best = std::sqrt(32.0 * n);
  const long long places = (long long)sms * Sh::kPerSm, widest = std::min(1024LL, (long long)(2.0 * best) + kCgRun);
  long long span = 0, cost = 0;
  for (long long cuts = (n + widest - 1) / widest; cuts <= (long long)(3.0 * n / best) + 1; cuts++) {
    const long long w = ((n + cuts - 1) / cuts + kCgRun - 1) / kCgRun * kCgRun;
    const long long rounds = (rows * groups * ((n + w - 1) / w) + places - 1) / places;
    if (!span || rounds * (w + 48) < cost) {
      span = w;
      cost = rounds * (w + 48);
    }
  }
  const long long cuts = (n + span - 1) / span;
  (cgemm_kernel<TM, PAIRS><<<dim3((unsigned)rows, (unsigned)cuts, (unsigned)groups), Sh::kThreads, Sh::kSmem, s>>>(
       A, n, X, m, first, Y),
   count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

// Y += A X.
template <bool PAIRS>
int cgemm_all(const float2* A, int n, const float2* X, int m, float2* Y, int sms, cudaStream_t s) {
  // remainders of up to 32 right-hand sides in a tile of their own
  const int wide = m % 64 > 32 ? (m + 63) / 64 : m / 64, first = 64 * wide, left = m - first;
  if (wide) {
    const int rc = cgemm_part<64, PAIRS>(A, n, X, m, 0, wide, Y, sms, s);
    if (rc) return rc;
  }
  if (left > 16) return cgemm_part<32, PAIRS>(A, n, X, m, first, 1, Y, sms, s);
  if (left > 0) return cgemm_part<16, PAIRS>(A, n, X, m, first, 1, Y, sms, s);
  return BEM_OK;
}

int launch_cgemm(const float2* A, int n, const float2* X, int m, float2* Y, int sms, cudaStream_t s) {
  const bool pairs = (n & 1) == 0 && ((uintptr_t)A & 15) == 0;
  return pairs ? cgemm_all<true>(A, n, X, m, Y, sms, s) : cgemm_all<false>(A, n, X, m, Y, sms, s);
}

}  // namespace
}  // namespace bemb
