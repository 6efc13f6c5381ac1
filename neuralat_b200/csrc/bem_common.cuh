// Shared definitions for the B200 boundary-element kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "../../include/bem_b200.h"

namespace bemb {

// ---- quadrature ---------------------------------------------------------
// Six-point degree-4 triangle rule (Dunavant), the rule the reference uses for
// regular pairs, the mass matrix and listener potentials
// (src/bem/cuda/include/gauss.h:106-126).  Points are given by barycentric
// orbits (a, a, 1-2a); weights sum to one.  Point q has its dominant
// barycentric weight at local vertex q % 3, which the kernels exploit.
constexpr double kTriA1 = 0.44594849091596489;   // orbit 1: (1-2a1) on the dominant vertex
constexpr double kTriA2 = 0.091576213509770743;  // orbit 2
constexpr double kTriW1 = 0.22338158967801147;
constexpr double kTriW2 = 0.10995174365532187;

// barycentric coordinate of quadrature point q (0..5) at local vertex b (0..2)
__host__ __device__ constexpr double tri6_phi(int q, int b) {
  return (q < 3) ? ((q == b) ? 1.0 - 2.0 * kTriA1 : kTriA1) : ((q - 3 == b) ? 1.0 - 2.0 * kTriA2 : kTriA2);
}
__host__ __device__ constexpr double tri6_w(int q) { return q < 3 ? kTriW1 : kTriW2; }
// The rule is symmetric: w_q phi_b(q) = tri6_w_common(q) + tri6_w_own(q) [b == tri6_own(q)].
__host__ __device__ constexpr int tri6_own(int q) { return q < 3 ? q : q - 3; }
__host__ __device__ constexpr double tri6_w_common(int q) { return tri6_w(q) * (q < 3 ? kTriA1 : kTriA2); }
__host__ __device__ constexpr double tri6_w_own(int q) { return tri6_w(q) * (1.0 - 3.0 * (q < 3 ? kTriA1 : kTriA2)); }

// Gauss-Legendre 4-point rule on [-1, 1] (gauss.h:44-54).
constexpr double kGL4x0 = 0.86113631159405258, kGL4x1 = 0.33998104358485626;
constexpr double kGL4w0 = 0.34785484513745385, kGL4w1 = 0.65214515486254614;
__host__ __device__ constexpr double gl4_x(int i) {
  return i == 0 ? kGL4x0 : i == 1 ? kGL4x1 : i == 2 ? -kGL4x1 : -kGL4x0;
}
__host__ __device__ constexpr double gl4_w(int i) { return (i == 0 || i == 3) ? kGL4w0 : kGL4w1; }

constexpr float kEps = 1e-3f;  // r clamp of the reference kernels (potential.h:16-23)

// ---- packed FP32 pairs (sm_100 f32x2 arithmetic) ---------------------------
// One instruction applies the same IEEE round-to-nearest operation to both
// lanes of a float2, so a packed expression gives bit-identical results to
// the two scalar ones while issuing half the instructions.
// e / d for 0 <= e < 2^24 and d >= 1, with rd = 1.f / d computed once by the
// caller: a float multiply and one correction step instead of an integer
// division sequence in the inner loops.
__device__ __forceinline__ int div_by(int e, int d, float rd) {
  int q = __float2int_rz((float)e * rd);
  const int r = e - q * d;
  q += (r >= d) - (r < 0);
  return q;
}

__device__ __forceinline__ float2 f2_fma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 f2_mul(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f2_add(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f2_sub(float2 a, float2 b) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
constexpr double kPi = 3.14159265358979323846;
constexpr float kInv4Pi = (float)(1.0 / (4.0 * kPi));

// ---- geometry -------------------------------------------------------------
// One record per triangle, 32 words.  Quadrature points in rule order
// (q = 0..5), unit normal, centroid, area = J/2, and the three vertex ids.
struct __align__(16) TriRec {
  float qp[18];
  float n[3];
  float c[3];
  float area;
  int v[3];
  float h;  // n . v0 (plane offset)
  int leave;  // sorted order: bit b set if the next triangle of the block does not hold v[b] in slot b
};
static_assert(sizeof(TriRec) == 128, "TriRec must be 128 bytes");

// Burton-Miller companion record, sorted order: the points of the 3-point
// degree-2 triangle rule (phi = 2/3 at the point's own vertex, 1/6 at the
// others; weights 1/3) used by the <2,3> Burton-Miller bindings, and the
// surface curls n x grad(phi_b) of the three P1 functions (rows b).
struct __align__(16) BmRec {
  float qp[9];
  float curl[9];
  float pad[2];
};
static_assert(sizeof(BmRec) == 80, "BmRec must be 80 bytes");

constexpr int kTile = 16;               // triangles per geometry tile
constexpr int kTileCorners = 3 * kTile;  // 48

// Per-tile local-vertex tables, one per 16-triangle tile of the sorted order.
struct __align__(16) TileRec {
  int nlv;                       // number of distinct vertices in the tile
  int ntri;                      // triangles in the tile (last tile may be short)
  int pad0, pad1;
  int vid[kTileCorners];         // global vertex id of each local vertex
  uint8_t corner_lv[kTileCorners];     // local vertex of corner (3*t + a)
  uint8_t lv_ptr[kTileCorners + 4];    // CSR: corners of local vertex l are lv_corner[lv_ptr[l]..lv_ptr[l+1])
  uint8_t lv_corner[kTileCorners];
  uint8_t pad2[12];
};
static_assert(sizeof(TileRec) % 16 == 0, "TileRec alignment");

// Blocks of 32 sorted triangles, ordered within the block as paths over shared
// edges, with the local vertices of each triangle permuted (in the sorted
// records only) so that a vertex kept from one triangle to the next stays in
// its slot.  Corner 32 a + t is slot a of the block's triangle t.
constexpr int kBlock = 32;
constexpr int kBlockCorners = 3 * kBlock;
struct __align__(16) BlockRec {
  int nlv;                         // distinct vertices
  int most;                        // most corners of one vertex
  int pad[2];
  int vid[kBlockCorners];          // global vertex id of each local vertex
  uint8_t ptr[kBlockCorners + 4];  // corners of local vertex l: corner[ptr[l]..ptr[l+1])
  uint8_t corner[kBlockCorners];
  uint8_t pad2[12];
};
static_assert(sizeof(BlockRec) % 16 == 0, "BlockRec alignment");

// Header at the start of the geometry workspace.  All offsets in bytes from
// the start of the workspace.
struct GeomHeader {
  uint32_t magic;
  int nv, nt, ntiles;
  int n_edge, n_vert;  // ordered singular pairs sharing 2 / 1 vertices
  int max_valence;
  int err;  // status word: set to 1 by an assembly kernel whose bounded wait expired on this geometry
  uint64_t off_vertices;   // float[nv*3] (copy of the input)
  uint64_t off_triangles;  // int[nt*3] (copy of the input)
  uint64_t off_perm;       // int[nt]  sorted position -> triangle id
  uint64_t off_trirec;     // TriRec[nt] in sorted order
  uint64_t off_trirec_orig;  // TriRec[nt] in input order
  uint64_t off_tiles;      // TileRec[ntiles]
  uint64_t off_edge_pairs;  // int2[n_edge]  (test tri, trial tri), input ids
  uint64_t off_vert_pairs;  // int2[n_vert], first those with test < trial (half of them)
  uint64_t off_normals;    // float[nt*3]
  uint64_t off_curls;      // float[nt*9]   rows: n x grad(phi_b)
  uint64_t off_bmrec;      // BmRec[nt] in sorted order
  uint64_t off_slots;      // int[nt]  sorted position -> local vertex of each slot (2 bits each) and leave bits
  uint64_t off_blocks;     // BlockRec[nblocks]
  uint64_t bytes;
};
constexpr uint32_t kGeomMagic = 0x42454D34u;  // "BEM4"

// Device-side view of a built geometry.
struct GeomView {
  int nv, nt, ntiles, nblocks, n_edge, n_vert;
  const float* vertices;
  const int* triangles;
  const int* perm;
  const int* slots;        // sorted position -> input-order local vertex of slot a in bits 2a, 2a + 1
  const TriRec* rec;       // sorted order
  const TriRec* rec_orig;  // input order
  const TileRec* tiles;
  const BlockRec* blocks;
  const int2* edge_pairs;
  const int2* vert_pairs;
  const float* normals;
  const float* curls;
  const BmRec* bm;         // sorted order
  int* err;                // the header's status word (GeomHeader::err)
};

// Symmetric regular-pair work units (test block g, trial block j >= g) in
// order: test block g owns the n - g trial blocks from itself on, so
// U(g) = g n - g (g - 1) / 2 units come before it.
__device__ __forceinline__ long long tile_units_before(long long g, long long n) { return g * n - g * (g - 1) / 2; }

__device__ __forceinline__ int tile_group_of(long long pos, int n) {
  const double b = 2.0 * n + 1.0;
  const double disc = b * b - 8.0 * (double)pos;
  long long g = (long long)((b - sqrt(disc > 0.0 ? disc : 0.0)) * 0.5);
  if (g < 0) g = 0;
  if (g > n - 1) g = n - 1;
  while (g + 1 < n && tile_units_before(g + 1, n) <= pos) g++;
  while (g > 0 && tile_units_before(g, n) > pos) g--;
  return (int)g;
}

// ---- small math -------------------------------------------------------------
// FP64 phases of touching triangles are small (k times their size): Taylor sums
// up to x^15 and x^16, below 1e-16 off for |x| <= pi / 4; the library beyond.
__device__ __forceinline__ void sincos_touch(double x, double* s, double* c) {
  if (fabs(x) > 0.78539816339744831) {
    sincos(x, s, c);
    return;
  }
  const double t = x * x;
  double p = -1.0 / 1307674368000.0;
  p = fma(p, t, 1.0 / 6227020800.0);
  p = fma(p, t, -1.0 / 39916800.0);
  p = fma(p, t, 1.0 / 362880.0);
  p = fma(p, t, -1.0 / 5040.0);
  p = fma(p, t, 1.0 / 120.0);
  p = fma(p, t, -1.0 / 6.0);
  *s = fma(p * t, x, x);
  double q = 1.0 / 20922789888000.0;
  q = fma(q, t, -1.0 / 87178291200.0);
  q = fma(q, t, 1.0 / 479001600.0);
  q = fma(q, t, -1.0 / 3628800.0);
  q = fma(q, t, 1.0 / 40320.0);
  q = fma(q, t, -1.0 / 720.0);
  q = fma(q, t, 1.0 / 24.0);
  q = fma(q, t, -0.5);
  *c = fma(q, t, 1.0);
}

// sine and cosine of a touching pair's phase
template <typename R>
__device__ __forceinline__ void sincos_t(R x, R* s, R* c);
template <>
__device__ __forceinline__ void sincos_t<double>(double x, double* s, double* c) {
  sincos_touch(x, s, c);
}
// FP32 (edge and vertex pairs of the touching-pair kernels): the hardware
// approximation, accurate to a few 1e-7 absolute for the |k r| <= ~1 of
// touching triangles (the regular kernels use it at larger arguments).
template <>
__device__ __forceinline__ void sincos_t<float>(float x, float* s, float* c) {
  __sincosf(x, s, c);
}

// Totals over the warp of N values per lane: value v in total[v] (one warp's
// shared memory, ROUNDUP(N, 32) entries), visible to all lanes on return.
// Groups of 32 values by a transpose: every round halves the values a lane
// keeps, so a group costs 31 shuffles instead of 5 per value.
template <int N, typename R>
__device__ __forceinline__ void warp_totals(const R (&v)[N], R* total) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int g = 0; g < N; g += 32) {
    R t[32];
#pragma unroll
    for (int i = 0; i < 32; i++) t[i] = g + i < N ? v[g + i < N ? g + i : 0] : R(0);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      const bool hi = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < o; i++) {
        const R send = hi ? t[i] : t[i + o];
        const R keep = hi ? t[i + o] : t[i];
        t[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    total[g + lane] = t[0];
  }
  __syncwarp();
}

// 1 / r and r from r^2 (r clamped to kEps as in potential.h).
template <typename R>
__device__ __forceinline__ void inv_dist(R r2, R* r, R* inv_r);
template <>
__device__ __forceinline__ void inv_dist<double>(double r2, double* r, double* inv_r) {
  r2 = fmax(r2, (double)kEps * (double)kEps);
  const double ri = rsqrt(r2);
  *inv_r = ri;
  *r = r2 * ri;
}
template <>
__device__ __forceinline__ void inv_dist<float>(float r2, float* r, float* inv_r) {
  const float ri = fminf(rsqrtf(r2), 1.0f / kEps);
  *inv_r = ri;
  *r = fmaxf(r2 * ri, kEps);
}

struct f3 {
  float x, y, z;
};
__device__ __forceinline__ f3 make3(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 sub(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ float dot3(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

struct d3 {
  double x, y, z;
};
__device__ __forceinline__ d3 sub(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double dot3(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 cross3(d3 a, d3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

__device__ __forceinline__ void atomic_add_c64(float2* p, float re, float im) {
  atomicAdd(p, make_float2(re, im));  // vector red.global.add.v2.f32 (sm_90+)
}

}  // namespace bemb

namespace bemb {
// process-wide count of kernel launches issued by this library (host side)
void count_launch();
void count_launches(unsigned long long n);
unsigned long long launch_count();
}  // namespace bemb

// error-checking helper for host code inside the library; a reported error is
// cleared, or the next call's check of its launches would report it once more
#define BEM_CUDA_TRY(expr)                          \
  do {                                              \
    cudaError_t _e = (expr);                        \
    if (_e != cudaSuccess) {                        \
      cudaGetLastError();                           \
      return BEM_ERR_CUDA;                          \
    }                                               \
  } while (0)

namespace bemb {
// Set-up of a kernel once on each device (one static object per kernel or per
// group of kernels set up together).  The
// limit of a kernel's dynamic shared memory belongs to the kernel on the current
// device and to all host threads: it is set once, to the largest size that any
// launch asks for, since a thread that set its own call's size could lower it
// between another thread's call and that call's launch.
class DeviceOnce {
 public:
  // set(): a bem_status
  template <typename F>
  int operator()(F&& set) {
    int dev = 0;
    BEM_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;  // beyond: each time
    if (done_.load(std::memory_order_acquire) & bit) return BEM_OK;
    const int rc = set();
    if (rc == BEM_OK) done_.fetch_or(bit, std::memory_order_release);
    return rc;
  }
  // the limit of dynamic shared memory
  template <typename Kernel>
  int shared_memory(Kernel kernel, size_t bytes) {
    return (*this)([&]() -> int {
      BEM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
      return BEM_OK;
    });
  }

 private:
  std::atomic<unsigned long long> done_{0};
};
}  // namespace bemb
