// Dense Galerkin assembly of the Helmholtz single-layer (V) and double-layer
// (K) matrices in the P1 vertex basis, plus the P1 mass matrix.
//
// Reference behaviour (file:line inside the NeuralAT project):
//   regular pairs     src/bem/cuda/bind.cu:67-79, integrand.h:187-235,280-329
//   singular pairs    src/bem/cuda/bind.cu:81-152, integrand.h:63-185,331-394
//   kernels           src/bem/cuda/include/potential.h:18-32 (r >= 1e-3 clamp)
//   mass matrix       src/bem/cuda/bind.cu:10-21, integrand.h:257-278
//
// Design (B200): the reference launches one block per test triangle, sweeps
// every trial triangle with one thread each, recomputes r and exp(ikr)
// separately for V and for K, and scatters 18 float atomics per pair into the
// N x N matrix.  Here:
//   * one pass evaluates each quadrature-point pair once for BOTH operators
//     (shared r, rsqrt and sincos), with the 6-point rule's constant weights
//     folded into immediate FMA operands;
//   * V and K together (regular_strip_vk_kernel): each unordered pair once, a
//     warp walks a 32-triangle test block (one triangle per lane) along the
//     trial triangles and sums their columns in registers (strip.cuh); one
//     operator alone (regular_vk_kernel): a CTA owns 32 test triangles (one
//     per lane) x one 16-triangle trial tile, the 8 warps broadcasting their
//     trial triangles from shared memory, and pair blocks go to a
//     shared-memory "corner" slab (test corner x trial corner);
//   * both reduce the corners on chip onto distinct vertices, so each matrix
//     entry receives about one vector atomic per triangle pair instead of the
//     reference's 18 scalar atomics;
//   * touching pairs are masked out of the regular pass and integrated by
//     separate Sauter-Schwab kernels (coincident pairs in FP64), one warp per
//     pair over a precomputed pair list (no O(T^2) adjacency scan).

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "async_copy.cuh"
#include "bem_common.cuh"
#include "sauter_schwab.cuh"
#include "strip.cuh"

namespace bemb {

int geom_view(const void* geom, GeomView* v, GeomHeader* out_hdr);

extern int g_tc_promote;    // tensor-core matvec accumulator segment (tc_matvec.cu)
extern int g_gmres_reorth;  // Gram-Schmidt passes of the Arnoldi step (linalg.cu)
extern int g_arn_max_cluster;  // largest Arnoldi cluster size (linalg.cu)
extern int g_arn_mode;         // Arnoldi step variant (linalg.cu)
extern int g_gmres_block;      // block Krylov space for several right-hand sides (linalg.cu)
extern int g_tc_wait_us;       // bounded-wait limit of the tensor-core kernels (tc_matvec.cu)
extern std::atomic<int> g_tc_skip_fill;  // test hook of the tensor-core kernel (tc_matvec.cu)

namespace {
extern int g_tune_chunk;
extern int g_tune_ctas_per_sm;
}  // namespace

namespace {

// ---------------------------------------------------------------------------
// Regular triangle pairs.
// ---------------------------------------------------------------------------
constexpr int kRegThreads = 256;
constexpr int kRegWarps = kRegThreads / 32;
constexpr int kTestTris = 32;                  // one test triangle per lane
constexpr int kTestCorners = 3 * kTestTris;     // 96
constexpr int kSlotStride = kTileCorners + 1;   // 49 float2: conflict-free column writes

template <bool DO_V, bool DO_K>
struct RegSmem {
  float2 slotV[DO_V ? kTestCorners : 1][kSlotStride];
  float2 slotK[DO_K ? kTestCorners : 1][kSlotStride];
  TriRec trial[kTile];
  TileRec tileJ;
  TileRec tileI[2];
};

// 3x3 P1 blocks of one (test, trial) pair under the 6x6 point rule:
//   aV[3a+b] = sum_pq C_ap C_bq e^{ikr}/r,
//   aK[3a+b] = sum_pq C_ap C_bq dn_p (c + kr s + i(s - kr c)) / r^3,
// with C_aq = w_q phi_a(q), dn_p = n_j . (y - x_p) (constant over the trial
// plane), r clamped to >= 1e-3 (potential.h:21-23).  The 1/(4 pi), the
// areas and the double layer's minus sign are applied by the caller.
template <bool DO_V, bool DO_K>
__device__ __forceinline__ void pair_block(const float (&xq)[18], const float (&yq)[18], float njx, float njy,
                                           float njz, float cjx, float cjy, float cjz, float k, float2 (&aV)[9],
                                           float2 (&aK)[9]) {
#pragma unroll
  for (int e = 0; e < 9; e++) {
    aV[e] = make_float2(0.f, 0.f);
    aK[e] = make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int p = 0; p < 6; p++) {
    const float px = xq[3 * p], py = xq[3 * p + 1], pz = xq[3 * p + 2];
    const float dn = njx * (cjx - px) + njy * (cjy - py) + njz * (cjz - pz);
    float2 tV[3], tK[3];
#pragma unroll
    for (int b = 0; b < 3; b++) {
      tV[b] = make_float2(0.f, 0.f);
      tK[b] = make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const float dx = yq[3 * q] - px, dy = yq[3 * q + 1] - py, dz = yq[3 * q + 2] - pz;
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const float rinv = fminf(rsqrtf(r2), 1.0f / kEps);
      const float r = fmaxf(r2 * rinv, kEps);
      float s, c;
      __sincosf(k * r, &s, &c);
      const float gvr = c * rinv, gvi = s * rinv;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const float w = (float)(tri6_w(q) * tri6_phi(q, b));
        if (DO_V) {
          tV[b].x = fmaf(w, gvr, tV[b].x);
          tV[b].y = fmaf(w, gvi, tV[b].y);
        }
      }
      if (DO_K) {
        const float rinv2 = rinv * rinv;
        const float gkr = fmaf(k, s, gvr) * rinv2;   // (c + kr s) / r^3
        const float gki = fmaf(-k, c, gvi) * rinv2;  // (s - kr c) / r^3
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const float w = (float)(tri6_w(q) * tri6_phi(q, b));
          tK[b].x = fmaf(w, gkr, tK[b].x);
          tK[b].y = fmaf(w, gki, tK[b].y);
        }
      }
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float wa = (float)(tri6_w(p) * tri6_phi(p, a));
      const float wk = wa * dn;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        if (DO_V) {
          aV[3 * a + b].x = fmaf(wa, tV[b].x, aV[3 * a + b].x);
          aV[3 * a + b].y = fmaf(wa, tV[b].y, aV[3 * a + b].y);
        }
        if (DO_K) {
          aK[3 * a + b].x = fmaf(wk, tK[b].x, aK[3 * a + b].x);
          aK[3 * a + b].y = fmaf(wk, tK[b].y, aK[3 * a + b].y);
        }
      }
    }
  }
}

__device__ __forceinline__ void copy_words(void* dst, const void* src, int bytes, int tid, int nthreads) {
  const int4* s = (const int4*)src;
  int4* d = (int4*)dst;
  for (int i = tid; i < bytes / 16; i += nthreads) d[i] = s[i];
}

// Work item = (group of 32 test triangles = 2 tiles) x (chunk of `chunk`
// trial tiles).  Items are dealt round-robin to a persistent grid.
// One work item: test group `grp` (32 triangles = 2 tiles) against the trial
// tiles [ch * chunk, ch * chunk + chunk).
template <bool DO_V, bool DO_K>
__device__ __forceinline__ void regular_item(RegSmem<DO_V, DO_K>& sm, const GeomView& g, float k,
                                             float2* __restrict__ V, float2* __restrict__ K, float v_scale,
                                             float k_scale, int grp, int ch, int chunk) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = g.nt, nv = g.nv;
  {
    const int tile0 = 2 * grp;
    const bool has_t1 = tile0 + 1 < g.ntiles;

    // test triangle of this lane (all warps hold the same 32)
    const int ti = grp * kTestTris + lane;
    const bool valid_i = ti < nt;
    const TriRec& ri = g.rec[valid_i ? ti : nt - 1];
    float xq[18];
#pragma unroll
    for (int e = 0; e < 18; e++) xq[e] = ri.qp[e];
    const float area_i = ri.area;
    const int iv0 = ri.v[0], iv1 = ri.v[1], iv2 = ri.v[2];

    __syncthreads();  // previous item's gather has finished with tileI
    copy_words(&sm.tileI[0], &g.tiles[tile0], sizeof(TileRec), tid, kRegThreads);
    if (has_t1) copy_words(&sm.tileI[1], &g.tiles[tile0 + 1], sizeof(TileRec), tid, kRegThreads);

    const int jt_begin = ch * chunk;
    const int jt_end = min(jt_begin + chunk, g.ntiles);
    for (int jt = jt_begin; jt < jt_end; jt++) {
      __syncthreads();  // gather of the previous trial tile is done with the slots
      copy_words(&sm.tileJ, &g.tiles[jt], sizeof(TileRec), tid, kRegThreads);
      const int ntriJ = min(kTile, nt - jt * kTile);
      copy_words(sm.trial, &g.rec[jt * kTile], ntriJ * (int)sizeof(TriRec), tid, kRegThreads);
      __syncthreads();

      // ---- compute: each warp takes trial triangles warp and warp + 8 ----
#pragma unroll 1
      for (int tt = warp; tt < ntriJ; tt += kRegWarps) {
        const TriRec& rj = sm.trial[tt];
        float yq[18];
#pragma unroll
        for (int e = 0; e < 18; e++) yq[e] = rj.qp[e];
        float2 aV[9], aK[9];
        pair_block<DO_V, DO_K>(xq, yq, rj.n[0], rj.n[1], rj.n[2], rj.c[0], rj.c[1], rj.c[2], k, aV, aK);
        const int j0 = rj.v[0], j1 = rj.v[1], j2 = rj.v[2];
        const bool touching = (iv0 == j0) | (iv0 == j1) | (iv0 == j2) | (iv1 == j0) | (iv1 == j1) | (iv1 == j2) |
                              (iv2 == j0) | (iv2 == j1) | (iv2 == j2);
        const float aa = (valid_i && !touching) ? area_i * rj.area : 0.f;
        const float sv = aa * v_scale, sk = aa * k_scale;
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
          for (int b = 0; b < 3; b++) {
            if (DO_V) sm.slotV[3 * lane + a][3 * tt + b] = make_float2(aV[3 * a + b].x * sv, aV[3 * a + b].y * sv);
            if (DO_K) sm.slotK[3 * lane + a][3 * tt + b] = make_float2(aK[3 * a + b].x * sk, aK[3 * a + b].y * sk);
          }
      }
      __syncthreads();

      // ---- reduce corner slots onto distinct vertices, one atomic per entry ----
      // Pass 1, in place: for every trial corner column, the row of test
      // vertex A's first corner gets the sum over A's test corners (corner
      // rows of different vertices are disjoint); pass 2: entry (A, B) sums
      // B's trial corners along that row.
      const int nI0 = sm.tileI[0].nlv;
      const int nI1 = has_t1 ? sm.tileI[1].nlv : 0;
      const int nJ = sm.tileJ.nlv;
      const int ncol = 3 * ntriJ;
      const float rcol = 1.f / (float)ncol, rJ = 1.f / (float)(nJ > 0 ? nJ : 1);
      for (int e = tid; e < (nI0 + nI1) * ncol; e += kRegThreads) {
        const int ai = div_by(e, ncol, rcol);
        const int col = e - ai * ncol;
        const int s = ai >= nI0;
        const int a = ai - s * nI0;
        const TileRec& TI = sm.tileI[s];
        const int ca0 = TI.lv_ptr[a], ca1 = TI.lv_ptr[a + 1];
        const int rep = s * kTileCorners + TI.lv_corner[ca0];
        float2 v = make_float2(0.f, 0.f), kk = make_float2(0.f, 0.f);
        if (DO_V) v = sm.slotV[rep][col];
        if (DO_K) kk = sm.slotK[rep][col];
        for (int ca = ca0 + 1; ca < ca1; ca++) {
          const int row = s * kTileCorners + TI.lv_corner[ca];
          if (DO_V) {
            v.x += sm.slotV[row][col].x;
            v.y += sm.slotV[row][col].y;
          }
          if (DO_K) {
            kk.x += sm.slotK[row][col].x;
            kk.y += sm.slotK[row][col].y;
          }
        }
        if (DO_V) sm.slotV[rep][col] = v;
        if (DO_K) sm.slotK[rep][col] = kk;
      }
      __syncthreads();
      for (int e = tid; e < (nI0 + nI1) * nJ; e += kRegThreads) {
        const int ai = div_by(e, nJ, rJ);
        const int b = e - ai * nJ;
        const int s = ai >= nI0;
        const int a = ai - s * nI0;
        const TileRec& TI = sm.tileI[s];
        const int rep = s * kTileCorners + TI.lv_corner[TI.lv_ptr[a]];
        float2 acc_v = make_float2(0.f, 0.f), acc_k = make_float2(0.f, 0.f);
        const int cb0 = sm.tileJ.lv_ptr[b], cb1 = sm.tileJ.lv_ptr[b + 1];
        for (int cb = cb0; cb < cb1; cb++) {
          const int col = sm.tileJ.lv_corner[cb];
          if (DO_V) {
            acc_v.x += sm.slotV[rep][col].x;
            acc_v.y += sm.slotV[rep][col].y;
          }
          if (DO_K) {
            acc_k.x += sm.slotK[rep][col].x;
            acc_k.y += sm.slotK[rep][col].y;
          }
        }
        const size_t idx = (size_t)TI.vid[a] * nv + sm.tileJ.vid[b];
        if (DO_V) atomicAdd(&V[idx], acc_v);
        if (DO_K) atomicAdd(&K[idx], acc_k);
      }
    }
  }
}

// Single problem: items dealt round-robin to a persistent grid.
template <bool DO_V, bool DO_K>
__global__ void __launch_bounds__(kRegThreads, 2)
    regular_vk_kernel(GeomView g, float k, float2* __restrict__ V, float2* __restrict__ K, float v_scale,
                      float k_scale, int chunk, int n_chunks, int n_items) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RegSmem<DO_V, DO_K>& sm = *reinterpret_cast<RegSmem<DO_V, DO_K>*>(smem_raw);
  for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
    const int grp = item / n_chunks;
    regular_item<DO_V, DO_K>(sm, g, k, V, K, v_scale, k_scale, grp, item - grp * n_chunks, chunk);
  }
}

// ---------------------------------------------------------------------------
// Symmetric evaluation of the regular pairs (V and K together).  G(|x - y|)
// is symmetric, so each unordered non-touching pair {i, j} is evaluated once
// and scattered both ways:
//   V_ji = V_ij^T,
//   K_ij uses the trial plane of j (dn_j(p) = n_j . (c_j - x_p)),
//   K_ji uses the plane of i at the trial points (dn_i(q) = n_i . (c_i - y_q)),
// both from the same r, sincos and kernel values, on a warp's strip walk
// (strip.cuh).
//
// Bound by the FP32 pipe.  The rule is symmetric, w_q phi_b(q) = common(q) +
// own(q) [b = own vertex of q], so with g_b and h_b the values at the two
// points of vertex b the trial sums are
//   t_b = own_1 (g_b + rho h_b) + common_1 sum_c (g_c + sigma h_c),
// and likewise over the test points: one sum per own vertex and one common
// sum, combined when a column is flushed.  About 37 FP32-pipe operations per
// point pair against 42 for weights applied point by point.  The arithmetic
// runs on packed pairs (the two points of a trial vertex): the same rounding
// as scalar operations in fewer issued instructions.
//
// Measured on B200 with 20 480 triangles: 12.6 ms (both operators; FP32 pipe
// 64 % of its cycles, issue 63 %), of which 1.6 ms are the column reductions,
// against 19.0 ms for 16 x 16-triangle tiles whose 3 x 3 blocks all went
// through shared memory between block barriers.  Two CTAs of four warps per SM
// with everything unrolled (no spills) took 14.6 ms for the whole assembly with
// one item per warp (13.5 in rounds), three CTAs at 168 registers 15.1 ms, four at 128 registers 18.2 ms (spills).
// ---------------------------------------------------------------------------
constexpr float kRho = (float)(tri6_w_own(3) / tri6_w_own(0));
constexpr float kSigma = (float)(tri6_w_common(3) / tri6_w_common(0));
constexpr float kTau = (float)(tri6_w_common(0) / tri6_w_own(0));

// A bounded wait of the assembly kernels expired somewhere in this process
// (read and cleared by bem_assembly_status).  The waits themselves check the
// status word of the geometry they assemble (GeomView::err), so an expiry on
// one geometry does not affect assemblies of other geometries.
__device__ int g_asm_err;

using VkWarp = StripWarp<18, false>;

struct VkStrip {
  float k, v_scale, k_scale;
  float2* V;
  float2* K;
  // sums of the open columns: own-vertex part [3 a + b] and common part [b]
  // of V_ij, K_ij and K_ji^T
  float2 eV[9], eK[9], eM[9], cV[3], cK[3], cM[3];

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int e = 0; e < 9; e++) eV[e] = eK[e] = eM[e] = make_float2(0.f, 0.f);
#pragma unroll
    for (int b = 0; b < 3; b++) cV[b] = cK[b] = cM[b] = make_float2(0.f, 0.f);
  }

  __device__ __forceinline__ void load(VkWarp& sw, const StripTest& t, const GeomView& g, int lane) {
    const TriRec& r = g.rec[min(t.grp * kBlock + lane, g.nt - 1)];
#pragma unroll
    for (int e = 0; e < 18; e++) sw.xs[e][lane] = r.qp[e];
  }

  __device__ __forceinline__ void pair(const VkWarp& sw, const StripTest& t, const TriRec& rj, const BmRec&, float w,
                                       int lane) {
    const float4* r4 = (const float4*)&rj;
    const float4 q0 = r4[0], q1 = r4[1], q2 = r4[2], q3 = r4[3], q4 = r4[4], q5 = r4[5];
    // the points of trial vertex b: orbit 1 and orbit 2
    const float2 yx[3] = {{q0.x, q2.y}, {q0.w, q3.x}, {q1.z, q3.w}};
    const float2 yy[3] = {{q0.y, q2.z}, {q1.x, q3.y}, {q1.w, q4.x}};
    const float2 yz[3] = {{q0.z, q2.w}, {q1.y, q3.z}, {q2.x, q4.y}};
    const float njx = q4.z, njy = q4.w, njz = q5.x, cjx = q5.y, cjy = q5.z, cjz = q5.w;
    float2 dq[3];  // n_i . (c_i - y_q)
    float dr[3];   // rho times the second orbit's
#pragma unroll
    for (int b = 0; b < 3; b++)
      dq[b] = f2_fma(f2(t.nx), f2_sub(f2(t.cx), yx[b]),
                     f2_fma(f2(t.ny), f2_sub(f2(t.cy), yy[b]), f2_mul(f2(t.nz), f2_sub(f2(t.cz), yz[b]))));
#pragma unroll
    for (int b = 0; b < 3; b++) dr[b] = kRho * dq[b].y;
    const float2 k2 = f2(k), nk2 = f2(-k);
#pragma unroll
    for (int o = 0; o < 2; o++) {  // orbit of the test points
      const float so = w * (float)(o == 0 ? tri6_w_own(0) * tri6_w_own(0) : tri6_w_own(3) * tri6_w_own(0));
      const float sc = w * (float)(o == 0 ? tri6_w_common(0) * tri6_w_own(0) : tri6_w_common(3) * tri6_w_own(0));
      const float2 so2 = f2(so), sc2 = f2(sc);
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const float px = sw.xs[9 * o + 3 * a][lane], py = sw.xs[9 * o + 3 * a + 1][lane],
                    pz = sw.xs[9 * o + 3 * a + 2][lane];
        const float dn = njx * (cjx - px) + njy * (cjy - py) + njz * (cjz - pz);
        float2 tV[3], tK[3], tM[3];
        float2 sVr, sVi, sKr, sKi, sMr, sMi;  // sums over the vertices, per orbit
        float2 ri[3], kr[3], s[3], c[3];
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const float2 dx = f2_sub(yx[b], f2(px)), dy = f2_sub(yy[b], f2(py)), dz = f2_sub(yz[b], f2(pz));
          float2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
          r2.x = fmaxf(r2.x, kEps * kEps);  // r >= 1e-3, to a rounding
          r2.y = fmaxf(r2.y, kEps * kEps);
          ri[b] = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
          kr[b] = f2_mul(k2, f2_mul(r2, ri[b]));
        }
#pragma unroll
        for (int b = 0; b < 3; b++) {
          __sincosf(kr[b].x, &s[b].x, &c[b].x);
          __sincosf(kr[b].y, &s[b].y, &c[b].y);
        }
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const float2 ri2 = f2_mul(ri[b], ri[b]);
          const float2 gr = f2_mul(c[b], ri[b]), gi = f2_mul(s[b], ri[b]);  // e^{ikr} / r
          const float2 hr = f2_mul(f2_fma(k2, s[b], gr), ri2), hi = f2_mul(f2_fma(nk2, c[b], gi), ri2);  // (1 - ikr) e^{ikr} / r^3
          tV[b] = make_float2(fmaf(kRho, gr.y, gr.x), fmaf(kRho, gi.y, gi.x));
          tK[b] = make_float2(fmaf(kRho, hr.y, hr.x), fmaf(kRho, hi.y, hi.x));
          tM[b] = make_float2(fmaf(dr[b], hr.y, dq[b].x * hr.x), fmaf(dr[b], hi.y, dq[b].x * hi.x));
          sVr = b ? f2_add(sVr, gr) : gr;
          sVi = b ? f2_add(sVi, gi) : gi;
          sKr = b ? f2_add(sKr, hr) : hr;
          sKi = b ? f2_add(sKi, hi) : hi;
          sMr = b ? f2_fma(dq[b], hr, sMr) : f2_mul(dq[b], hr);
          sMi = b ? f2_fma(dq[b], hi, sMi) : f2_mul(dq[b], hi);
        }
        const float2 sV = make_float2(fmaf(kSigma, sVr.y, sVr.x), fmaf(kSigma, sVi.y, sVi.x));
        const float2 sK = make_float2(fmaf(kSigma, sKr.y, sKr.x), fmaf(kSigma, sKi.y, sKi.x));
        const float2 sM = make_float2(fmaf(kSigma, sMr.y, sMr.x), fmaf(kSigma, sMi.y, sMi.x));
        const float2 sod = f2(so * dn), scd = f2(sc * dn), tau = f2(kTau);
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const float2 v = f2_fma(tau, sV, tV[b]), kk = f2_fma(tau, sK, tK[b]), m = f2_fma(tau, sM, tM[b]);
          eV[3 * a + b] = f2_fma(so2, v, eV[3 * a + b]);
          cV[b] = f2_fma(sc2, v, cV[b]);
          eK[3 * a + b] = f2_fma(sod, kk, eK[3 * a + b]);
          cK[b] = f2_fma(scd, kk, cK[b]);
          eM[3 * a + b] = f2_fma(so2, m, eM[3 * a + b]);
          cM[b] = f2_fma(sc2, m, cM[b]);
        }
      }
    }
  }

  template <int B>
  __device__ __forceinline__ void take(VkWarp& sw, int i, int lane) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float2 v = f2_add(eV[3 * a + B], cV[B]), kk = f2_add(eK[3 * a + B], cK[B]);
      sw.col4[i][32 * a + lane] = make_float4(v.x, v.y, kk.x, kk.y);
      sw.col2[i][32 * a + lane] = f2_add(eM[3 * a + B], cM[B]);
      eV[3 * a + B] = eK[3 * a + B] = eM[3 * a + B] = make_float2(0.f, 0.f);
    }
    cV[B] = cK[B] = cM[B] = make_float2(0.f, 0.f);
  }

  __device__ __forceinline__ void store(const GeomView& g, int A, int B, const float4& s4, const float2& s2) const {
    if (s4.x == 0.f && s4.y == 0.f && s4.z == 0.f && s4.w == 0.f && s2.x == 0.f && s2.y == 0.f) return;
    const size_t ab = (size_t)A * g.nv + B, ba = (size_t)B * g.nv + A;
    const float2 v = make_float2(s4.x * v_scale, s4.y * v_scale);
    atomicAdd(&V[ab], v);
    atomicAdd(&V[ba], v);
    atomicAdd(&K[ab], make_float2(s4.z * k_scale, s4.w * k_scale));
    atomicAdd(&K[ba], make_float2(s2.x * k_scale, s2.y * k_scale));
  }
};

// One problem: a warp takes one item (or, past the grid's size, every
// grid-width-th).
__global__ void __launch_bounds__(kStripThreads, 2)
    regular_strip_vk_kernel(const __grid_constant__ GeomView g, float k, float2* __restrict__ V, float2* __restrict__ K, float v_scale,
                            float k_scale, StripItems P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  VkWarp& sw = reinterpret_cast<VkWarp*>(smem_raw)[threadIdx.x >> 5];
  launch_next();
  strip_init(sw);
  VkStrip pol;
  pol.k = k;
  pol.v_scale = v_scale;
  pol.k_scale = k_scale;
  pol.V = V;
  pol.K = K;
  pol.clear();
  StripTest test;
  unsigned uses = 0;
  const long long warps = (long long)gridDim.x * kStripWarps;
  for (long long item = (long long)blockIdx.x * kStripWarps + (threadIdx.x >> 5); item < P.items; item += warps)
    strip_item(sw, test, g, pol, P, item, uses, &g_asm_err);
}

// ---------------------------------------------------------------------------
// Touching pairs: Sauter-Schwab quadrature (sauter_schwab.cuh) on the reference
// triangle (0,0),(1,0),(1,1) (integrand.h:54-185), shared vertices first
// (integrand.h:351-387).  A warp per pair, the lanes split the 4^4
// Gauss-Legendre points; the sums are transposed over the lanes and added with
// one atomic per entry.  Both triangles start at a shared vertex, so the
// difference is d = y1 F1 + y2 F2 - x1 E1 - x2 E2 in their edges E1 = a1 - a0,
// E2 = a2 - a1 (F of the trial triangle), without the vertices' own size.
//
// What the symmetries save:
//   * coincident pairs (FP64): the six regions are three and their mirrors, so
//     V = T + T^T from three, with |d|^2 from the triangle's metric; (y - x).n
//     vanishes, so K gets the mass term only;
//   * pairs with one common vertex (FP32): the two regions are mirrors, so one
//     sweep of the unordered pair gives V_ij, V_ji = V_ij^T, K_ij and K_ji;
//   * pairs with a common edge (FP32) have no such symmetry: ordered pairs.
// All pairs go into one launch, so that the types fill the chip together.  It
// may start while the regular pairs' kernel still runs (programmatic launch;
// both only add to the matrices): beside it on small meshes, in the gaps of its
// last round on large ones.  Measured on B200, the three types together: 20 480
// triangles 705 us (coincident 389, edge 329 and vertex pairs 515 us before),
// 320 triangles 18 us (19 + 12 + 12, one after the other, before).  More than
// one warp per coincident pair of a small mesh gains nothing.
// ---------------------------------------------------------------------------
constexpr int kTouchThreads = 128;
constexpr int kTouchWarps = kTouchThreads / 32;

struct TouchShared {
  double c[kTouchWarps][32];
  float f[kTouchWarps][64];
};

// Gauss-Legendre point pt of the 4^4 rule on [0,1]^4 and its weight.
template <typename R>
__device__ __forceinline__ void touch_point(int pt, R& xi, R& e1, R& e2, R& e3, R& w) {
  const int i0 = pt >> 6, i1 = (pt >> 4) & 3, i2 = (pt >> 2) & 3, i3 = pt & 3;
  xi = R(0.5) * (R(gl4_x(i0)) + R(1));
  e1 = R(0.5) * (R(gl4_x(i1)) + R(1));
  e2 = R(0.5) * (R(gl4_x(i2)) + R(1));
  e3 = R(0.5) * (R(gl4_x(i3)) + R(1));
  w = R(gl4_w(i0)) * R(gl4_w(i1)) * R(gl4_w(i2)) * R(gl4_w(i3));
}

// Coincident pair (ti, ti).
template <bool DO_V, bool DO_K>
__device__ __forceinline__ void touch_coincident(const GeomView& g, int ti, float k, float2* __restrict__ V,
                                                 float2* __restrict__ K, float v_scale,
                                                 float mass_coeff, double* total) {
  const int lane = threadIdx.x & 31;
  const int v[3] = {g.triangles[3 * ti], g.triangles[3 * ti + 1], g.triangles[3 * ti + 2]};
  double E1[3], E2[3], cr[3];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const double a1 = (double)g.vertices[3 * v[1] + e];
    E1[e] = a1 - (double)g.vertices[3 * v[0] + e];
    E2[e] = (double)g.vertices[3 * v[2] + e] - a1;
  }
  cr[0] = E1[1] * E2[2] - E1[2] * E2[1];
  cr[1] = E1[2] * E2[0] - E1[0] * E2[2];
  cr[2] = E1[0] * E2[1] - E1[1] * E2[0];
  const double J2 = cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2];  // (2 area)^2
  const size_t nv = (size_t)g.nv;
  if (DO_V) {
    const double g11 = E1[0] * E1[0] + E1[1] * E1[1] + E1[2] * E1[2], g22 = E2[0] * E2[0] + E2[1] * E2[1] + E2[2] * E2[2],
                 g12 = 2.0 * (E1[0] * E2[0] + E1[1] * E2[1] + E1[2] * E2[2]);
    const double jw = J2 / 16.0, kk = (double)k;
    double t[12];  // entries (0,0) (0,1) (0,2) (1,1) (1,2) (2,2), (re, im)
#pragma unroll
    for (int e = 0; e < 12; e++) t[e] = 0.0;
    auto region = [&](double x1, double x2, double y1, double y2, double w) {
      const double u = y1 - x1, s = y2 - x2;
      const double r2 = fmax(u * (u * g11 + s * g12) + s * s * g22, (double)kEps * (double)kEps);
      const double ri = rsqrt(r2);
      double sn, cs;
      sincos_touch(kk * (r2 * ri), &sn, &cs);
      const double gr = cs * ri * w, gi = sn * ri * w;
      const double lx[3] = {1.0 - x1, x1 - x2, x2}, ly[3] = {1.0 - y1, y1 - y2, y2};
      int e = 0;
#pragma unroll
      for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = a; b < 3; b++, e++) {
          const double f = lx[a] * ly[b] + ly[a] * lx[b];
          t[2 * e] += f * gr;
          t[2 * e + 1] += f * gi;
        }
    };
#pragma unroll 1
    for (int pt = lane; pt < 256; pt += 32) {
      double xi, e1, e2, e3, w;
      touch_point<double>(pt, xi, e1, e2, e3, w);
      const double e12 = e1 * e2, e123 = e12 * e3, sc = xi * xi * xi * e1 * e1 * e2 * w * jw;
      region(xi, xi * (1.0 - e1 + e12), xi * (1.0 - e123), xi * (1.0 - e1), sc);
      region(xi, xi * (e1 - e12 + e123), xi * (1.0 - e12), xi * (e1 - e12), sc);
      region(xi * (1.0 - e123), xi * (e1 - e123), xi, xi * (e1 - e12), sc);
    }
    warp_totals<12>(t, total);
    if (lane < 9) {
      const int a = lane / 3, b = lane % 3, lo = min(a, b), hi = max(a, b);
      const int e = lo == 0 ? hi : (lo == 1 ? 2 + hi : 5);
      atomicAdd(&V[v[a] * nv + v[b]], make_float2((float)(total[2 * e] * (double)v_scale),
                                                  (float)(total[2 * e + 1] * (double)v_scale)));
    }
  }
  if (DO_K && mass_coeff != 0.f && lane < 9) {
    // P1 mass block (integrand.h:257-278): area * sum_q w_q phi_a phi_b
    const int a = lane / 3, b = lane % 3;
    double m = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q++) m += tri6_w(q) * tri6_phi(q, a) * tri6_phi(q, b);
    atomicAdd(&K[v[a] * nv + v[b]], make_float2((float)(mass_coeff * 0.5 * sqrt(J2) * m), 0.f));
  }
}

// Pair (ti, tj) with a common edge (NCOMMON = 2), or the unordered pair with one
// common vertex (NCOMMON = 1), which also gives V_ji and K_ji.
template <int NCOMMON, bool DO_V, bool DO_K>
__device__ __forceinline__ void touch_pair(const GeomView& g, int ti, int tj, float k, float2* __restrict__ V,
                                           float2* __restrict__ K, float v_scale, float k_scale, float* total) {
  const int lane = threadIdx.x & 31;
  const int s0 = g.triangles[3 * ti], s1 = g.triangles[3 * ti + 1], s2 = g.triangles[3 * ti + 2];
  const int t0 = g.triangles[3 * tj], t1 = g.triangles[3 * tj + 1], t2 = g.triangles[3 * tj + 2];
  const Perm6 pm = reorder6<NCOMMON>(s0, s1, s2, t0, t1, t2);
  const int vi[3] = {sel3(s0, s1, s2, pm.i0), sel3(s0, s1, s2, pm.i1), sel3(s0, s1, s2, pm.i2)};
  const int vj[3] = {sel3(t0, t1, t2, pm.j0), sel3(t0, t1, t2, pm.j1), sel3(t0, t1, t2, pm.j2)};
  float E1[3], E2[3], F1[3], F2[3];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const float a1 = g.vertices[3 * vi[1] + e], b1 = g.vertices[3 * vj[1] + e];
    E1[e] = a1 - g.vertices[3 * vi[0] + e];
    E2[e] = g.vertices[3 * vi[2] + e] - a1;
    F1[e] = b1 - g.vertices[3 * vj[0] + e];
    F2[e] = g.vertices[3 * vj[2] + e] - b1;
  }
  float ni[3], nj[3];  // unit normals
#pragma unroll
  for (int e = 0; e < 3; e++) {
    ni[e] = g.normals[3 * ti + e];
    nj[e] = g.normals[3 * tj + e];
  }
  auto twice_area = [](const float (&a)[3], const float (&b)[3]) {
    const float x = a[1] * b[2] - a[2] * b[1], y = a[2] * b[0] - a[0] * b[2], z = a[0] * b[1] - a[1] * b[0];
    return sqrtf(x * x + y * y + z * z);
  };
  const float jw = twice_area(E1, E2) * twice_area(F1, F2) / 16.f;
  // V_ij (9), K_ij (9) and, for a common vertex, K_ji^T (9), (re, im), by re-ordered slot 3 a + b
  constexpr bool kMirror = NCOMMON == 1;
  constexpr int oK = DO_V ? 9 : 0, oM = oK + (DO_K ? 9 : 0), kEntries = oM + (DO_K && kMirror ? 9 : 0);
  float2 acc[kEntries];
#pragma unroll
  for (int e = 0; e < kEntries; e++) acc[e] = make_float2(0.f, 0.f);
  auto region = [&](float x1, float x2, float y1, float y2, float w) {
    float d[3];
#pragma unroll
    for (int e = 0; e < 3; e++)
      d[e] = NCOMMON == 2 ? (y1 - x1) * E1[e] + y2 * F2[e] - x2 * E2[e]  // F1 = E1, the shared edge
                          : y1 * F1[e] + y2 * F2[e] - x1 * E1[e] - x2 * E2[e];
    const float r2 = fmaxf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2], kEps * kEps);
    const float ri = rsqrtf(r2), kr = k * (r2 * ri);
    float s, c;
    __sincosf(kr, &s, &c);
    const float riw = ri * w;
    const float lx[3] = {1.f - x1, x1 - x2, x2}, ly[3] = {1.f - y1, y1 - y2, y2};
    if (DO_V) {
      const float2 gv = make_float2(c * riw, s * riw);
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const float2 gy = f2_mul(f2(ly[b]), gv);
#pragma unroll
        for (int a = 0; a < 3; a++) acc[3 * a + b] = f2_fma(f2(lx[a]), gy, acc[3 * a + b]);
      }
    }
    if (DO_K) {
      const float dj = d[0] * nj[0] + d[1] * nj[1] + d[2] * nj[2];     // (y - x) . n_j
      const float di = -(d[0] * ni[0] + d[1] * ni[1] + d[2] * ni[2]);  // (x - y) . n_i
      const float f = ri * ri * riw;
      const float2 h = make_float2(fmaf(kr, s, c) * f, fmaf(-kr, c, s) * f);
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const float2 hy = f2_mul(f2(ly[b]), h);
#pragma unroll
        for (int a = 0; a < 3; a++) {
          acc[oK + 3 * a + b] = f2_fma(f2(lx[a] * dj), hy, acc[oK + 3 * a + b]);
          if (kMirror) acc[oM + 3 * a + b] = f2_fma(f2(lx[a] * di), hy, acc[oM + 3 * a + b]);
        }
      }
    }
  };
#pragma unroll 1
  for (int pt = lane; pt < 256; pt += 32) {
    float xi, e1, e2, e3, w;
    touch_point<float>(pt, xi, e1, e2, e3, w);
    ss_regions<NCOMMON, float>(xi, e1, e2, e3, w * jw, region);
  }
  float t[2 * kEntries];
#pragma unroll
  for (int e = 0; e < kEntries; e++) {
    t[2 * e] = acc[e].x;
    t[2 * e + 1] = acc[e].y;
  }
  warp_totals<2 * kEntries>(t, total);
  if (lane < kEntries) {
    const int e = lane % 9, A = vi[e / 3], B = vj[e % 3];
    const bool isV = DO_V && lane < 9;
    const float sc = isV ? v_scale : k_scale;
    const float2 x = make_float2(total[2 * lane] * sc, total[2 * lane + 1] * sc);
    const size_t ab = (size_t)A * g.nv + B, ba = (size_t)B * g.nv + A;
    if (isV) {
      atomicAdd(&V[ab], x);
      if (kMirror) atomicAdd(&V[ba], x);
    } else {
      atomicAdd(&K[lane >= oM ? ba : ab], x);
    }
  }
}

// Warp `w` of one problem's touching pairs: the triangles, the edge pairs, the
// unordered vertex pairs.
__host__ __device__ inline long long touch_warps(const GeomView& g) { return (long long)g.nt + g.n_edge + g.n_vert / 2; }
template <bool DO_V, bool DO_K>
__device__ __forceinline__ void touch_warp(const GeomView& g, long long w, float k, float2* __restrict__ V,
                                           float2* __restrict__ K, float v_scale, float k_scale, float mass_coeff,
                                           TouchShared& sm) {
  const int warp = threadIdx.x >> 5;
  const long long n0 = g.nt;
  if (w < n0) {
    touch_coincident<DO_V, DO_K>(g, (int)w, k, V, K, v_scale, mass_coeff, sm.c[warp]);
  } else if (w < n0 + g.n_edge) {
    const int2 p = g.edge_pairs[w - n0];
    touch_pair<2, DO_V, DO_K>(g, p.x, p.y, k, V, K, v_scale, k_scale, sm.f[warp]);
  } else {
    const int2 p = g.vert_pairs[w - n0 - g.n_edge];
    touch_pair<1, DO_V, DO_K>(g, p.x, p.y, k, V, K, v_scale, k_scale, sm.f[warp]);
  }
}

template <bool DO_V, bool DO_K>
__global__ void __launch_bounds__(kTouchThreads)
    touch_vk_kernel(const __grid_constant__ GeomView g, float k, float2* __restrict__ V,
                    float2* __restrict__ K, float v_scale, float k_scale, float mass_coeff) {
  __shared__ TouchShared sm;
  const long long w = (long long)blockIdx.x * kTouchWarps + (threadIdx.x >> 5);
  if (w < touch_warps(g)) touch_warp<DO_V, DO_K>(g, w, k, V, K, v_scale, k_scale, mass_coeff, sm);
  wait_previous();
}

// ---------------------------------------------------------------------------
// Batched assembly: many problems (meshes of uneven size, wavenumbers) in one
// persistent launch.  Regular work items of all problems (runs of strip
// steps, each unordered pair once) form one queue that warps drain with an
// atomic counter (dynamic load balance); touching
// pairs of all problems are concatenated per type.
// ---------------------------------------------------------------------------
struct BatchProblem {
  GeomView g;
  float k;
  StripItems items;
  float2* V;
  float2* K;
  long long item_begin;   // prefix sum of regular items
  long long touch_begin;  // prefix sum of touching-pair warps
};

struct BatchHeader {
  unsigned long long next_item;  // queue head (zeroed before each launch)
  int nproblems;
  int pad;
  long long total_items, total_touch;
};

__device__ __forceinline__ int find_problem(const BatchProblem* probs, int np, long long x, bool touch) {
  int lo = 0, hi = np - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const long long b = touch ? probs[mid].touch_begin : probs[mid].item_begin;
    if (b <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Each unordered regular pair of every problem once; the warps draw the items.
__global__ void __launch_bounds__(kStripThreads, 2)
    regular_strip_vk_batch_kernel(BatchHeader* __restrict__ hdr, const BatchProblem* __restrict__ probs, float v_scale,
                                  float k_scale) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  VkWarp& sw = reinterpret_cast<VkWarp*>(smem_raw)[threadIdx.x >> 5];
  launch_next();
  strip_init(sw);
  const int np = hdr->nproblems;
  const long long total = hdr->total_items;
  VkStrip pol;
  pol.v_scale = v_scale;
  pol.k_scale = k_scale;
  pol.clear();
  StripTest test;
  unsigned uses = 0;
  for (;;) {
    long long item = 0;
    if ((threadIdx.x & 31) == 0) item = (long long)atomicAdd(&hdr->next_item, 1ull);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= total) break;
    const BatchProblem& P = probs[find_problem(probs, np, item, false)];
    pol.k = P.k;
    pol.V = P.V;
    pol.K = P.K;
    test.grp = -1;  // another problem's block may have the same number
    strip_item(sw, test, P.g, pol, P.items, item - P.item_begin, uses, &g_asm_err);
  }
}

__global__ void __launch_bounds__(kTouchThreads)
    touch_vk_batch_kernel(const BatchHeader* __restrict__ hdr, const BatchProblem* __restrict__ probs, float v_scale,
                          float k_scale, float mass_coeff) {
  __shared__ TouchShared sm;
  const long long w = (long long)blockIdx.x * kTouchWarps + (threadIdx.x >> 5);
  if (w < hdr->total_touch) {
    const BatchProblem& P = probs[find_problem(probs, hdr->nproblems, w, true)];
    touch_warp<true, true>(P.g, w - P.touch_begin, P.k, P.V, P.K, v_scale, k_scale, mass_coeff, sm);
  }
  wait_previous();
}

// Dense P1 mass matrix, one thread per triangle (bind.cu:10-21).
__global__ void mass_kernel(GeomView g, float2* __restrict__ M, float coeff) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nt) return;
  const TriRec& r = g.rec_orig[i];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) {
      double m = 0.0;
#pragma unroll
      for (int q = 0; q < 6; q++) m += tri6_w(q) * tri6_phi(q, a) * tri6_phi(q, b);
      atomicAdd(&M[(size_t)r.v[a] * g.nv + r.v[b]], make_float2((float)(coeff * r.area * m), 0.f));
    }
}

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

template <bool DO_V, bool DO_K>
int launch_regular(const GeomView& g, float k, float2* V, float2* K, float v_scale, float k_scale, cudaStream_t s) {
  const int smem = (int)sizeof(RegSmem<DO_V, DO_K>);
  static DeviceOnce once;
  if (const int rc = once.shared_memory(regular_vk_kernel<DO_V, DO_K>, smem)) return rc;
  const int n_groups = (g.nt + kTestTris - 1) / kTestTris;
  int occ = 0;
  BEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, regular_vk_kernel<DO_V, DO_K>, kRegThreads, smem));
  if (g_tune_ctas_per_sm > 0 && g_tune_ctas_per_sm < occ) occ = g_tune_ctas_per_sm;
  const int grid = sm_count() * (occ > 0 ? occ : 1);
  // chunk of trial tiles per work item: enough items to balance the grid
  int chunk = (int)((long long)n_groups * g.ntiles / (8LL * grid));
  chunk = chunk < 1 ? 1 : (chunk > 64 ? 64 : chunk);
  if (g_tune_chunk > 0) chunk = 2 * std::min(g_tune_chunk, g.ntiles);  // the knob counts blocks of 32
  const int n_chunks = (g.ntiles + chunk - 1) / chunk;
  const int n_items = n_groups * n_chunks;
  (regular_vk_kernel<DO_V, DO_K><<<grid < n_items ? grid : n_items, kRegThreads, smem, s>>>(
      g, k, V, K, v_scale, k_scale, chunk, n_chunks, n_items), count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

template <bool DO_V, bool DO_K>
int launch_touch(const GeomView& g, float k, float2* V, float2* K, float v_scale, float k_scale, float mass_coeff,
                 cudaStream_t s) {
  EarlyLaunch l((unsigned)((touch_warps(g) + kTouchWarps - 1) / kTouchWarps), kTouchThreads, 0, s);
  if (!(DO_V && DO_K)) l.cfg.numAttrs = 0;  // regular_vk_kernel does not start it early
  BEM_CUDA_TRY(cudaLaunchKernelEx(&l.cfg, touch_vk_kernel<DO_V, DO_K>, g, k, V, K, v_scale, k_scale, mass_coeff));
  count_launch();
  return BEM_OK;
}

}  // namespace

namespace {
// Persistent grid of a strip kernel.
template <typename KernelT>
int strip_grid(KernelT kernel, DeviceOnce& once, int most_per_sm, long long* grid) {
  const int smem = (int)(kStripWarps * sizeof(VkWarp));
  if (const int rc = once.shared_memory(kernel, smem)) return rc;
  int occ = 0;
  BEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kStripThreads, smem));
  if (most_per_sm > 0 && most_per_sm < occ) occ = most_per_sm;
  *grid = (long long)sm_count() * (occ > 0 ? occ : 1);
  return BEM_OK;
}

int launch_strip_vk(const GeomView& g, float k, float2* V, float2* K, float v_scale, float k_scale, cudaStream_t s) {
  static DeviceOnce once;
  long long grid = 0;
  int rc = strip_grid(regular_strip_vk_kernel, once, 0, &grid);
  if (rc) return rc;
  const StripItems P = strip_items(g.nv, g.nblocks, grid * kStripWarps, kStripRounds, 2, g_tune_chunk, 0, 0);
  const long long blocks = (P.items + kStripWarps - 1) / kStripWarps;
  grid *= kStripRounds;
  (regular_strip_vk_kernel<<<(unsigned)(grid < blocks ? grid : blocks), kStripThreads, kStripWarps * sizeof(VkWarp), s>>>(
       g, k, V, K, v_scale, k_scale, P),
   count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}
}  // namespace

// V and/or (mass_coeff M + k_coeff K), both overwritten.
int assemble_vk(const GeomView& g, float k, float2* V, float2* Kout, float mass_coeff, float k_coeff, cudaStream_t s) {
  const size_t bytes = sizeof(float2) * (size_t)g.nv * g.nv;
  if (V) BEM_CUDA_TRY(cudaMemsetAsync(V, 0, bytes, s));
  if (Kout) BEM_CUDA_TRY(cudaMemsetAsync(Kout, 0, bytes, s));
  const float v_scale = kInv4Pi;
  const float k_scale = -kInv4Pi * k_coeff;  // K = -(...)/(4 pi)
  int rc;
  if (V && Kout) {
    if ((rc = launch_strip_vk(g, k, V, Kout, v_scale, k_scale, s))) return rc;
    return launch_touch<true, true>(g, k, V, Kout, v_scale, k_scale, mass_coeff, s);
  } else if (V) {
    if ((rc = launch_regular<true, false>(g, k, V, nullptr, v_scale, 0.f, s))) return rc;
    return launch_touch<true, false>(g, k, V, nullptr, v_scale, 0.f, 0.f, s);
  } else if (Kout) {
    if ((rc = launch_regular<false, true>(g, k, nullptr, Kout, 0.f, k_scale, s))) return rc;
    return launch_touch<false, true>(g, k, nullptr, Kout, 0.f, k_scale, mass_coeff, s);
  }
  return BEM_OK;
}

int assemble_mass(const GeomView& g, float2* M, float coeff, bool zero, cudaStream_t s) {
  if (zero) BEM_CUDA_TRY(cudaMemsetAsync(M, 0, sizeof(float2) * (size_t)g.nv * g.nv, s));
  (mass_kernel<<<(g.nt + 127) / 128, 128, 0, s>>>(g, M, coeff), count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

}  // namespace bemb

// ---------------------------------------------------------------------------
// Batched assembly host side and tuning knobs.
// ---------------------------------------------------------------------------
#include <vector>

namespace bemb {

namespace {
int g_tune_chunk = 0;        // trial blocks (32 triangles) per regular work item (0: automatic)
int g_tune_ctas_per_sm = 0;  // persistent CTAs per SM (0: occupancy limit; not for V and K of one problem)

struct PinnedStage {
  void* buf = nullptr;
  size_t cap = 0;
  cudaEvent_t ev = nullptr;
  ~PinnedStage() {
    if (buf) cudaFreeHost(buf);
    if (ev) cudaEventDestroy(ev);
  }
};
thread_local PinnedStage t_stage;

inline size_t al256b(size_t x) { return (x + 255) / 256 * 256; }
}  // namespace

// Reads and clears the flag that an assembly kernel's bounded wait expired
// (synchronises the stream).
int assembly_status(int* err_host, cudaStream_t s) {
  int zero = 0;
  BEM_CUDA_TRY(cudaMemcpyFromSymbolAsync(err_host, g_asm_err, sizeof(int), 0, cudaMemcpyDeviceToHost, s));
  BEM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_asm_err, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, s));
  BEM_CUDA_TRY(cudaStreamSynchronize(s));
  return BEM_OK;
}

int set_tuning(int key, int value) {
  if (value < 0) return BEM_ERR_INVALID_ARGUMENT;
  switch (key) {
    case BEM_TUNE_ASSEMBLY_CHUNK: g_tune_chunk = value; return BEM_OK;
    case BEM_TUNE_ASSEMBLY_CTAS_PER_SM: g_tune_ctas_per_sm = value; return BEM_OK;
    case BEM_TUNE_TC_PROMOTE: g_tc_promote = value; return BEM_OK;
    case BEM_TUNE_GMRES_REORTH:
      if (value > 2) return BEM_ERR_INVALID_ARGUMENT;
      g_gmres_reorth = value;
      return BEM_OK;
    case BEM_TUNE_ARNOLDI_CLUSTER:
      if (value > 16) return BEM_ERR_INVALID_ARGUMENT;
      g_arn_max_cluster = value;
      return BEM_OK;
    case BEM_TUNE_ARNOLDI_MODE:
      if (value > 3) return BEM_ERR_INVALID_ARGUMENT;
      g_arn_mode = value;
      return BEM_OK;
    case BEM_TUNE_TC_WAIT_US:
      g_tc_wait_us = value;
      return BEM_OK;
    case BEM_TUNE_TC_TEST_SKIP_FILL:
      g_tc_skip_fill.store(value);
      return BEM_OK;
    case BEM_TUNE_GMRES_BLOCK:
      if (value > 1) return BEM_ERR_INVALID_ARGUMENT;
      g_gmres_block = value;
      return BEM_OK;
  }
  return BEM_ERR_INVALID_ARGUMENT;
}

int get_tuning(int key) {
  switch (key) {
    case BEM_TUNE_ASSEMBLY_CHUNK: return g_tune_chunk;
    case BEM_TUNE_ASSEMBLY_CTAS_PER_SM: return g_tune_ctas_per_sm;
    case BEM_TUNE_TC_PROMOTE: return g_tc_promote;
    case BEM_TUNE_GMRES_REORTH: return g_gmres_reorth;
    case BEM_TUNE_ARNOLDI_CLUSTER: return g_arn_max_cluster;
    case BEM_TUNE_ARNOLDI_MODE: return g_arn_mode;
    case BEM_TUNE_TC_WAIT_US: return g_tc_wait_us;
    case BEM_TUNE_TC_TEST_SKIP_FILL: return g_tc_skip_fill.load();
    case BEM_TUNE_GMRES_BLOCK: return g_gmres_block;
  }
  return -1;
}

size_t batch_workspace_bytes(int np) {
  return al256b(sizeof(BatchHeader)) + al256b(sizeof(BatchProblem) * (size_t)(np > 0 ? np : 1));
}

int assemble_vk_batch(const GeomView* views, const float* ks, float2* const* Vs, float2* const* Ks, int np,
                      float mass_coeff, float k_coeff, void* ws, size_t ws_bytes, cudaStream_t s) {
  if (np <= 0) return BEM_ERR_INVALID_ARGUMENT;
  if (!ws || ws_bytes < batch_workspace_bytes(np)) return BEM_ERR_WORKSPACE;
  static DeviceOnce once;
  long long grid = 0;
  const int rc = strip_grid(regular_strip_vk_batch_kernel, once, g_tune_ctas_per_sm, &grid);
  if (rc) return rc;
  // host descriptors
  const size_t hbytes = al256b(sizeof(BatchHeader)), pbytes = sizeof(BatchProblem) * (size_t)np;
  if (!t_stage.ev) BEM_CUDA_TRY(cudaEventCreateWithFlags(&t_stage.ev, cudaEventDisableTiming));
  BEM_CUDA_TRY(cudaEventSynchronize(t_stage.ev));  // previous upload from the staging buffer is done
  if (t_stage.cap < hbytes + pbytes) {
    if (t_stage.buf) cudaFreeHost(t_stage.buf);
    t_stage.cap = 2 * (hbytes + pbytes);
    BEM_CUDA_TRY(cudaHostAlloc(&t_stage.buf, t_stage.cap, cudaHostAllocDefault));
  }
  BatchHeader* hh = (BatchHeader*)t_stage.buf;
  BatchProblem* hp = (BatchProblem*)((char*)t_stage.buf + hbytes);
  std::memset(hh, 0, sizeof(BatchHeader));
  hh->nproblems = np;
  long long items = 0, touch = 0, steps = 0;
  for (int p = 0; p < np; p++) steps += strip_steps(views[p].nblocks);
  // about 8 items per warp over the whole batch, at most 16 trial blocks each
  const long long share = std::min<long long>(512, std::max<long long>(4, steps / (8 * grid * kStripWarps)));
  const size_t elem = sizeof(float2);
  for (int p = 0; p < np; p++) {
    const GeomView& g = views[p];
    if (!Vs[p] || !Ks[p]) return BEM_ERR_INVALID_ARGUMENT;
    if (!std::isfinite(ks[p])) return BEM_ERR_NONFINITE;
    BEM_CUDA_TRY(cudaMemsetAsync(Vs[p], 0, elem * (size_t)g.nv * g.nv, s));
    BEM_CUDA_TRY(cudaMemsetAsync(Ks[p], 0, elem * (size_t)g.nv * g.nv, s));
    BatchProblem& P = hp[p];
    P.g = g;
    P.k = ks[p];
    P.items = strip_items(g.nv, g.nblocks, std::max(1LL, strip_steps(g.nblocks) / share), 1, 4, g_tune_chunk, 0, 0);
    P.V = Vs[p];
    P.K = Ks[p];
    P.item_begin = items;
    items += P.items.items;
    P.touch_begin = touch;
    touch += touch_warps(g);
  }
  hh->total_items = items;
  hh->total_touch = touch;
  BatchHeader* dh = (BatchHeader*)ws;
  BatchProblem* dp = (BatchProblem*)((char*)ws + hbytes);
  BEM_CUDA_TRY(cudaMemcpyAsync(ws, t_stage.buf, hbytes + pbytes, cudaMemcpyHostToDevice, s));
  BEM_CUDA_TRY(cudaEventRecord(t_stage.ev, s));
  const float v_scale = kInv4Pi, k_scale = -kInv4Pi * k_coeff;
  const long long blocks = (items + kStripWarps - 1) / kStripWarps;
  (regular_strip_vk_batch_kernel<<<(unsigned)(grid < blocks ? grid : blocks), kStripThreads,
                                   kStripWarps * sizeof(VkWarp), s>>>(dh, dp, v_scale, k_scale),
   count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  EarlyLaunch l((unsigned)((touch + kTouchWarps - 1) / kTouchWarps), kTouchThreads, 0, s);
  BEM_CUDA_TRY(cudaLaunchKernelEx(&l.cfg, touch_vk_batch_kernel, (const BatchHeader*)dh, (const BatchProblem*)dp,
                                  v_scale, k_scale, mass_coeff));
  count_launch();
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

}  // namespace bemb
