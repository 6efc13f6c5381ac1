// Fused Burton-Miller assembly: both matrices of the reference's
// neumann2dirichlet (src/bem/solver.py:118-126) in one pass,
//   lhs = BM_LHS + 1/2 M,     rhs = BM_RHS - (i / (2k)) M,
// at the <2,3> rules of its "_approx" bindings (bind.cu:204-215): the 3-point
// degree-2 triangle rule for regular pairs, 2-point Gauss-Legendre
// Sauter-Schwab quadrature for touching pairs.  At the exact <4,6> rules the
// same pair is the reference's HBIE system (solver.py:106-116):
//   1/2 M - K + (i/k) W = BM_LHS + 1/2 M   (W = curl term - k^2 n.n G),
//   -V - (i/k)(K' + 1/2 M) = BM_RHS - (i/(2k)) M,
// so the kernels are templated on the rule (TN points per triangle, LN
// Gauss-Legendre points per Sauter-Schwab axis).
//
// Kernels (potential.h:42-65, integrand.h:94-101,216-221,314-322), x on the
// test triangle i, y on the trial triangle j, G = e^{ikr}/r and
// H = (1 - ikr) e^{ikr} / r^3 (the 1/(4 pi) applied last):
//   BM_LHS(i,j) = -ik (n_i.n_j) G + H (y - x).n_j + (i/k) G (curl_i . curl_j)
//   BM_RHS(i,j) = -G + (i/k) H (x - y).n_i
// The curl term uses the P1 surface curls, constant per triangle, so the
// Galerkin block needs only the weight sum of G over the pair.
//
// Regular pairs: G, H (y-x).n_j and H (x-y).n_i are symmetric / swapped under
// i <-> j, so one evaluation of r and sincos per quadrature-point pair of an
// UNORDERED pair gives all four blocks lhs_ij, lhs_ji, rhs_ij, rhs_ji:
//   S = sum C C G,  T = sum C C H (y-x).n_j,  U = sum C C H (x-y).n_i
//   lhs_ij = -ik nn S + T + (i/k) s cc      lhs_ji^T = -ik nn S + U + (i/k) s cc
//   rhs_ij = -S + (i/k) U                   rhs_ji^T = -S + (i/k) T
// with s = sum_ab S_ab (the P1 functions sum to one) and cc_ab the curl
// products, summed in registers along a warp's strip walk (strip.cuh).
// Touching pairs: one warp per pair evaluates both kernels at each
// Sauter-Schwab point (shared r and sincos); the coincident pass (FP64) adds
// the mass terms.  A batch (meshes, wavenumbers) uses the same kernels with a
// work queue over all problems.

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>

#include "async_copy.cuh"
#include "bem_common.cuh"
#include "sauter_schwab.cuh"
#include "strip.cuh"

namespace bemb {

namespace {

// C(q, b) = w_q phi_b(q): centroid rule 1/3; 3-point rule 1/3 * (q == b ?
// 2/3 : 1/6); 6-point rule as the V/K assembly.
template <int TN>
__host__ __device__ constexpr float bm_c(int q, int b) {
  return TN == 1 ? 1.0f / 3.0f
                 : (TN == 3 ? (q == b ? 2.0f / 9.0f : 1.0f / 18.0f) : (float)(tri6_w(q) * tri6_phi(q, b)));
}

// A bounded wait of the Burton-Miller kernels expired (read by bm_status).
__device__ int g_bm_err;

// G and H = (1 - ikr) G / r^2 (times 4 pi) at two trial points, FP32 pairs.
__device__ __forceinline__ void bm_point2(float2 dx, float2 dy, float2 dz, float k, float2& gr, float2& gi,
                                          float2& hr, float2& hi) {
  float2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
  r2.x = fmaxf(r2.x, kEps * kEps);  // r >= 1e-3, to a rounding
  r2.y = fmaxf(r2.y, kEps * kEps);
  const float2 ri = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
  const float2 kr = f2_mul(f2(k), f2_mul(r2, ri)), ri2 = f2_mul(ri, ri);
  float2 s, c;
  __sincosf(kr.x, &s.x, &c.x);
  __sincosf(kr.y, &s.y, &c.y);
  gr = f2_mul(c, ri);
  gi = f2_mul(s, ri);
  hr = f2_mul(f2_fma(f2(k), s, gr), ri2);
  hi = f2_mul(f2_fma(f2(-k), c, gi), ri2);
}

// The same at one point: (G, H).
__device__ __forceinline__ void bm_point(float dx, float dy, float dz, float k, float2& g, float2& h) {
  const float r2 = fmaxf(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), kEps * kEps);
  const float ri = rsqrtf(r2), ri2 = ri * ri;
  float s, c;
  __sincosf(k * (r2 * ri), &s, &c);
  g = make_float2(c * ri, s * ri);
  h = make_float2(fmaf(k, s, g.x) * ri2, fmaf(-k, c, g.y) * ri2);
}

template <int TN>
using BmWarp = StripWarp<3 * TN + 9, true>;
constexpr int kBmPanel = 2, kBmPanelItems = 8;  // strip_items

// Strip walk of the Burton-Miller pair (strip.cuh): the open columns hold
// lhs_ij, lhs_ji^T and rhs_ij; rhs_ji^T - rhs_ij = (i/k)(T - U) = (i/k)(lhs_ij
// - lhs_ji^T) entry by entry, so it follows from the reduced sums.  Rows of xs:
// the test points, then the test curls.
//
// Measured on B200 at the 3-point rule, the whole assembly: 8286 triangles 1.49
// ms, 20 480 triangles 8.3 ms, against 2.20 and 12.7 ms for 16 x 16-triangle
// tiles reduced in shared memory (at 9 point pairs per triangle pair the
// reduction took over half of the time).  Issue slots and FP32 pipe 58 and 50 %
// busy; the atomics' DRAM traffic (23 GB at 20 480 triangles with contiguous
// items) is why the items go in panels (strip_items).
template <int TN>
struct BmStrip {
  float k, kinv;
  float2* L;
  float2* R;
  // the curl terms, which cancel over a vertex star, apart from the others
  float2 aL[9], aT[9], aR[9], aC[9];

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int e = 0; e < 9; e++) aL[e] = aT[e] = aR[e] = aC[e] = make_float2(0.f, 0.f);
  }

  __device__ __forceinline__ void load(BmWarp<TN>& sw, const StripTest& t, const GeomView& g, int lane) {
    const int at = min(t.grp * kBlock + lane, g.nt - 1);
    const TriRec& r = g.rec[at];
    const BmRec& b = g.bm[at];
#pragma unroll
    for (int e = 0; e < 3 * TN; e++) sw.xs[e][lane] = TN == 3 ? b.qp[e] : (TN == 6 ? r.qp[e] : r.c[e]);
#pragma unroll
    for (int e = 0; e < 9; e++) sw.xs[3 * TN + e][lane] = b.curl[e];
  }

  __device__ __forceinline__ void pair(const BmWarp<TN>& sw, const StripTest& t, const TriRec& rj, const BmRec& bj,
                                       float w, int lane) {
    const float* yq = TN == 3 ? bj.qp : (TN == 6 ? rj.qp : rj.c);
    const float njx = rj.n[0], njy = rj.n[1], njz = rj.n[2], cjx = rj.c[0], cjy = rj.c[1], cjz = rj.c[2];
    const float sc = w * kInv4Pi;
    const float knn = k * (t.nx * njx + t.ny * njy + t.nz * njz);
    float dq[TN];  // n_i . (c_i - y_q)
#pragma unroll
    for (int q = 0; q < TN; q++)
      dq[q] = t.nx * (t.cx - yq[3 * q]) + t.ny * (t.cy - yq[3 * q + 1]) + t.nz * (t.cz - yq[3 * q + 2]);
    float2 total = make_float2(0.f, 0.f);  // weight sum of G over the pair
#pragma unroll
    for (int p = 0; p < TN; p++) {
      const float px = sw.xs[3 * p][lane], py = sw.xs[3 * p + 1][lane], pz = sw.xs[3 * p + 2][lane];
      const float dn = njx * (cjx - px) + njy * (cjy - py) + njz * (cjz - pz);  // (y - x).n_j on plane j
      // trial sums of G, H and dq H, by vertex
      float2 tS[3], tH[3], tU[3];
      if constexpr (TN == 1) {
        float2 g, h;
        bm_point(yq[0] - px, yq[1] - py, yq[2] - pz, k, g, h);
#pragma unroll
        for (int b = 0; b < 3; b++) {
          tS[b] = f2_mul(f2(1.f / 3.f), g);
          tH[b] = f2_mul(f2(1.f / 3.f), h);
          tU[b] = f2_mul(f2(dq[0] / 3.f), h);
        }
      } else if constexpr (TN == 3) {
        float2 gr, gi, hr, hi;
        bm_point2(f2_sub(make_float2(yq[0], yq[3]), f2(px)), f2_sub(make_float2(yq[1], yq[4]), f2(py)),
                f2_sub(make_float2(yq[2], yq[5]), f2(pz)), k, gr, gi, hr, hi);
        tS[0] = make_float2(gr.x, gi.x);
        tS[1] = make_float2(gr.y, gi.y);
        tH[0] = make_float2(hr.x, hi.x);
        tH[1] = make_float2(hr.y, hi.y);
        bm_point(yq[6] - px, yq[7] - py, yq[8] - pz, k, tS[2], tH[2]);
        float2 sS = f2_add(f2_add(tS[0], tS[1]), tS[2]), sH = f2_add(f2_add(tH[0], tH[1]), tH[2]), sU;
#pragma unroll
        for (int b = 0; b < 3; b++) tU[b] = f2_mul(f2(dq[b]), tH[b]);
        sU = f2_add(f2_add(tU[0], tU[1]), tU[2]);
        // w phi_b = 1/18 + 1/6 [b == q]
#pragma unroll
        for (int b = 0; b < 3; b++) {
          tS[b] = f2_fma(f2(1.f / 6.f), tS[b], f2_mul(f2(1.f / 18.f), sS));
          tH[b] = f2_fma(f2(1.f / 6.f), tH[b], f2_mul(f2(1.f / 18.f), sH));
          tU[b] = f2_fma(f2(1.f / 6.f), tU[b], f2_mul(f2(1.f / 18.f), sU));
        }
      } else {
        constexpr float o0 = (float)tri6_w_own(0), o3 = (float)tri6_w_own(3), c0 = (float)tri6_w_common(0),
                        c3 = (float)tri6_w_common(3);
        float2 cS = make_float2(0.f, 0.f), cH = cS, cU = cS;
#pragma unroll
        for (int b = 0; b < 3; b++) {
          float2 gr, gi, hr, hi;
          const int i0 = 3 * b, i3 = 9 + 3 * b;
          bm_point2(f2_sub(make_float2(yq[i0], yq[i3]), f2(px)), f2_sub(make_float2(yq[i0 + 1], yq[i3 + 1]), f2(py)),
                  f2_sub(make_float2(yq[i0 + 2], yq[i3 + 2]), f2(pz)), k, gr, gi, hr, hi);
          const float2 d = make_float2(dq[b], dq[b + 3]);
          const float2 ur = f2_mul(d, hr), ui = f2_mul(d, hi);
          tS[b] = make_float2(fmaf(o3, gr.y, o0 * gr.x), fmaf(o3, gi.y, o0 * gi.x));
          tH[b] = make_float2(fmaf(o3, hr.y, o0 * hr.x), fmaf(o3, hi.y, o0 * hi.x));
          tU[b] = make_float2(fmaf(o3, ur.y, o0 * ur.x), fmaf(o3, ui.y, o0 * ui.x));
          cS.x += fmaf(c3, gr.y, c0 * gr.x);
          cS.y += fmaf(c3, gi.y, c0 * gi.x);
          cH.x += fmaf(c3, hr.y, c0 * hr.x);
          cH.y += fmaf(c3, hi.y, c0 * hi.x);
          cU.x += fmaf(c3, ur.y, c0 * ur.x);
          cU.y += fmaf(c3, ui.y, c0 * ui.x);
        }
#pragma unroll
        for (int b = 0; b < 3; b++) {
          tS[b] = f2_add(tS[b], cS);
          tH[b] = f2_add(tH[b], cH);
          tU[b] = f2_add(tU[b], cU);
        }
      }
      const float wp = (float)(TN == 1 ? 1.0 : (TN == 3 ? 1.0 / 3.0 : tri6_w(p)));
      total = f2_fma(f2(wp), f2_add(f2_add(tS[0], tS[1]), tS[2]), total);
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const float2 z = make_float2(knn * tS[b].y, -knn * tS[b].x);  // -ik (n_i.n_j) S
        tH[b] = f2_fma(f2(dn), tH[b], z);
        tS[b] = make_float2(fmaf(-kinv, tU[b].y, -tS[b].x), fmaf(kinv, tU[b].x, -tS[b].y));  // -S + (i/k) U
        tU[b] = f2_add(tU[b], z);
      }
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const float2 wa = f2(sc * bm_c<TN>(p, a));
#pragma unroll
        for (int b = 0; b < 3; b++) {
          aL[3 * a + b] = f2_fma(wa, tH[b], aL[3 * a + b]);
          aT[3 * a + b] = f2_fma(wa, tU[b], aT[3 * a + b]);
          aR[3 * a + b] = f2_fma(wa, tS[b], aR[3 * a + b]);
        }
      }
    }
    const float2 v = make_float2(-total.y * (sc * kinv), total.x * (sc * kinv));  // (i/k) times the sum
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float cx = sw.xs[3 * TN + 3 * a][lane], cy = sw.xs[3 * TN + 3 * a + 1][lane],
                  cz = sw.xs[3 * TN + 3 * a + 2][lane];
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const float2 cc = f2(cx * bj.curl[3 * b] + cy * bj.curl[3 * b + 1] + cz * bj.curl[3 * b + 2]);
        aC[3 * a + b] = f2_fma(cc, v, aC[3 * a + b]);
      }
    }
  }

  template <int B>
  __device__ __forceinline__ void take(BmWarp<TN>& sw, int i, int lane) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float2 l = f2_add(aL[3 * a + B], aC[3 * a + B]), lt = f2_add(aT[3 * a + B], aC[3 * a + B]);
      sw.col4[i][32 * a + lane] = make_float4(l.x, l.y, lt.x, lt.y);
      sw.col2[i][32 * a + lane] = aR[3 * a + B];
      aL[3 * a + B] = aT[3 * a + B] = aR[3 * a + B] = aC[3 * a + B] = make_float2(0.f, 0.f);
    }
  }

  __device__ __forceinline__ void store(const GeomView& g, int A, int B, const float4& s, const float2& r) const {
    if (s.x == 0.f && s.y == 0.f && s.z == 0.f && s.w == 0.f && r.x == 0.f && r.y == 0.f) return;
    const size_t ab = (size_t)A * g.nv + B, ba = (size_t)B * g.nv + A;
    atomicAdd(&L[ab], make_float2(s.x, s.y));
    atomicAdd(&L[ba], make_float2(s.z, s.w));
    atomicAdd(&R[ab], r);
    atomicAdd(&R[ba], make_float2(fmaf(s.w - s.y, kinv, r.x), fmaf(s.x - s.z, kinv, r.y)));
  }
};

// ---- problem descriptors (one problem, or a batch) ----
struct BmProblem {
  GeomView g;
  float k;
  StripItems items;
  long long item_begin;     // prefix sum of work items
  long long pair_begin[3];  // prefix sums of coincident / edge / vertex pairs
  float2* L;
  float2* R;
};

struct BmHeader {
  unsigned long long next_item;  // queue head (zeroed before each launch)
  int nproblems;
  int pad;
  long long total_items;
  long long total_pairs[3];
};

__device__ __forceinline__ int bm_find(const BmProblem* probs, int np, long long x, int which) {
  int lo = 0, hi = np - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const long long b = which < 0 ? probs[mid].item_begin : probs[mid].pair_begin[which];
    if (b <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Regular pairs of one problem: a warp takes one work item (or, past the grid's
// size, every grid-width-th).
template <int TN>
__global__ void __launch_bounds__(kStripThreads, 2)
    regular_bm_kernel(const __grid_constant__ BmProblem P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BmWarp<TN>& sw = reinterpret_cast<BmWarp<TN>*>(smem_raw)[threadIdx.x >> 5];
  launch_next();
  strip_init(sw);
  BmStrip<TN> pol;
  pol.k = P.k;
  pol.kinv = 1.0f / P.k;
  pol.L = P.L;
  pol.R = P.R;
  pol.clear();
  StripTest test;
  unsigned uses = 0;
  const long long warps = (long long)gridDim.x * kStripWarps;
  for (long long item = (long long)blockIdx.x * kStripWarps + (threadIdx.x >> 5); item < P.items.items; item += warps)
    strip_item(sw, test, P.g, pol, P.items, item, uses, &g_bm_err);
}

template <int TN>
__global__ void __launch_bounds__(kStripThreads, 2)
    regular_bm_batch_kernel(BmHeader* __restrict__ hdr, const BmProblem* __restrict__ probs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BmWarp<TN>& sw = reinterpret_cast<BmWarp<TN>*>(smem_raw)[threadIdx.x >> 5];
  launch_next();
  strip_init(sw);
  const int np = hdr->nproblems;
  const long long total = hdr->total_items;
  BmStrip<TN> pol;
  pol.clear();
  StripTest test;
  unsigned uses = 0;
  for (;;) {
    long long item = 0;
    if ((threadIdx.x & 31) == 0) item = (long long)atomicAdd(&hdr->next_item, 1ull);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= total) break;
    const BmProblem& P = probs[bm_find(probs, np, item, -1)];
    pol.k = P.k;
    pol.kinv = 1.0f / P.k;
    pol.L = P.L;
    pol.R = P.R;
    test.grp = -1;  // another problem's block may have the same number
    strip_item(sw, test, P.g, pol, P.items, item - P.item_begin, uses, &g_bm_err);
  }
}

// Both Burton-Miller kernels at d = y - x, without the 1/(4 pi):
// lhs_main = -ik nn G + H d.n_j, aux = (i/k) G, rhs = -G + (i/k) H (-d).n_i.
template <typename R>
__device__ __forceinline__ void bm_eval(R dx, R dy, R dz, const R (&ni)[3], const R (&nj)[3], R nn, R k, R kinv,
                                        R& lr, R& li, R& ar, R& ai, R& rr, R& ri) {
  R r, ir;
  inv_dist<R>(dx * dx + dy * dy + dz * dz, &r, &ir);
  const R kr = k * r;
  R s, c;
  sincos_t<R>(kr, &s, &c);
  const R gr = c * ir, gi = s * ir;
  const R ir2 = ir * ir;
  const R hr = (c + kr * s) * ir * ir2, hi = (s - kr * c) * ir * ir2;
  const R dnj = dx * nj[0] + dy * nj[1] + dz * nj[2];     // (y - x).n_j
  const R dni = -(dx * ni[0] + dy * ni[1] + dz * ni[2]);  // (x - y).n_i
  lr = k * nn * gi + hr * dnj;
  li = -k * nn * gr + hi * dnj;
  ar = -gi * kinv;
  ai = gr * kinv;
  rr = -gr - hi * dni * kinv;
  ri = -gi + hr * dni * kinv;
}

// Lanes per touching pair: the LN^4 Gauss points of the 4-D rule are split
// over 16 lanes when there are at most 16 of them (two pairs per warp, at
// the 2-point rule of the <2,3> orders), else over the whole warp.
template <int LN>
struct BmSingLanes {
  static constexpr int kPoints = LN * LN * LN * LN;
  static constexpr int kW = kPoints <= 16 ? 16 : 32;
  static constexpr int kPairsPerWarp = 32 / kW;
};

// One touching pair (index `local` of its type) on W = BmSingLanes<LN>::kW
// lanes (lane `sub` of them); the coincident pass also adds 1/2 M to lhs and
// -(i/(2k)) M to rhs.  `store` is false for the idle half of a warp whose
// last pair is missing (it computes a copy of a valid pair, for the
// shuffles, and adds nothing).
template <typename R, int NCOMMON, int LN>
__device__ __forceinline__ void singular_bm_pair(const BmProblem& P, int local, int sub, bool store) {
  constexpr int W = BmSingLanes<LN>::kW;
  const GeomView& g = P.g;
  int ti = local, tj = local;
  if (NCOMMON == 2) {
    ti = g.edge_pairs[local].x;
    tj = g.edge_pairs[local].y;
  } else if (NCOMMON == 1) {
    ti = g.vert_pairs[local].x;
    tj = g.vert_pairs[local].y;
  }
  const int s0 = g.triangles[3 * ti], s1 = g.triangles[3 * ti + 1], s2 = g.triangles[3 * ti + 2];
  const int t0 = g.triangles[3 * tj], t1 = g.triangles[3 * tj + 1], t2 = g.triangles[3 * tj + 2];
  const Perm6 pm = reorder6<NCOMMON>(s0, s1, s2, t0, t1, t2);
  const int pi_[3] = {pm.i0, pm.i1, pm.i2}, pj_[3] = {pm.j0, pm.j1, pm.j2};
  const int sv[3] = {s0, s1, s2}, tv[3] = {t0, t1, t2};
  R a[3][3], b[3][3], oa[3][3], ob[3][3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int va = sel3(s0, s1, s2, pi_[c]), vb = sel3(t0, t1, t2, pj_[c]);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      a[c][d] = (R)g.vertices[3 * va + d];
      b[c][d] = (R)g.vertices[3 * vb + d];
      oa[c][d] = (R)g.vertices[3 * sv[c] + d];
      ob[c][d] = (R)g.vertices[3 * tv[c] + d];
    }
  }
  R ni[3], nj[3], Ji, Jj;
  {
    const R e1[3] = {oa[1][0] - oa[0][0], oa[1][1] - oa[0][1], oa[1][2] - oa[0][2]};
    const R e2[3] = {oa[2][0] - oa[0][0], oa[2][1] - oa[0][1], oa[2][2] - oa[0][2]};
    const R cr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    Ji = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
    for (int d = 0; d < 3; d++) ni[d] = cr[d] / Ji;
  }
  {
    const R e1[3] = {ob[1][0] - ob[0][0], ob[1][1] - ob[0][1], ob[1][2] - ob[0][2]};
    const R e2[3] = {ob[2][0] - ob[0][0], ob[2][1] - ob[0][1], ob[2][2] - ob[0][2]};
    const R cr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    Jj = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
    for (int d = 0; d < 3; d++) nj[d] = cr[d] / Jj;
  }
  const R kk = (R)P.k, kinv = R(1) / kk;
  const R nn = ni[0] * nj[0] + ni[1] * nj[1] + ni[2] * nj[2];
  // t[4 e + (0, 1, 2, 3)] = (lhs re, lhs im, rhs re, rhs im) of block entry
  // e = 3 ii + jj (re-ordered slots), t[36], t[37] = the weight sum of the
  // curl term's (i/k) G; t[38..63] stay zero (padding for the reduction)
  R t[64];
#pragma unroll
  for (int e = 0; e < 64; e++) t[e] = 0;
  auto region = [&](R x1, R x2, R y1, R y2, R ww) {
    const R lx[3] = {R(1) - x1, x1 - x2, x2};
    const R ly[3] = {R(1) - y1, y1 - y2, y2};
    R xp[3], yp[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      xp[d] = lx[0] * a[0][d] + lx[1] * a[1][d] + lx[2] * a[2][d];
      yp[d] = ly[0] * b[0][d] + ly[1] * b[1][d] + ly[2] * b[2][d];
    }
    R lr, li, ar, ai, rr, ri;
    bm_eval<R>(yp[0] - xp[0], yp[1] - xp[1], yp[2] - xp[2], ni, nj, nn, kk, kinv, lr, li, ar, ai, rr, ri);
#pragma unroll
    for (int ii = 0; ii < 3; ii++)
#pragma unroll
      for (int jj = 0; jj < 3; jj++) {
        const R f = lx[ii] * ly[jj] * ww;
        const int e = 3 * ii + jj;
        t[4 * e] += lr * f;
        t[4 * e + 1] += li * f;
        t[4 * e + 2] += rr * f;
        t[4 * e + 3] += ri * f;
      }
    t[36] += ar * ww;
    t[37] += ai * ww;
  };
  const R jw = Ji * Jj / R(16);
  constexpr int NPT = BmSingLanes<LN>::kPoints;
#pragma unroll 1
  for (int pt = sub; pt < NPT; pt += W) {
    const int i0 = pt / (LN * LN * LN), i1 = (pt / (LN * LN)) % LN, i2 = (pt / LN) % LN, i3 = pt % LN;
    const R xi = R(0.5) * (R(gl_x<LN>(i0)) + R(1)), e1 = R(0.5) * (R(gl_x<LN>(i1)) + R(1));
    const R e2 = R(0.5) * (R(gl_x<LN>(i2)) + R(1)), e3 = R(0.5) * (R(gl_x<LN>(i3)) + R(1));
    const R w0 = R(gl_w<LN>(i0)) * R(gl_w<LN>(i1)) * R(gl_w<LN>(i2)) * R(gl_w<LN>(i3)) * jw;
    ss_regions<NCOMMON, R>(xi, e1, e2, e3, w0, region);
  }
  // transpose-reduce over the W lanes (xor offsets < W stay inside the
  // pair's lanes): every round halves the values a lane keeps, so lane `sub`
  // ends with the totals of values (64 / W) sub + i in t[i]
#pragma unroll
  for (int o = W / 2, half = 32; o >= 1; o >>= 1, half >>= 1) {
    const bool hi = (sub & o) != 0;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const R send = hi ? t[i] : t[i + half];
      const R keep = hi ? t[i + half] : t[i];
      t[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  // W = 16: lane e (< 9) holds entry e (lhs re, im, rhs re, im), lane 9 the
  // curl sums; W = 32: lane 2e holds entry e's lhs, lane 2e + 1 its rhs,
  // lane 18 the curl sums
  constexpr int kAuxLane = W == 16 ? 9 : 18;
  const R aux_re = __shfl_sync(0xffffffffu, t[0], kAuxLane, W);
  const R aux_im = __shfl_sync(0xffffffffu, t[1], kAuxLane, W);
  const int e = W == 16 ? sub : (sub >> 1);
  const bool do_lhs = W == 16 ? sub < 9 : (sub < 18 && (sub & 1) == 0);
  const bool do_rhs = W == 16 ? sub < 9 : (sub < 18 && (sub & 1) == 1);
  if (!store || !(do_lhs || do_rhs)) return;
  const int ii = e / 3, jj = e % 3;      // re-ordered slots
  const int ia = pi_[ii], jb = pj_[jj];  // original local vertices
  const R sc = R(kInv4Pi);
  const R m = NCOMMON == 3 ? R(0.5) * Ji * (ia == jb ? R(2) : R(1)) / R(12) : R(0);  // P1 mass: area (1 + [a == b]) / 12
  const size_t at = (size_t)sel3(s0, s1, s2, ia) * g.nv + sel3(t0, t1, t2, jb);
  if (do_lhs) {
    R cp = 0;
    for (int d = 0; d < 3; d++) cp += (R)g.curls[9 * ti + 3 * ia + d] * (R)g.curls[9 * tj + 3 * jb + d];
    R lre = (t[0] + aux_re * cp) * sc, lim = (t[1] + aux_im * cp) * sc;
    if (NCOMMON == 3) lre += R(0.5) * m;
    atomicAdd(&P.L[at], make_float2((float)lre, (float)lim));
  }
  if (do_rhs) {
    const int o = W == 16 ? 2 : 0;
    R rre = t[o] * sc, rim = t[o + 1] * sc;
    if (NCOMMON == 3) rim -= R(0.5) * kinv * m;
    atomicAdd(&P.R[at], make_float2((float)rre, (float)rim));
  }
}

// Pair index of this warp's lanes (kPairsPerWarp pairs per warp): `first` is
// the warp's first pair, `sub` the lane within the pair.
template <int LN>
__device__ __forceinline__ long long bm_sing_pair_index(long long* first, int* sub) {
  constexpr int W = BmSingLanes<LN>::kW, PPW = BmSingLanes<LN>::kPairsPerWarp;
  const int lane = threadIdx.x & 31;
  *first = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * PPW;
  *sub = lane & (W - 1);
  return *first + lane / W;
}

// The kernels of the three types and of the regular pairs only add to the
// matrices, so each may start while the one before it still runs (programmatic
// launch; each waits for it before it ends).  One launch for all types instead
// would have the FP64 type's registers for all: 127 us against 87 at 8286
// triangles.
template <typename R, int NCOMMON, int LN>
__global__ void __launch_bounds__(128) singular_bm_kernel(const __grid_constant__ BmProblem P, int npairs) {
  launch_next();
  long long first;
  int sub;
  const long long pair = bm_sing_pair_index<LN>(&first, &sub);
  if (first < npairs) {  // uniform over the warp
    const bool store = pair < npairs;
    singular_bm_pair<R, NCOMMON, LN>(P, (int)(store ? pair : first), sub, store);
  }
  wait_previous();
}

template <typename R, int NCOMMON, int LN>
__global__ void __launch_bounds__(128)
    singular_bm_batch_kernel(const BmHeader* __restrict__ hdr, const BmProblem* __restrict__ probs) {
  launch_next();
  constexpr int which = NCOMMON == 3 ? 0 : (NCOMMON == 2 ? 1 : 2);
  long long first;
  int sub;
  long long pair = bm_sing_pair_index<LN>(&first, &sub);
  const long long total = hdr->total_pairs[which];
  if (first < total) {  // uniform over the warp
    const bool store = pair < total;
    if (!store) pair = first;
    const BmProblem& P = probs[bm_find(probs, hdr->nproblems, pair, which)];
    singular_bm_pair<R, NCOMMON, LN>(P, (int)(pair - P.pair_begin[which]), sub, store);
  }
  wait_previous();
}

inline size_t al256(size_t x) { return (x + 255) / 256 * 256; }

int bm_sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

// Host staging of the batch descriptors (pinned, reused; one per host thread).
struct BmStage {
  void* buf = nullptr;
  size_t cap = 0;
  cudaEvent_t ev = nullptr;
  ~BmStage() {
    if (buf) cudaFreeHost(buf);
    if (ev) cudaEventDestroy(ev);
  }
};
thread_local BmStage t_bm_stage;

int bm_check(float k, const float2* L, const float2* R) {
  if (!L || !R) return BEM_ERR_INVALID_ARGUMENT;
  if (!std::isfinite(k)) return BEM_ERR_NONFINITE;
  if (k == 0.f) return BEM_ERR_INVALID_ARGUMENT;  // the Burton-Miller coupling i/k
  return BEM_OK;
}

// Persistent grid of a regular kernel.
template <int TN, typename KernelT>
int bm_grid(KernelT kernel, DeviceOnce& once, long long* grid) {
  const int smem = (int)(kStripWarps * sizeof(BmWarp<TN>));
  if (const int rc = once.shared_memory(kernel, smem)) return rc;
  int occ = 0;
  BEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kStripThreads, smem));
  *grid = (long long)bm_sm_count() * (occ > 0 ? occ : 1);
  return BEM_OK;
}

}  // namespace

size_t bm_workspace_bytes(int np) {
  return al256(sizeof(BmHeader)) + al256(sizeof(BmProblem) * (size_t)(np > 0 ? np : 1));
}

namespace {

template <int TN>
int bm_single_grid(long long* grid) {
  static DeviceOnce once;
  return bm_grid<TN>(regular_bm_kernel<TN>, once, grid);
}

template <int TN>
int bm_batch_grid(long long* grid) {
  static DeviceOnce once;
  return bm_grid<TN>(regular_bm_batch_kernel<TN>, once, grid);
}

int bm_rule(int order, int* tn) {
  if (order == BEM_ORDER_EXACT) *tn = 6;
  else if (order == BEM_ORDER_APPROX) *tn = 3;
  else if (order == BEM_ORDER_APPROX_1) *tn = 1;
  else return BEM_ERR_INVALID_ARGUMENT;
  return BEM_OK;
}

// The regular pairs first, then the touching pairs, which may start beside the
// launch before them: the many small blocks fill the regular kernel's last
// round (the other way round its equal shares start unequally late: 1617
// against 1516 us at 8286 triangles).
template <int LN, typename Kernel, typename... Args>
int bm_touch_launch(Kernel kernel, long long pairs, cudaStream_t s, Args... args) {
  if (pairs == 0) return BEM_OK;
  const int ppb = 4 * BmSingLanes<LN>::kPairsPerWarp;  // pairs per block of 4 warps
  EarlyLaunch l((unsigned)((pairs + ppb - 1) / ppb), 128, 0, s);
  BEM_CUDA_TRY(cudaLaunchKernelEx(&l.cfg, kernel, args...));
  count_launch();
  return BEM_OK;
}

template <int TN, typename Kernel, typename... Args>
int bm_regular_launch(Kernel kernel, long long grid, long long items, cudaStream_t s, Args... args) {
  (kernel<<<(unsigned)std::min(grid, (items + kStripWarps - 1) / kStripWarps), kStripThreads,
            kStripWarps * sizeof(BmWarp<TN>), s>>>(args...),
   count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

template <int TN, int LN>
int bm_single_launch(const BmProblem& P, long long grid, long long items, cudaStream_t s) {
  const GeomView& g = P.g;
  int rc;
  if ((rc = bm_regular_launch<TN>(regular_bm_kernel<TN>, grid * kStripRounds, items, s, P))) return rc;
  if ((rc = bm_touch_launch<LN>(singular_bm_kernel<double, 3, LN>, g.nt, s, P, g.nt))) return rc;
  if ((rc = bm_touch_launch<LN>(singular_bm_kernel<float, 2, LN>, g.n_edge, s, P, g.n_edge))) return rc;
  return bm_touch_launch<LN>(singular_bm_kernel<float, 1, LN>, g.n_vert, s, P, g.n_vert);
}

template <int TN, int LN>
int bm_batch_launch(BmHeader* dh, BmProblem* dp, long long grid, long long items, const long long* pairs,
                    cudaStream_t s) {
  const BmHeader* h = dh;
  const BmProblem* p = dp;
  int rc;
  if ((rc = bm_regular_launch<TN>(regular_bm_batch_kernel<TN>, grid, items, s, dh, p))) return rc;
  if ((rc = bm_touch_launch<LN>(singular_bm_batch_kernel<double, 3, LN>, pairs[0], s, h, p))) return rc;
  if ((rc = bm_touch_launch<LN>(singular_bm_batch_kernel<float, 2, LN>, pairs[1], s, h, p))) return rc;
  return bm_touch_launch<LN>(singular_bm_batch_kernel<float, 1, LN>, pairs[2], s, h, p);
}

}  // namespace

// lhs = BM_LHS + 1/2 M and rhs = BM_RHS - (i/(2k)) M of one problem (both
// nv x nv complex64, overwritten) at `order` (the reference's <2,3> for
// neumann2dirichlet; <4,6> gives its HBIE system).
int assemble_bm(const GeomView& g, int order, float k, float2* L, float2* R, cudaStream_t s) {
  int rc = bm_check(k, L, R), tn = 0;
  if (rc) return rc;
  if ((rc = bm_rule(order, &tn))) return rc;
  long long grid = 0;
  rc = tn == 6 ? bm_single_grid<6>(&grid) : (tn == 3 ? bm_single_grid<3>(&grid) : bm_single_grid<1>(&grid));
  if (rc) return rc;
  BEM_CUDA_TRY(cudaMemsetAsync(L, 0, sizeof(float2) * (size_t)g.nv * g.nv, s));
  BEM_CUDA_TRY(cudaMemsetAsync(R, 0, sizeof(float2) * (size_t)g.nv * g.nv, s));
  BmProblem P;
  std::memset(&P, 0, sizeof(P));
  P.g = g;
  P.k = k;
  P.items = strip_items(g.nv, g.nblocks, grid * kStripWarps, 1, 4, 0, kBmPanel, kBmPanelItems);
  P.L = L;
  P.R = R;
  const long long items = P.items.items;
  rc = tn == 6   ? bm_single_launch<6, 4>(P, grid, items, s)
       : tn == 3 ? bm_single_launch<3, 2>(P, grid, items, s)
                 : bm_single_launch<1, 2>(P, grid, items, s);
  if (rc) return rc;
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

// The same for many problems: one queue-driven launch over every problem's
// regular pairs, one launch per touching-pair type.
int assemble_bm_batch(const GeomView* views, const float* ks, float2* const* Ls, float2* const* Rs, int np, int order,
                      void* ws, size_t ws_bytes, cudaStream_t s) {
  if (np <= 0 || !views || !ks || !Ls || !Rs) return BEM_ERR_INVALID_ARGUMENT;
  if (!ws || ws_bytes < bm_workspace_bytes(np)) return BEM_ERR_WORKSPACE;
  int rc, tn = 0;
  for (int p = 0; p < np; p++)
    if ((rc = bm_check(ks[p], Ls[p], Rs[p]))) return rc;
  if ((rc = bm_rule(order, &tn))) return rc;
  long long grid = 0;
  rc = tn == 6 ? bm_batch_grid<6>(&grid) : (tn == 3 ? bm_batch_grid<3>(&grid) : bm_batch_grid<1>(&grid));
  if (rc) return rc;

  const size_t hbytes = al256(sizeof(BmHeader)), pbytes = sizeof(BmProblem) * (size_t)np;
  BmStage& st = t_bm_stage;
  if (!st.ev) BEM_CUDA_TRY(cudaEventCreateWithFlags(&st.ev, cudaEventDisableTiming));
  BEM_CUDA_TRY(cudaEventSynchronize(st.ev));  // the previous upload from the staging buffer is done
  if (st.cap < hbytes + pbytes) {
    if (st.buf) cudaFreeHost(st.buf);
    st.buf = nullptr;
    st.cap = 0;
    BEM_CUDA_TRY(cudaHostAlloc(&st.buf, 2 * (hbytes + pbytes), cudaHostAllocDefault));
    st.cap = 2 * (hbytes + pbytes);
  }
  BmHeader* hh = (BmHeader*)st.buf;
  BmProblem* hp = (BmProblem*)((char*)st.buf + hbytes);
  std::memset(hh, 0, sizeof(BmHeader));
  std::memset(hp, 0, pbytes);
  hh->nproblems = np;
  long long steps = 0;
  for (int p = 0; p < np; p++) steps += strip_steps(views[p].nblocks);
  // about 8 items per warp over the whole batch, at most 16 trial blocks each
  const long long share = std::min<long long>(512, std::max<long long>(4, steps / (8 * grid * kStripWarps)));
  long long items = 0, pairs[3] = {0, 0, 0};
  for (int p = 0; p < np; p++) {
    const GeomView& g = views[p];
    BEM_CUDA_TRY(cudaMemsetAsync(Ls[p], 0, sizeof(float2) * (size_t)g.nv * g.nv, s));
    BEM_CUDA_TRY(cudaMemsetAsync(Rs[p], 0, sizeof(float2) * (size_t)g.nv * g.nv, s));
    BmProblem& P = hp[p];
    P.g = g;
    P.k = ks[p];
    P.items = strip_items(g.nv, g.nblocks, std::max(1LL, strip_steps(g.nblocks) / share), 1, 4, 0, kBmPanel,
                          kBmPanelItems);
    P.item_begin = items;
    P.pair_begin[0] = pairs[0];
    P.pair_begin[1] = pairs[1];
    P.pair_begin[2] = pairs[2];
    pairs[0] += g.nt;
    pairs[1] += g.n_edge;
    pairs[2] += g.n_vert;
    items += P.items.items;
    P.L = Ls[p];
    P.R = Rs[p];
  }
  hh->total_items = items;
  for (int t = 0; t < 3; t++) hh->total_pairs[t] = pairs[t];
  BmHeader* dh = (BmHeader*)ws;
  BmProblem* dp = (BmProblem*)((char*)ws + hbytes);
  BEM_CUDA_TRY(cudaMemcpyAsync(ws, st.buf, hbytes + pbytes, cudaMemcpyHostToDevice, s));
  BEM_CUDA_TRY(cudaEventRecord(st.ev, s));
  rc = tn == 6   ? bm_batch_launch<6, 4>(dh, dp, grid, items, pairs, s)
       : tn == 3 ? bm_batch_launch<3, 2>(dh, dp, grid, items, pairs, s)
                 : bm_batch_launch<1, 2>(dh, dp, grid, items, pairs, s);
  if (rc) return rc;
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

// Reads and clears the flag that a Burton-Miller kernel's bounded wait
// expired (synchronises the stream).
int bm_status(int* err_host, cudaStream_t s) {
  int zero = 0;
  BEM_CUDA_TRY(cudaMemcpyFromSymbolAsync(err_host, g_bm_err, sizeof(int), 0, cudaMemcpyDeviceToHost, s));
  BEM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_bm_err, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, s));
  BEM_CUDA_TRY(cudaStreamSynchronize(s));
  return BEM_OK;
}

}  // namespace bemb
