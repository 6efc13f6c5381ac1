// Hand-written adjoint of the listener pressures p = -S g + D u with
// (1/2 M - K) u = -V g (src/bem/solver.py:97-104,140-147).
//
// For a loss with gradient pbar = dL/dp* (PyTorch's convention),
//   lambda = (1/2 M - K)^{-H} D^H pbar                      (adjoint solve)
//   dL/dg* = -S^H pbar - V^H lambda
//   dL/dx  = Re[ -pbar^H dS g + pbar^H dD u - lambda^H dV g
//                - 1/2 lambda^H dM u + lambda^H dK u ]       (vertex coordinates)
// The second line needs only conjugate-transposed applications; the last is
// a "kernel-derivative assembly": one pass over every triangle pair (and
// listener-triangle pair) differentiates the quadrature sum through the
// quadrature points, the areas and the trial normals, contracted with the
// vectors on the fly, so no derivative matrix is ever stored.
//
// With G = e^{ikr}/(4 pi r), d = y - x, f = G'(r)/r, the double-layer kernel
// is K = f (d.n_y) and, for a pair term F = a (bV G + bK K):
//   grad_y F = (a bV f + a bK f' (d.n)/r) d + a bK f n,  grad_x F = -grad_y F,
//   grad_n F = a bK f d,
// with the reference's clamp r -> max(r, 1e-3) (potential.h:21-23): inside it
// G and K's radial factor are constant, so their r-derivatives vanish.

#include <algorithm>
#include <cmath>

#include "async_copy.cuh"
#include "bem_common.cuh"
#include "sauter_schwab.cuh"
#include "strip.cuh"

namespace bemb {

int geom_view(const void* geom, GeomView* v, GeomHeader* out_hdr);

namespace {

// sine and cosine of a phase k r in the regular pairs
__device__ __forceinline__ void sincos_phase(float x, float* s, float* c) { __sincosf(x, s, c); }

// One quadrature-point pair.  Accumulates (all times W):
//   F  += Re(a (bV G + bK K))
//   gy += grad_y Re(...)     (grad_x is its negative)
//   gn += grad_n Re(...)
__device__ __forceinline__ void point_grad(const float d[3], const float n[3], float k, float ar, float ai, float bvr,
                                           float bvi, float bkr, float bki, float W, float& F, float gy[3],
                                           float gn[3]) {
  float r = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  const bool clamped = r < kEps;
  if (clamped) r = kEps;
  const float u = 1.f / r;
  float s, c;
  sincosf(k * r, &s, &c);
  const float Gr = u * c, Gi = u * s;                                     // G (without 1/4pi)
  const float Gpr = u * (-u * c - k * s), Gpi = u * (-u * s + k * c);     // G'
  const float fr = Gpr * u, fi = Gpi * u;                                 // f = G'/r
  const float t1 = 2.f * u * u - k * k, t2 = -2.f * k * u;
  const float Gppr = Gr * t1 - Gi * t2, Gppi = Gr * t2 + Gi * t1;         // G''
  const float fpr = (Gppr - Gpr * u) * u, fpi = (Gppi - Gpi * u) * u;     // f'
  const float dn = d[0] * n[0] + d[1] * n[1] + d[2] * n[2];
  const float aVr = ar * bvr - ai * bvi, aVi = ar * bvi + ai * bvr;       // a bV
  const float aKr = ar * bkr - ai * bki, aKi = ar * bki + ai * bkr;       // a bK
  const float ReG = aVr * Gr - aVi * Gi;
  const float ReK = (aKr * fr - aKi * fi) * dn;
  F += W * (ReG + ReK);
  const float ReAVf = clamped ? 0.f : (aVr * fr - aVi * fi);
  const float ReAKfp = clamped ? 0.f : (aKr * fpr - aKi * fpi);
  const float c1 = W * (ReAVf + ReAKfp * dn * u);
  const float c2 = W * (aKr * fr - aKi * fi);
#pragma unroll
  for (int e = 0; e < 3; e++) {
    gy[e] += c1 * d[e] + c2 * n[e];
    gn[e] += c2 * d[e];
  }
}

// d(area)/d(v_c) = 1/2 n x (v_{c+2} - v_{c+1});   normal chain:
// d(E)/d(v_c) += (v_{c+1} - v_{c+2}) x t,  t = (I - n n^T) dE/dn / |c|.
template <typename R>
__device__ __forceinline__ void area_normal_grad(const R v[3][3], R dE_dA_over, const R dEdn[3], bool use_n,
                                                 R out[3][3]) {
  const R e1[3] = {v[1][0] - v[0][0], v[1][1] - v[0][1], v[1][2] - v[0][2]};
  const R e2[3] = {v[2][0] - v[0][0], v[2][1] - v[0][1], v[2][2] - v[0][2]};
  const R cr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
  const R cn = sqrt(cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
  const R n[3] = {cr[0] / cn, cr[1] / cn, cr[2] / cn};
  R t[3] = {0, 0, 0};
  if (use_n) {
    const R nd = n[0] * dEdn[0] + n[1] * dEdn[1] + n[2] * dEdn[2];
    for (int e = 0; e < 3; e++) t[e] = (dEdn[e] - nd * n[e]) / cn;
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
    const R ea[3] = {v[c2][0] - v[c1][0], v[c2][1] - v[c1][1], v[c2][2] - v[c1][2]};  // v_{c+2} - v_{c+1}
    // 1/2 n x ea, scaled by dE/dA
    const R ag[3] = {R(0.5) * (n[1] * ea[2] - n[2] * ea[1]), R(0.5) * (n[2] * ea[0] - n[0] * ea[2]),
                     R(0.5) * (n[0] * ea[1] - n[1] * ea[0])};
    const R eb[3] = {-ea[0], -ea[1], -ea[2]};  // v_{c+1} - v_{c+2}
    const R ng[3] = {eb[1] * t[2] - eb[2] * t[1], eb[2] * t[0] - eb[0] * t[2], eb[0] * t[1] - eb[1] * t[0]};
#pragma unroll
    for (int e = 0; e < 3; e++) out[c][e] = dE_dA_over * ag[e] + ng[e];
  }
}

__device__ __forceinline__ double2 lerp3(const float2* vec, int v0, int v1, int v2, double l0, double l1, double l2) {
  const float2 a = vec[v0], b = vec[v1], c = vec[v2];
  return make_double2(l0 * a.x + l1 * b.x + l2 * c.x, l0 * a.y + l1 * b.y + l2 * c.y);
}

// ---------------------------------------------------------------------------
// Regular pairs (touching pairs masked), each unordered pair once.  A warp owns
// a 32-triangle test block (a triangle per lane) and walks along the trial
// triangles as the assembly does (strip.cuh): the pair (i, j) and its mirror
// (j, i) share r, the sincos and the kernel's derivatives.  With
//   G = e^{ikr} / r,  h = -G'/r = (1 - ikr) G / r^2,  e = (G'/r)'/r = (3 h - k^2 G) / r^2,
// d = y - x, dj = d.n_j (a function of the test point p), di = -d.n_i (of the
// trial point q), and the products of both orders, l = lambda conjugated,
//   Y = l_p g_q + l_q g_p,  Z2 = l_p u_q,  Z3 = l_q u_p,
// the pair adds F = -Re[Y G] - dj Re[Z2 h] - di Re[Z3 h] to the energy, and
//   grad_y F = -grad_x F = c1 d - m2 n_j + m3 n_i,
//   c1 = Re[Y h] + dj Re[Z2 e] + di Re[Z3 e],  m2 = Re[Z2 h],  m3 = Re[Z3 h],
//   grad_{n_j} F = -m2 d,  grad_{n_i} F = m3 d
// (c1 = 0 where r is clamped).  m2 and m3 are only summed over p and over q;
// the terms with n_j, n_i, dj, di and the normals' gradients follow from those
// sums once per pair.
//
// Bound by the FP32 pipe: about 64 operations per unordered point pair, on
// packed pairs (the two points of a trial vertex).  Measured on B200 with 5120
// triangles: 1.43 ms (FP32 pipe 71 % of its cycles), against 12.0 ms for ordered
// pairs with the densities interpolated in FP64 for every pair and library sincos
// calls.  Vertex gradients, 300 to 8000 triangles at 130 to 1300 Hz, are 0.1 to
// 0.7 times as far off 64 bits as those (FP64 sums over the blocks outweigh the
// hardware's sincos).
// ---------------------------------------------------------------------------
constexpr int kAdjThreads = 128;
constexpr int kAdjWarps = kAdjThreads / 32;

struct AdjWarp {
  TriRec trial[2][kBlock];
  float2 val[kBlock][18];   // trial points (b, b + 3): lambda, g, u (re, im) times the rule's weight
  float xs[18][32];         // test points
  float ps[36][32];         // 6 p + {lambda, g, u} (re, im) times the rule's weight
  float out[kBlock][13];    // a trial triangle's corners, energy and normal, summed over the test block
  double sum[13][32];       // the test triangles' own
  uint64_t full[2];
};

// lambda, g, u at the six points of triangle r, times the rule's weights.
__device__ __forceinline__ void adj_values(const TriRec& r, const float2* lam, const float2* gvec, const float2* uvec,
                                           float (&out)[36]) {
  const float2* src[3] = {lam, gvec, uvec};
#pragma unroll
  for (int f = 0; f < 3; f++) {
    const float2 v[3] = {src[f][r.v[0]], src[f][r.v[1]], src[f][r.v[2]]};
#pragma unroll
    for (int q = 0; q < 6; q++) {
      double re = 0.0, im = 0.0;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        re += tri6_w(q) * tri6_phi(q, b) * v[b].x;
        im += tri6_w(q) * tri6_phi(q, b) * v[b].y;
      }
      out[6 * q + 2 * f] = (float)re;
      out[6 * q + 2 * f + 1] = (float)im;
    }
  }
}

// Adds the sums of triangle r (corners 0..8, energy 9, normal 10..12).
__device__ __forceinline__ void adj_store(const GeomView& g, const TriRec& r, const double (&t)[13],
                                          double* __restrict__ grad) {
  // the area and the normal follow the vertices in input order (the sorted
  // record may hold them in another order): the cross product's sign is the
  // stored normal's
  double v[3][3];
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) v[c][e] = g.vertices[3 * r.v[c] + e];
  const double e1[3] = {v[1][0] - v[0][0], v[1][1] - v[0][1], v[1][2] - v[0][2]};
  const double e2[3] = {v[2][0] - v[0][0], v[2][1] - v[0][1], v[2][2] - v[0][2]};
  const double side = (e1[1] * e2[2] - e1[2] * e2[1]) * r.n[0] + (e1[2] * e2[0] - e1[0] * e2[2]) * r.n[1] +
                      (e1[0] * e2[1] - e1[1] * e2[0]) * r.n[2];
  const double sgn = side < 0.0 ? -1.0 : 1.0;
  const double dEdn[3] = {sgn * t[10], sgn * t[11], sgn * t[12]};
  double out[3][3];
  area_normal_grad<double>(v, t[9] / (double)r.area, dEdn, true, out);
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) atomicAdd(&grad[3 * r.v[c] + e], t[3 * c + e] + out[c][e]);
}

__global__ void __launch_bounds__(kAdjThreads, 2)
    grad_regular_kernel(const __grid_constant__ GeomView g, float k, const float2* __restrict__ lam,
                        const float2* __restrict__ gvec, const float2* __restrict__ uvec, double* __restrict__ grad,
                        long long chunk, long long n_steps) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  AdjWarp& sw = reinterpret_cast<AdjWarp*>(smem_raw)[threadIdx.x >> 5];
  launch_next();
  const int lane = threadIdx.x & 31, nb = g.nblocks;
  if (lane == 0) {
    mbar_init(&sw.full[0], 1);
    mbar_init(&sw.full[1], 1);
    mbar_init_fence();
  }
  __syncwarp();
  auto fetch = [&](int jb, int b) {
    const uint32_t bytes = (uint32_t)(min(kBlock, g.nt - jb * kBlock) * sizeof(TriRec));
    mbar_expect_tx(&sw.full[b], bytes);
    bulk_load(sw.trial[b], &g.rec[jb * kBlock], bytes, &sw.full[b]);
  };
  long long pos = ((long long)blockIdx.x * kAdjWarps + (threadIdx.x >> 5)) * chunk;
  const long long end = pos + chunk < n_steps ? pos + chunk : n_steps;
  if (pos >= end) return;  // uniform over the warp
  int grp = tile_group_of(pos >> 5, nb), jb = grp + (int)((pos >> 5) - tile_units_before(grp, nb)), cur = -1;
  if (lane == 0) fetch(jb, 0);
  TriRec ri;  // the lane's triangle
  bool valid = false;
  auto store_test = [&]() {
    double t[13];
#pragma unroll
    for (int e = 0; e < 13; e++) t[e] = sw.sum[e][lane];
    if (valid) adj_store(g, ri, t, grad);
  };
  const float2 k2 = f2(k), nk2 = f2(-k), nkk2 = f2(-k * k);
  for (unsigned uses = 0; pos < end; uses++) {
    const int t0 = (int)(pos & 31), t1 = (int)(end - pos < 32 - t0 ? t0 + (end - pos) : 32), bf = uses & 1;
    pos += t1 - t0;
    int next_grp = grp, next_jb = jb + 1;
    if (next_jb == nb) next_jb = ++next_grp;
    __syncwarp();  // every lane is done with buffer bf ^ 1, with val and with out
    if (lane == 0 && pos < end) fetch(next_jb, bf ^ 1);
    if (grp != cur) {
      if (cur >= 0) store_test();
      cur = grp;
      valid = grp * kBlock + lane < g.nt;
      ri = g.rec[valid ? grp * kBlock + lane : g.nt - 1];
      float v[36];
      adj_values(ri, lam, gvec, uvec, v);
#pragma unroll
      for (int e = 0; e < 36; e++) sw.ps[e][lane] = v[e];
#pragma unroll
      for (int e = 0; e < 18; e++) sw.xs[e][lane] = ri.qp[e];
#pragma unroll
      for (int e = 0; e < 13; e++) sw.sum[e][lane] = 0.0;
    }
    if (!mbar_wait(&sw.full[bf], (uses >> 1) & 1u, g.err)) mbar_wait_drain(&sw.full[bf], (uses >> 1) & 1u);
    const int ntri = min(kBlock, g.nt - jb * kBlock), stop = min(t1, ntri);
    if (lane < ntri) {  // the values at the trial points, a triangle per lane
      float v[36];
      adj_values(sw.trial[bf][lane], lam, gvec, uvec, v);
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int f = 0; f < 6; f++) sw.val[lane][6 * b + f] = make_float2(v[6 * b + f], v[6 * (b + 3) + f]);
    }
    __syncwarp();
    float gi[9], Ni[3] = {0.f, 0.f, 0.f}, Fi = 0.f;  // test side, over the block
#pragma unroll
    for (int e = 0; e < 9; e++) gi[e] = 0.f;
#pragma unroll 1
    for (int t = t0; t < stop; t++) {
      const TriRec& rj = sw.trial[bf][t];
      const int j0 = rj.v[0], j1 = rj.v[1], j2 = rj.v[2];
      const bool touching = (ri.v[0] == j0) | (ri.v[0] == j1) | (ri.v[0] == j2) | (ri.v[1] == j0) |
                            (ri.v[1] == j1) | (ri.v[1] == j2) | (ri.v[2] == j0) | (ri.v[2] == j1) | (ri.v[2] == j2);
      const bool once = jb > grp || t > lane;  // on the test block itself each unordered pair once
      const float W = (valid && !touching && once) ? ri.area * rj.area * kInv4Pi : 0.f;
      float red[16];
#pragma unroll
      for (int e = 0; e < 16; e++) red[e] = 0.f;
      if (__any_sync(0xffffffffu, W != 0.f)) {
        const float nj[3] = {rj.n[0], rj.n[1], rj.n[2]}, cj[3] = {rj.c[0], rj.c[1], rj.c[2]};
        float2 y[3][3], di[3], U[3][3], s2[3], s3[3];
#pragma unroll
        for (int b = 0; b < 3; b++) {
#pragma unroll
          for (int e = 0; e < 3; e++) {
            y[b][e] = make_float2(rj.qp[3 * b + e], rj.qp[9 + 3 * b + e]);
            U[b][e] = make_float2(0.f, 0.f);
          }
          di[b] = f2_fma(f2(ri.n[0]), f2_sub(f2(ri.c[0]), y[b][0]),
                         f2_fma(f2(ri.n[1]), f2_sub(f2(ri.c[1]), y[b][1]),
                                f2_mul(f2(ri.n[2]), f2_sub(f2(ri.c[2]), y[b][2]))));
          s2[b] = s3[b] = make_float2(0.f, 0.f);
        }
        float2 yg = make_float2(0.f, 0.f);  // sum of Re[Y G]
        float F = 0.f;
        float nsi[3] = {0.f, 0.f, 0.f}, nsj[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
        for (int o = 0; o < 2; o++) {  // orbit of the test points
          const float own = (float)(o == 0 ? 1.0 - 3.0 * kTriA1 : 1.0 - 3.0 * kTriA2),
                      all = (float)(o == 0 ? kTriA1 : kTriA2);
#pragma unroll
          for (int a = 0; a < 3; a++) {
            const int p = 3 * o + a;
            const float x[3] = {sw.xs[3 * p][lane], sw.xs[3 * p + 1][lane], sw.xs[3 * p + 2][lane]};
            const float dj = nj[0] * (cj[0] - x[0]) + nj[1] * (cj[1] - x[1]) + nj[2] * (cj[2] - x[2]);
            const float* ps = &sw.ps[6 * p][lane];
            const float2 plr = f2(ps[0]), pli = f2(ps[32]), pnlr = f2(-ps[0]), pgr = f2(ps[64]), pgi = f2(ps[96]),
                         pngi = f2(-ps[96]), pur = f2(ps[128]), pui = f2(ps[160]), pnui = f2(-ps[160]);
            float2 T[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}}, t2 = make_float2(0.f, 0.f), t3 = t2;
#pragma unroll
            for (int b = 0; b < 3; b++) {
              const float2 dx = f2_sub(y[b][0], f2(x[0])), dy = f2_sub(y[b][1], f2(x[1])),
                           dz = f2_sub(y[b][2], f2(x[2]));
              const float2 q2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
              const float2 r2 = make_float2(fmaxf(q2.x, kEps * kEps), fmaxf(q2.y, kEps * kEps));
              const float2 u = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
              const float2 kr = f2_mul(k2, f2_mul(r2, u)), u2 = f2_mul(u, u);
              float2 sn, cs;
              sincos_phase(kr.x, &sn.x, &cs.x);
              sincos_phase(kr.y, &sn.y, &cs.y);
              const float2 Gr = f2_mul(cs, u), Gi = f2_mul(sn, u);
              const float2 hr = f2_mul(f2_fma(k2, sn, Gr), u2), hi = f2_mul(f2_fma(nk2, cs, Gi), u2);
              const float2 er = f2_mul(f2_fma(nkk2, Gr, f2_mul(f2(3.f), hr)), u2),
                           ei = f2_mul(f2_fma(nkk2, Gi, f2_mul(f2(3.f), hi)), u2);
              const float2* qv = &sw.val[t][6 * b];
              const float2 qlr = qv[0], qli = qv[1], qgr = qv[2], qgi = qv[3], qur = qv[4], qui = qv[5];
              // real parts and negated imaginary parts
              const float2 Yr = f2_fma(plr, qgr, f2_fma(pli, qgi, f2_fma(qlr, pgr, f2_mul(qli, pgi))));
              const float2 Yn = f2_fma(pli, qgr, f2_fma(pnlr, qgi, f2_fma(qli, pgr, f2_mul(qlr, pngi))));
              const float2 Z2r = f2_fma(plr, qur, f2_mul(pli, qui)), Z2n = f2_fma(pli, qur, f2_mul(pnlr, qui));
              const float2 Z3r = f2_fma(qlr, pur, f2_mul(qli, pui)), Z3n = f2_fma(qli, pur, f2_mul(qlr, pnui));
              yg = f2_fma(Yr, Gr, f2_fma(Yn, Gi, yg));
              const float2 m2 = f2_fma(Z2r, hr, f2_mul(Z2n, hi)), m3 = f2_fma(Z3r, hr, f2_mul(Z3n, hi));
              const float2 w2 = f2_fma(Z2r, er, f2_mul(Z2n, ei)), w3 = f2_fma(Z3r, er, f2_mul(Z3n, ei));
              float2 c1 = f2_fma(Yr, hr, f2_fma(Yn, hi, f2_fma(f2(dj), w2, f2_mul(di[b], w3))));
              c1.x = q2.x < kEps * kEps ? 0.f : c1.x;
              c1.y = q2.y < kEps * kEps ? 0.f : c1.y;
              T[0] = f2_fma(c1, dx, T[0]);
              T[1] = f2_fma(c1, dy, T[1]);
              T[2] = f2_fma(c1, dz, T[2]);
              U[b][0] = f2_fma(c1, dx, U[b][0]);
              U[b][1] = f2_fma(c1, dy, U[b][1]);
              U[b][2] = f2_fma(c1, dz, U[b][2]);
              t2 = f2_add(t2, m2);
              t3 = f2_add(t3, m3);
              s2[b] = f2_add(s2[b], m2);
              s3[b] = f2_add(s3[b], m3);
            }
            const float p2 = t2.x + t2.y, p3 = t3.x + t3.y;
            F = fmaf(-dj, p2, F);
#pragma unroll
            for (int e = 0; e < 3; e++) {
              // grad_x = -(sum c1 d - m2 n_j + m3 n_i)
              const float gx = -W * (T[e].x + T[e].y - p2 * nj[e] + p3 * ri.n[e]);
#pragma unroll
              for (int c = 0; c < 3; c++) gi[3 * c + e] = fmaf(c == a ? own + all : all, gx, gi[3 * c + e]);
              nsj[e] = fmaf(p2, x[e] - cj[e], nsj[e]);    // -sum m2 d, test part
              nsi[e] = fmaf(-p3, x[e] - ri.c[e], nsi[e]);  // sum m3 d, test part
            }
          }
        }
        // trial side
        const float sI[3] = {ri.n[0], ri.n[1], ri.n[2]};
#pragma unroll
        for (int b = 0; b < 3; b++) {
          F -= di[b].x * s3[b].x + di[b].y * s3[b].y;
#pragma unroll
          for (int e = 0; e < 3; e++) {
            const float u1 = U[b][e].x - s2[b].x * nj[e] + s3[b].x * sI[e];
            const float u2 = U[b][e].y - s2[b].y * nj[e] + s3[b].y * sI[e];
#pragma unroll
            for (int c = 0; c < 3; c++)
              red[3 * c + e] += (float)tri6_phi(b, c) * u1 + (float)tri6_phi(b + 3, c) * u2;
            nsj[e] -= s2[b].x * (y[b][e].x - cj[e]) + s2[b].y * (y[b][e].y - cj[e]);
            nsi[e] += s3[b].x * (y[b][e].x - ri.c[e]) + s3[b].y * (y[b][e].y - ri.c[e]);
          }
        }
        F -= yg.x + yg.y;
        Fi = fmaf(W, F, Fi);
#pragma unroll
        for (int e = 0; e < 3; e++) Ni[e] = fmaf(W, nsi[e], Ni[e]);
#pragma unroll
        for (int e = 0; e < 9; e++) red[e] *= W;
        red[9] = W * F;
#pragma unroll
        for (int e = 0; e < 3; e++) red[10 + e] = W * nsj[e];
      }
      // sums over the lanes: every round halves the values a lane keeps, lane
      // 2 v (and 2 v + 1) ends with value v
#pragma unroll
      for (int o = 16, half = 8; half >= 1; o >>= 1, half >>= 1) {
        const bool hi = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < half; i++) {
          const float send = hi ? red[i] : red[i + half];
          const float keep = hi ? red[i + half] : red[i];
          red[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      red[0] += __shfl_xor_sync(0xffffffffu, red[0], 1);
      if ((lane & 1) == 0 && lane < 26) sw.out[t][lane >> 1] = red[0];
    }
#pragma unroll
    for (int e = 0; e < 9; e++) sw.sum[e][lane] += (double)gi[e];
    sw.sum[9][lane] += (double)Fi;
#pragma unroll
    for (int e = 0; e < 3; e++) sw.sum[10 + e][lane] += (double)Ni[e];
    __syncwarp();  // out is complete
    if (lane >= t0 && lane < stop) {
      double t[13];
#pragma unroll
      for (int e = 0; e < 13; e++) t[e] = (double)sw.out[lane][e];
      adj_store(g, sw.trial[bf][lane], t, grad);
    }
    grp = next_grp;
    jb = next_jb;
  }
  store_test();
}

// ---------------------------------------------------------------------------
// Touching pairs: Sauter-Schwab points (sauter_schwab.cuh), a warp per pair, in
// the notation of the regular pairs.  The difference runs in the triangles'
// edges from the shared vertex (d = y1 F1 + y2 F2 - x1 E1 - x2 E2), and values
// at the points in the densities' differences along them.
//   * coincident pairs (FP64): three of the six regions, each with its mirror.
//     d lies in the plane, so only c1 = Re[Y h] and m = Re[(Z3 - Z2) h] remain,
//     summed with the coordinates of d in E1 and E2;
//   * common edge (FP64): ordered pairs;
//   * common vertex (FP32): the two regions are mirrors, so each unordered pair
//     once.
// Measured on B200 with 5120 triangles: 458 us in one launch beside the other
// terms, against 121 + 329 + 250 us with six regions, library sincos, square
// roots and divisions, and both orders of the vertex pairs.
// ---------------------------------------------------------------------------
struct AdjTouchShared {
  double c[kAdjWarps][32];
  float f[kAdjWarps][32];
};

// The three vertices' values of a density as value and differences along the
// edges: f(x1, x2) = f0 + x1 (f1 - f0) + x2 (f2 - f1).
template <typename R>
struct Along {
  R re[3], im[3];
  __device__ __forceinline__ void load(const float2* f, const int (&v)[3]) {
    const float2 a = f[v[0]], b = f[v[1]], c = f[v[2]];
    re[0] = (R)a.x;
    im[0] = (R)a.y;
    re[1] = (R)b.x - (R)a.x;
    im[1] = (R)b.y - (R)a.y;
    re[2] = (R)c.x - (R)b.x;
    im[2] = (R)c.y - (R)b.y;
  }
  __device__ __forceinline__ void at(R x1, R x2, R& r, R& i) const {
    r = re[0] + x1 * re[1] + x2 * re[2];
    i = im[0] + x1 * im[1] + x2 * im[2];
  }
};

// r >= 1e-3 clamped: 1/r, e^{ikr}/r and (1 - ikr) e^{ikr}/r^3; true if not clamped.
template <typename R>
__device__ __forceinline__ bool touch_kernel(R q2, R k, R& u, R& Gr, R& Gi, R& hr, R& hi) {
  const bool free = q2 >= (R)kEps * (R)kEps;
  R r;
  inv_dist<R>(q2, &r, &u);
  R s, c;
  sincos_t<R>(k * r, &s, &c);
  Gr = c * u;
  Gi = s * u;
  hr = (Gr + k * s) * u * u;
  hi = (Gi - k * c) * u * u;
  return free;
}

__device__ __forceinline__ void adj_add(double* __restrict__ grad, const int (&v)[3], const double (&t)[3][3]) {
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) atomicAdd(&grad[3 * v[c] + e], t[c][e]);
}

__device__ __forceinline__ void grad_coincident(const GeomView& g, int ti, float kf, const float2* __restrict__ lam,
                                                const float2* __restrict__ gvec, const float2* __restrict__ uvec,
                                                double* __restrict__ grad, double* total) {
  const int lane = threadIdx.x & 31;
  const int v[3] = {g.triangles[3 * ti], g.triangles[3 * ti + 1], g.triangles[3 * ti + 2]};
  double p[3][3], E1[3], E2[3], n[3];
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) p[c][e] = (double)g.vertices[3 * v[c] + e];
#pragma unroll
  for (int e = 0; e < 3; e++) {
    E1[e] = p[1][e] - p[0][e];
    E2[e] = p[2][e] - p[1][e];
  }
  n[0] = E1[1] * E2[2] - E1[2] * E2[1];
  n[1] = E1[2] * E2[0] - E1[0] * E2[2];
  n[2] = E1[0] * E2[1] - E1[1] * E2[0];
  const double J = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
  const double g11 = E1[0] * E1[0] + E1[1] * E1[1] + E1[2] * E1[2], g22 = E2[0] * E2[0] + E2[1] * E2[1] + E2[2] * E2[2],
               g12 = 2.0 * (E1[0] * E2[0] + E1[1] * E2[1] + E1[2] * E2[2]);
  Along<double> L, G, U;
  L.load(lam, v);
  G.load(gvec, v);
  U.load(uvec, v);
  const double k = (double)kf, jw = J * J / 16.0 * (double)kInv4Pi;
  // sums: energy, m times the coordinates of d, and for corners 1 and 2 (their
  // shape functions' differences sum to zero) c1 times them and m
  double t[9];
#pragma unroll
  for (int e = 0; e < 9; e++) t[e] = 0.0;
  auto region = [&](double x1, double x2, double y1, double y2, double w) {
    const double a = y1 - x1, b = y2 - x2;
    double u, Gr, Gi, hr, hi;
    const bool free = touch_kernel<double>(a * (a * g11 + b * g12) + b * b * g22, k, u, Gr, Gi, hr, hi);
    double lxr, lxi, lyr, lyi, gxr, gxi, gyr, gyi, uxr, uxi, uyr, uyi;
    L.at(x1, x2, lxr, lxi);
    L.at(y1, y2, lyr, lyi);
    G.at(x1, x2, gxr, gxi);
    G.at(y1, y2, gyr, gyi);
    U.at(x1, x2, uxr, uxi);
    U.at(y1, y2, uyr, uyi);
    // conj(l_x) g_y + conj(l_y) g_x and conj(l_y) u_x - conj(l_x) u_y: real and negated imaginary parts
    const double Yr = lxr * gyr + lxi * gyi + lyr * gxr + lyi * gxi, Yn = lxi * gyr - lxr * gyi + lyi * gxr - lyr * gxi;
    const double Zr = lyr * uxr + lyi * uxi - lxr * uyr - lxi * uyi, Zn = lyi * uxr - lyr * uxi - lxi * uyr + lxr * uyi;
    t[0] -= w * (Yr * Gr + Yn * Gi);
    const double c1 = free ? w * (Yr * hr + Yn * hi) : 0.0, m = w * (Zr * hr + Zn * hi);
    t[1] += m * a;
    t[2] += m * b;
    // shape functions 1 - s, s - t, t at (s, t) = y minus those at x
    const double d1 = a - b, d2 = b, ca = c1 * a, cb = c1 * b;
    t[3] += d1 * ca;
    t[4] += d1 * cb;
    t[5] += d1 * m;
    t[6] += d2 * ca;
    t[7] += d2 * cb;
    t[8] += d2 * m;
  };
#pragma unroll 1
  for (int pt = lane; pt < 256; pt += 32) {
    const int i0 = pt >> 6, i1 = (pt >> 4) & 3, i2 = (pt >> 2) & 3, i3 = pt & 3;
    const double xi = 0.5 * (gl4_x(i0) + 1.0), e1 = 0.5 * (gl4_x(i1) + 1.0), e2 = 0.5 * (gl4_x(i2) + 1.0),
                 e3 = 0.5 * (gl4_x(i3) + 1.0);
    const double e12 = e1 * e2, e123 = e12 * e3;
    const double sc = xi * xi * xi * e1 * e1 * e2 * gl4_w(i0) * gl4_w(i1) * gl4_w(i2) * gl4_w(i3) * jw;
    region(xi, xi * (1.0 - e1 + e12), xi * (1.0 - e123), xi * (1.0 - e1), sc);
    region(xi, xi * (e1 - e12 + e123), xi * (1.0 - e12), xi * (e1 - e12), sc);
    region(xi * (1.0 - e123), xi * (e1 - e123), xi, xi * (e1 - e12), sc);
  }
  warp_totals<9>(t, total);
  if (lane == 0) {
    double N[3], out[3][3], add[3][3];
#pragma unroll
    for (int e = 0; e < 3; e++) N[e] = total[1] * E1[e] + total[2] * E2[e];
    // weight J^2: both areas are this triangle's
    area_normal_grad<double>(p, 2.0 * total[0] / (0.5 * J), N, true, out);
#pragma unroll
    for (int e = 0; e < 3; e++) {
      const double q1 = total[3] * E1[e] + total[4] * E2[e] + total[5] * n[e] / J;
      const double q2 = total[6] * E1[e] + total[7] * E2[e] + total[8] * n[e] / J;
      add[0][e] = out[0][e] - q1 - q2;
      add[1][e] = out[1][e] + q1;
      add[2][e] = out[2][e] + q2;
    }
    adj_add(grad, v, add);
  }
}

// Pair (ti, tj) with a common edge (NCOMMON = 2, ordered) or a common vertex
// (NCOMMON = 1, unordered: with its mirror).
template <typename R, int NCOMMON>
__device__ __forceinline__ void grad_touch(const GeomView& g, int ti, int tj, float kf, const float2* __restrict__ lam,
                                           const float2* __restrict__ gvec, const float2* __restrict__ uvec,
                                           double* __restrict__ grad, R* total) {
  constexpr bool kMirror = NCOMMON == 1;
  const int lane = threadIdx.x & 31;
  const int s[3] = {g.triangles[3 * ti], g.triangles[3 * ti + 1], g.triangles[3 * ti + 2]};
  const int r[3] = {g.triangles[3 * tj], g.triangles[3 * tj + 1], g.triangles[3 * tj + 2]};
  const Perm6 pm = reorder6<NCOMMON>(s[0], s[1], s[2], r[0], r[1], r[2]);
  const int vi[3] = {sel3(s[0], s[1], s[2], pm.i0), sel3(s[0], s[1], s[2], pm.i1), sel3(s[0], s[1], s[2], pm.i2)};
  const int vj[3] = {sel3(r[0], r[1], r[2], pm.j0), sel3(r[0], r[1], r[2], pm.j1), sel3(r[0], r[1], r[2], pm.j2)};
  R E1[3], E2[3], F1[3], F2[3], ni[3], nj[3], Ji, Jj;
#pragma unroll
  for (int e = 0; e < 3; e++) {
    const R a1 = (R)g.vertices[3 * vi[1] + e], b1 = (R)g.vertices[3 * vj[1] + e];
    E1[e] = a1 - (R)g.vertices[3 * vi[0] + e];
    E2[e] = (R)g.vertices[3 * vi[2] + e] - a1;
    F1[e] = b1 - (R)g.vertices[3 * vj[0] + e];
    F2[e] = (R)g.vertices[3 * vj[2] + e] - b1;
  }
  // unit normals of the triangles in input order
  auto normal = [](const R (&a)[3], const R (&b)[3], const Perm6& q, bool test, R (&n)[3]) {
    n[0] = a[1] * b[2] - a[2] * b[1];
    n[1] = a[2] * b[0] - a[0] * b[2];
    n[2] = a[0] * b[1] - a[1] * b[0];
    const R J = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    const int c0 = test ? q.i0 : q.j0, c1 = test ? q.i1 : q.j1;
    const R sgn = (c1 - c0 + 3) % 3 == 1 ? R(1) : R(-1);  // an odd permutation turns the edges' cross product round
#pragma unroll
    for (int e = 0; e < 3; e++) n[e] *= sgn / J;
    return J;
  };
  Ji = normal(E1, E2, pm, true, ni);
  Jj = normal(F1, F2, pm, false, nj);
  Along<R> Li, Gi_, Ui, Lj, Gj, Uj;
  Li.load(lam, vi);
  Gj.load(gvec, vj);
  Uj.load(uvec, vj);
  if (kMirror) {
    Lj.load(lam, vj);
    Gi_.load(gvec, vi);
    Ui.load(uvec, vi);
  }
  const R k = (R)kf, jw = Ji * Jj / R(16) * R(kInv4Pi);
  // sums: energy; grad_y; grad_y times the shape functions of corners 1 and 2
  // of the test and of the trial triangle; gradients of the trial and of the
  // test normal
  constexpr int kSums = kMirror ? 22 : 19;
  R t[kSums];
#pragma unroll
  for (int e = 0; e < kSums; e++) t[e] = 0;
  auto region = [&](R x1, R x2, R y1, R y2, R w) {
    R d[3];
#pragma unroll
    for (int e = 0; e < 3; e++)
      d[e] = NCOMMON == 2 ? (y1 - x1) * E1[e] + y2 * F2[e] - x2 * E2[e]  // F1 = E1, the shared edge
                          : y1 * F1[e] + y2 * F2[e] - x1 * E1[e] - x2 * E2[e];
    R u, Gr, Gi, hr, hi;
    const bool free = touch_kernel<R>(d[0] * d[0] + d[1] * d[1] + d[2] * d[2], k, u, Gr, Gi, hr, hi);
    const R u2 = u * u, er = (R(3) * hr - k * k * Gr) * u2, ei = (R(3) * hi - k * k * Gi) * u2;
    const R dj = d[0] * nj[0] + d[1] * nj[1] + d[2] * nj[2];
    R lr, li, gr, gi, ur, ui;
    Li.at(x1, x2, lr, li);
    Gj.at(y1, y2, gr, gi);
    Uj.at(y1, y2, ur, ui);
    R Yr = lr * gr + li * gi, Yn = li * gr - lr * gi;
    const R Z2r = lr * ur + li * ui, Z2n = li * ur - lr * ui;
    const R m2 = w * (Z2r * hr + Z2n * hi);
    R wd = dj * (Z2r * er + Z2n * ei), E = dj * m2;
    R gy[3];
    if (kMirror) {
      const R di = -(d[0] * ni[0] + d[1] * ni[1] + d[2] * ni[2]);
      R pr, pi, qr, qi, wr, wi;
      Lj.at(y1, y2, pr, pi);
      Gi_.at(x1, x2, qr, qi);
      Ui.at(x1, x2, wr, wi);
      Yr += pr * qr + pi * qi;
      Yn += pi * qr - pr * qi;
      const R Z3r = pr * wr + pi * wi, Z3n = pi * wr - pr * wi;
      const R m3 = w * (Z3r * hr + Z3n * hi);
      wd += di * (Z3r * er + Z3n * ei);
      E += di * m3;
#pragma unroll
      for (int e = 0; e < 3; e++) {
        gy[e] = m3 * ni[e] - m2 * nj[e];
        t[(kMirror ? 19 : 0) + e] += m3 * d[e];
      }
    } else {
#pragma unroll
      for (int e = 0; e < 3; e++) gy[e] = -m2 * nj[e];
    }
    t[0] -= w * (Yr * Gr + Yn * Gi) + E;
    const R c1 = free ? w * (Yr * hr + Yn * hi + wd) : R(0);
    const R lx1 = x1 - x2, ly1 = y1 - y2;
#pragma unroll
    for (int e = 0; e < 3; e++) {
      gy[e] += c1 * d[e];
      t[1 + e] += gy[e];
      t[4 + e] += lx1 * gy[e];
      t[7 + e] += x2 * gy[e];
      t[10 + e] += ly1 * gy[e];
      t[13 + e] += y2 * gy[e];
      t[16 + e] -= m2 * d[e];
    }
  };
#pragma unroll 1
  for (int pt = lane; pt < 256; pt += 32) {
    const int i0 = pt >> 6, i1 = (pt >> 4) & 3, i2 = (pt >> 2) & 3, i3 = pt & 3;
    const R xi = R(0.5) * (R(gl4_x(i0)) + R(1)), e1 = R(0.5) * (R(gl4_x(i1)) + R(1));
    const R e2 = R(0.5) * (R(gl4_x(i2)) + R(1)), e3 = R(0.5) * (R(gl4_x(i3)) + R(1));
    ss_regions<NCOMMON, R>(xi, e1, e2, e3, R(gl4_w(i0)) * R(gl4_w(i1)) * R(gl4_w(i2)) * R(gl4_w(i3)) * jw, region);
  }
  warp_totals<kSums>(t, total);
  if (lane < 2) {  // lane 0: the test triangle, lane 1: the trial triangle
    const bool test = lane == 0;
    const int v[3] = {test ? s[0] : r[0], test ? s[1] : r[1], test ? s[2] : r[2]};
    double p[3][3], N[3], out[3][3];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int e = 0; e < 3; e++) p[c][e] = (double)g.vertices[3 * v[c] + e];
#pragma unroll
    for (int e = 0; e < 3; e++)
      N[e] = test ? (kMirror ? (double)total[(kMirror ? 19 : 0) + e] : 0.0) : (double)total[16 + e];
    area_normal_grad<double>(p, (double)total[0] / (0.5 * (double)(test ? Ji : Jj)), N, true, out);
    adj_add(grad, v, out);
    const int q[3] = {test ? vi[0] : vj[0], test ? vi[1] : vj[1], test ? vi[2] : vj[2]};
    const int o = test ? 4 : 10;
    const double sgn = test ? -1.0 : 1.0;  // grad_x = -grad_y
    double add[3][3];
#pragma unroll
    for (int e = 0; e < 3; e++) {
      add[1][e] = sgn * (double)total[o + e];
      add[2][e] = sgn * (double)total[o + 3 + e];
      add[0][e] = sgn * (double)total[1 + e] - add[1][e] - add[2][e];
    }
    adj_add(grad, q, add);
  }
}

// All touching pairs: warps over the triangles, the edge pairs, the unordered
// vertex pairs.  Only adds to the gradient, so it may start while the regular
// pairs' kernel runs (programmatic launch).
__global__ void __launch_bounds__(kAdjThreads)
    grad_touch_kernel(const __grid_constant__ GeomView g, float k, const float2* __restrict__ lam,
                      const float2* __restrict__ gvec, const float2* __restrict__ uvec, double* __restrict__ grad) {
  __shared__ AdjTouchShared sm;
  const int warp = threadIdx.x >> 5, w = blockIdx.x * kAdjWarps + warp;
  if (w < g.nt) {
    grad_coincident(g, w, k, lam, gvec, uvec, grad, sm.c[warp]);
  } else if (w < g.nt + g.n_edge) {
    const int2 p = g.edge_pairs[w - g.nt];
    grad_touch<double, 2>(g, p.x, p.y, k, lam, gvec, uvec, grad, sm.c[warp]);
  } else if (w < g.nt + g.n_edge + g.n_vert / 2) {
    const int2 p = g.vert_pairs[w - g.nt - g.n_edge];
    grad_touch<float, 1>(g, p.x, p.y, k, lam, gvec, uvec, grad, sm.f[warp]);
  }
  wait_previous();
}

// Listener terms Re[-pbar^H dS g + pbar^H dD u]: thread per triangle, loop
// over the listeners of one part (blockIdx.y; x fixed): only the trial side,
// its area and its normal.
__global__ void grad_listener_kernel(GeomView g, float k, const float* __restrict__ pts, int np, int part,
                                     const float2* __restrict__ pbar, const float2* __restrict__ gvec,
                                     const float2* __restrict__ uvec, double* __restrict__ grad) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.nt) return;
  const TriRec& rj = g.rec_orig[j];
  float bvr[6], bvi[6], bkr[6], bki[6];
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const double2 gq = lerp3(gvec, rj.v[0], rj.v[1], rj.v[2], tri6_phi(q, 0), tri6_phi(q, 1), tri6_phi(q, 2));
    const double2 uq = lerp3(uvec, rj.v[0], rj.v[1], rj.v[2], tri6_phi(q, 0), tri6_phi(q, 1), tri6_phi(q, 2));
    bvr[q] = -(float)gq.x;
    bvi[q] = -(float)gq.y;
    bkr[q] = (float)uq.x;
    bki[q] = (float)uq.y;
  }
  const float n[3] = {rj.n[0], rj.n[1], rj.n[2]};
  float F = 0.f, N[3] = {0, 0, 0}, U[6][3];
#pragma unroll
  for (int q = 0; q < 6; q++) U[q][0] = U[q][1] = U[q][2] = 0.f;
  const int p0 = blockIdx.y * part, p1 = min(np - p0, part) + p0;
  for (int p = p0; p < p1; p++) {
    const float ar = pbar[p].x, ai = -pbar[p].y;  // conj(pbar)
    const float x0 = pts[3 * p], x1 = pts[3 * p + 1], x2 = pts[3 * p + 2];
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const float d[3] = {rj.qp[3 * q] - x0, rj.qp[3 * q + 1] - x1, rj.qp[3 * q + 2] - x2};
      float gy[3] = {0, 0, 0};
      const float W = rj.area * kInv4Pi * (float)tri6_w(q);
      point_grad(d, n, k, ar, ai, bvr[q], bvi[q], bkr[q], bki[q], W, F, gy, N);
#pragma unroll
      for (int e = 0; e < 3; e++) U[q][e] += gy[e];
    }
  }
  float vj[3][3];
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) vj[c][e] = g.vertices[3 * rj.v[c] + e];
  float out[3][3];
  area_normal_grad<float>(vj, F / rj.area, N, true, out);
#pragma unroll
  for (int c = 0; c < 3; c++)
#pragma unroll
    for (int e = 0; e < 3; e++) {
      float s = out[c][e];
#pragma unroll
      for (int q = 0; q < 6; q++) s += (float)tri6_phi(q, c) * U[q][e];
      atomicAdd(&grad[3 * rj.v[c] + e], (double)s);
    }
}

// Mass term -1/2 Re[lambda^H dM u]: M_ab = A (1 + delta_ab)/12 per triangle.
__global__ void grad_mass_kernel(GeomView g, float mass_coeff, const float2* __restrict__ lam,
                                 const float2* __restrict__ uvec, double* __restrict__ grad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nt) return;
  const TriRec& r = g.rec_orig[i];
  double e = 0.0;
  for (int a = 0; a < 3; a++)
    for (int b = 0; b < 3; b++) {
      const float2 la = lam[r.v[a]], ub = uvec[r.v[b]];
      const double m = (a == b ? 2.0 : 1.0) / 12.0;
      e += m * ((double)la.x * ub.x + (double)la.y * ub.y);  // Re(conj(l) u)
    }
  double v[3][3];
  for (int c = 0; c < 3; c++)
    for (int d = 0; d < 3; d++) v[c][d] = g.vertices[3 * r.v[c] + d];
  double out[3][3];
  const double zero[3] = {0, 0, 0};
  area_normal_grad<double>(v, (double)mass_coeff * e, zero, false, out);  // dE/dA = coeff * e
  for (int c = 0; c < 3; c++)
    for (int d = 0; d < 3; d++) atomicAdd(&grad[3 * r.v[c] + d], out[c][d]);
}

// Y = A^H X (A: n x n complex64 row-major), m columns, Y overwritten.
__global__ void cmatmul_h_kernel(const float2* __restrict__ A, int n, const float2* __restrict__ X, int m,
                                 float2* __restrict__ Y, int rows_per_block) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= n) return;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(n, r0 + rows_per_block);
  for (int s = 0; s < m; s++) {
    double ar = 0.0, ai = 0.0;
    for (int r = r0; r < r1; r++) {
      const float2 a = A[(size_t)r * n + col];
      const float2 x = X[(size_t)r * m + s];
      ar += (double)a.x * x.x + (double)a.y * x.y;  // conj(a) x
      ai += (double)a.x * x.y - (double)a.y * x.x;
    }
    atomicAdd(&Y[(size_t)col * m + s], make_float2((float)ar, (float)ai));
  }
}

// out = conj(A)^T, tiled through shared memory.
__global__ void conj_transpose_kernel(const float2* __restrict__ A, int n, float2* __restrict__ out) {
  __shared__ float2 tile[32][33];
  const int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int row = by + r, col = bx + threadIdx.x;
    if (row < n && col < n) tile[r][threadIdx.x] = A[(size_t)row * n + col];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int row = bx + r, col = by + threadIdx.x;  // out[row][col] = conj(A[col][row])
    if (row < n && col < n) {
      const float2 v = tile[threadIdx.x][r];
      out[(size_t)row * n + col] = make_float2(v.x, -v.y);
    }
  }
}

// S^H pbar and D^H pbar: `lanes` lanes (a power of two, 32 at most) per trial
// triangle, each over every lanes-th listener.  A listener's six points are
// summed onto the triangle's vertices in FP32, the listeners and lanes in FP64,
// so that a vertex takes one FP32 addition per triangle however many lanes share
// it.  (With a thread per point and a grid of listener parts, each added on its
// own, the velocity gradient of 144 triangles and 615 listeners was 8.0e-7 off
// 64 bits; it is 1.9e-7 so, and 2.6e-7 with one thread per point and no parts.
// 2000 listeners x 80 triangles 79 us, 128 x 5120 27 us; in parts 261 and 27 us.)
__global__ void __launch_bounds__(128)
    b2p_adjoint_kernel(GeomView g, const float* __restrict__ pts, int np, int lanes, float k,
                       const float2* __restrict__ pbar, float2* __restrict__ out_s, float2* __restrict__ out_d) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x, at = id / lanes;
  const TriRec& r = g.rec_orig[at < g.nt ? at : g.nt - 1];  // past the end: for the shuffles only
  float y[18];
#pragma unroll
  for (int e = 0; e < 18; e++) y[e] = r.qp[e];
  const float n0 = r.n[0], n1 = r.n[1], n2 = r.n[2];
  double sum[12];  // S^H and D^H pbar at the vertices, (re, im)
#pragma unroll
  for (int e = 0; e < 12; e++) sum[e] = 0.0;
  for (int p = (int)(id & (lanes - 1)); p < np; p += lanes) {
    const float x0 = pts[3 * p], x1 = pts[3 * p + 1], x2 = pts[3 * p + 2];
    const float2 pb = pbar[p];
    float t[12];
#pragma unroll
    for (int e = 0; e < 12; e++) t[e] = 0.f;
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const float dx = y[3 * q] - x0, dy = y[3 * q + 1] - x1, dz = y[3 * q + 2] - x2;
      float rr = sqrtf(dx * dx + dy * dy + dz * dz);
      rr = fmaxf(rr, kEps);
      float s, c;
      sincosf(k * rr, &s, &c);
      const float u = 1.f / rr;
      const float gr = c * u, gi = s * u;
      const float dn = dx * n0 + dy * n1 + dz * n2;
      const float f = -dn * u * u * u, kr = k * rr;
      const float dr = (c + kr * s) * f, di = (s - kr * c) * f;
      // conj(kernel) * pbar
      const float z[4] = {gr * pb.x + gi * pb.y, gr * pb.y - gi * pb.x, dr * pb.x + di * pb.y, dr * pb.y - di * pb.x};
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int e = 0; e < 4; e++) t[4 * b + e] = fmaf((float)(tri6_w(q) * tri6_phi(q, b)), z[e], t[4 * b + e]);
    }
#pragma unroll
    for (int e = 0; e < 12; e++) sum[e] += (double)t[e];
  }
  for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
    for (int e = 0; e < 12; e++) sum[e] += __shfl_xor_sync(0xffffffffu, sum[e], o);
  if ((id & (lanes - 1)) != 0 || at >= g.nt) return;
  const double w = (double)r.area * (double)kInv4Pi;
#pragma unroll
  for (int b = 0; b < 3; b++) {
    if (out_s) atomicAdd(&out_s[r.v[b]], make_float2((float)(w * sum[4 * b]), (float)(w * sum[4 * b + 1])));
    if (out_d) atomicAdd(&out_d[r.v[b]], make_float2((float)(w * sum[4 * b + 2]), (float)(w * sum[4 * b + 3])));
  }
}

}  // namespace

}  // namespace bemb

using namespace bemb;

namespace {
// Listeners per part for a kernel with one thread per (item, part): parts
// until every SM holds about 1024 threads (a thread per triangle alone leaves
// most of the chip idle: 128 listeners x 5120 triangles 30 us in parts, 173 in one), at least 8
// listeners in each (a part starts by interpolating its densities).
int adj_part(int np, long long items, int sms) {
  const long long parts = std::max(1LL, 1024LL * sms / std::max(1LL, items));
  return (int)std::max<long long>(std::max(8LL, (np + 65534LL) / 65535), (np + parts - 1) / parts);
}
}  // namespace

extern "C" int bem_cmatmul_adjoint(const void* A, int n, const void* X, int m, void* Y, bem_stream_t stream) {
  if (n <= 0 || m <= 0 || !A || !X || !Y) return BEM_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  BEM_CUDA_TRY(cudaMemsetAsync(Y, 0, sizeof(float2) * (size_t)n * m, s));
  const int rpb = 128;
  dim3 grid((n + 127) / 128, (n + rpb - 1) / rpb);
  (cmatmul_h_kernel<<<grid, 128, 0, s>>>((const float2*)A, n, (const float2*)X, m, (float2*)Y, rpb), count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

extern "C" int bem_conj_transpose(const void* A, int n, void* out, bem_stream_t stream) {
  if (n <= 0 || !A || !out || A == out) return BEM_ERR_INVALID_ARGUMENT;
  dim3 grid((n + 31) / 32, (n + 31) / 32);
  (conj_transpose_kernel<<<grid, dim3(32, 8), 0, (cudaStream_t)stream>>>((const float2*)A, n, (float2*)out),
   count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

extern "C" int bem_boundary2potential_adjoint(const void* geom, const float* points, int np, float k,
                                              const void* pbar, void* out_s, void* out_d, bem_stream_t stream) {
  GeomView g;
  int rc = geom_view(geom, &g, nullptr);
  if (rc) return rc;
  if (np <= 0 || !points || !pbar || (!out_s && !out_d)) return BEM_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  if (out_s) BEM_CUDA_TRY(cudaMemsetAsync(out_s, 0, sizeof(float2) * (size_t)g.nv, s));
  if (out_d) BEM_CUDA_TRY(cudaMemsetAsync(out_d, 0, sizeof(float2) * (size_t)g.nv, s));
  int dev = 0, sms = 148;
  BEM_CUDA_TRY(cudaGetDevice(&dev));
  BEM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // lanes until every SM holds about 1024 threads, at least 2 listeners in each
  int lanes = 1;
  while (lanes < 32 && (long long)g.nt * lanes < 1024LL * sms && np >= 4 * lanes) lanes *= 2;
  const long long threads = (long long)g.nt * lanes;
  (b2p_adjoint_kernel<<<(unsigned)((threads + 127) / 128), 128, 0, s>>>(
       g, points, np, lanes, k, (const float2*)pbar, (float2*)out_s, (float2*)out_d),
   count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

extern "C" int bem_vertex_gradient(const void* geom, float k, const void* lambda, const void* neumann,
                                   const void* dirichlet, const float* points, int np, const void* pbar, double* grad,
                                   bem_stream_t stream) {
  GeomView g;
  int rc = geom_view(geom, &g, nullptr);
  if (rc) return rc;
  if (!lambda || !neumann || !dirichlet || !grad || np < 0 || (np > 0 && (!points || !pbar)))
    return BEM_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  const float2* lam = (const float2*)lambda;
  const float2* gv = (const float2*)neumann;
  const float2* uv = (const float2*)dirichlet;
  BEM_CUDA_TRY(cudaMemsetAsync(grad, 0, sizeof(double) * 3 * (size_t)g.nv, s));
  // regular pairs: equal runs of steps, in rounds over the resident warps
  int dev = 0, sms = 148, occ = 0;
  BEM_CUDA_TRY(cudaGetDevice(&dev));
  BEM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int smem = (int)(kAdjWarps * sizeof(AdjWarp));
  static DeviceOnce once;
  if ((rc = once.shared_memory(grad_regular_kernel, smem))) return rc;
  BEM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, grad_regular_kernel, kAdjThreads, smem));
  const long long n_steps = strip_steps(g.nblocks), warps = (long long)sms * (occ > 0 ? occ : 1) * kAdjWarps;
  const long long chunk = std::max(2LL, strip_part(n_steps, warps, kStripRounds));
  const long long blocks = ((n_steps + chunk - 1) / chunk + kAdjWarps - 1) / kAdjWarps;
  (grad_regular_kernel<<<(unsigned)blocks, kAdjThreads, smem, s>>>(g, k, lam, gv, uv, grad, chunk, n_steps),
   count_launch());
  const long long touch = (long long)g.nt + g.n_edge + g.n_vert / 2;
  EarlyLaunch early((unsigned)((touch + kAdjWarps - 1) / kAdjWarps), kAdjThreads, 0, s);
  BEM_CUDA_TRY(cudaLaunchKernelEx(&early.cfg, grad_touch_kernel, g, k, lam, gv, uv, grad));
  count_launch();
  (grad_mass_kernel<<<(g.nt + 127) / 128, 128, 0, s>>>(g, -0.5f, lam, uv, grad), count_launch());
  const int part = adj_part(np, g.nt, sms);
  if (np > 0)
    (grad_listener_kernel<<<dim3((g.nt + 127) / 128, (np + part - 1) / part), 128, 0, s>>>(g, k, points, np, part, (const float2*)pbar, gv, uv, grad),
     count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}
