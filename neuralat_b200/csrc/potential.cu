// Boundary-to-listener evaluation and triangle -> vertex averaging.
//
// Reference: src/bem/cuda/bind.cu:156-176 (explicit P x N potential matrix,
// one block per listener, 3 scalar atomics per (listener, triangle)),
// integrand.h:237-255,396-406 (6-point rule, target normal 0, trial normal),
// src/bem/solver.py:128-147 (matrix times vector), bind.cu:23-48
// (triangle2vertex).
//
// B200 design: `boundary2potential` never materialises the P x N matrices.  A
// thread owns a listener and walks along the sorted triangles, whose order
// keeps shared vertices in their slots (BlockRec): S and D share one distance
// and one sincos per quadrature point, and the potentials of a vertex are
// summed in registers until it leaves the path.  Only then they meet the
// right-hand sides, once per path vertex (1.15 per triangle) instead of once
// per quadrature point (6 per triangle).

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "bem_common.cuh"

namespace bemb {

int geom_view(const void* geom, GeomView* v, GeomHeader* out_hdr);

namespace {

// Explicit potential matrix: thread = (listener p, triangle j).
template <int LAYER>
__global__ void potential_matrix_kernel(GeomView g, const float* __restrict__ pts, int np, float k,
                                        float2* __restrict__ out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int p = blockIdx.y;
  if (j >= g.nt || p >= np) return;
  const TriRec& r = g.rec_orig[j];
  const float px = pts[3 * p], py = pts[3 * p + 1], pz = pts[3 * p + 2];
  float2 acc[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const float dx = r.qp[3 * q] - px, dy = r.qp[3 * q + 1] - py, dz = r.qp[3 * q + 2] - pz;
    float rr = sqrtf(dx * dx + dy * dy + dz * dz);
    rr = fmaxf(rr, kEps);
    float s, c;
    sincosf(k * rr, &s, &c);
    float gr, gi;
    if (LAYER == BEM_SINGLE_LAYER) {
      gr = c / rr;
      gi = s / rr;
    } else {
      const float dn = dx * r.n[0] + dy * r.n[1] + dz * r.n[2];  // (y - x) . n_y
      const float f = -dn / (rr * rr * rr);
      const float kr = k * rr;
      gr = (c + kr * s) * f;
      gi = (s - kr * c) * f;
    }
#pragma unroll
    for (int b = 0; b < 3; b++) {
      const float w = (float)(tri6_w(q) * tri6_phi(q, b));
      acc[b].x = fmaf(w, gr, acc[b].x);
      acc[b].y = fmaf(w, gi, acc[b].y);
    }
  }
  const float sc = r.area * kInv4Pi;
#pragma unroll
  for (int b = 0; b < 3; b++)
    atomicAdd(&out[(size_t)p * g.nv + r.v[b]], make_float2(acc[b].x * sc, acc[b].y * sc));
}

// Sums of one listener's potentials over the path, per trial slot: S phi_b and
// D phi_b, (re, im), without the sign of the double layer.
struct ListenSums {
  float2 s[3], d[3];
};

// Adds one triangle.  The rule's symmetry as in the assembly: with g_b, h_b
// the values at the two points of vertex b, the sum for b is
// own_1 (g_b + rho h_b + tau sum_c (g_c + sigma h_c)).
__device__ __forceinline__ void listen_triangle(const TriRec& r, float px, float py, float pz, float k,
                                                ListenSums& acc) {
  constexpr float kRho = (float)(tri6_w_own(3) / tri6_w_own(0)), kSigma = (float)(tri6_w_common(3) / tri6_w_common(0)),
                  kTau = (float)(tri6_w_common(0) / tri6_w_own(0));
  const float4* r4 = (const float4*)&r;
  const float4 q0 = r4[0], q1 = r4[1], q2 = r4[2], q3 = r4[3], q4 = r4[4], q5 = r4[5];
  const float2 yx[3] = {{q0.x, q2.y}, {q0.w, q3.x}, {q1.z, q3.w}};
  const float2 yy[3] = {{q0.y, q2.z}, {q1.x, q3.y}, {q1.w, q4.x}};
  const float2 yz[3] = {{q0.z, q2.w}, {q1.y, q3.z}, {q2.x, q4.y}};
  const float dn = q4.z * (q5.y - px) + q4.w * (q5.z - py) + q5.x * (q5.w - pz);  // n . (y - x) on the plane
  const float2 k2 = f2(k), nk2 = f2(-k);
  float2 tS[3], tD[3], sSr, sSi, sDr, sDi;
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const float2 dx = f2_sub(yx[b], f2(px)), dy = f2_sub(yy[b], f2(py)), dz = f2_sub(yz[b], f2(pz));
    float2 r2 = f2_fma(dx, dx, f2_fma(dy, dy, f2_mul(dz, dz)));
    r2.x = fmaxf(r2.x, kEps * kEps);  // r >= 1e-3, to a rounding
    r2.y = fmaxf(r2.y, kEps * kEps);
    const float2 ri = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
    const float2 kr = f2_mul(k2, f2_mul(r2, ri)), ri2 = f2_mul(ri, ri);
    // hardware sin/cos: the FP32 phase k r carries a relative error of ~2^-24,
    // which the hardware evaluation keeps (a few 1e-6 rad at k r ~ 100)
    float2 sn, cs;
    __sincosf(kr.x, &sn.x, &cs.x);
    __sincosf(kr.y, &sn.y, &cs.y);
    const float2 gr = f2_mul(cs, ri), gi = f2_mul(sn, ri);
    const float2 hr = f2_mul(f2_fma(k2, sn, gr), ri2), hi = f2_mul(f2_fma(nk2, cs, gi), ri2);
    tS[b] = make_float2(fmaf(kRho, gr.y, gr.x), fmaf(kRho, gi.y, gi.x));
    tD[b] = make_float2(fmaf(kRho, hr.y, hr.x), fmaf(kRho, hi.y, hi.x));
    sSr = b ? f2_add(sSr, gr) : gr;
    sSi = b ? f2_add(sSi, gi) : gi;
    sDr = b ? f2_add(sDr, hr) : hr;
    sDi = b ? f2_add(sDi, hi) : hi;
  }
  const float2 sS = make_float2(fmaf(kSigma, sSr.y, sSr.x), fmaf(kSigma, sSi.y, sSi.x));
  const float2 sD = make_float2(fmaf(kSigma, sDr.y, sDr.x), fmaf(kSigma, sDi.y, sDi.x));
  const float ws = r.area * (float)(tri6_w_own(0) / (4.0 * kPi)), wd = ws * dn;
#pragma unroll
  for (int b = 0; b < 3; b++) {
    acc.s[b] = f2_fma(f2(ws), f2_fma(f2(kTau), sS, tS[b]), acc.s[b]);
    acc.d[b] = f2_fma(f2(wd), f2_fma(f2(kTau), sD, tD[b]), acc.d[b]);
  }
}

constexpr int kLsThreads = 128;
constexpr int kLsWarps = kLsThreads / 32;
constexpr int kLsChunk = 16;  // triangles staged per warp

// out[p, s] += -S neumann + D dirichlet over the triangles of one run
// (blockIdx.y) for 32 listeners, up to M <= 4 right-hand sides: the products
// with the vertex densities stay in the listener's own registers.  Each warp
// walks a quarter of the run; their sums meet in shared memory and those of a
// cluster's runs in its first CTA (FP64, rounded once), so that few FP32 terms are added to an output
// one after the other.
//
// Bound by the FP32 and sincos units (about 125 instructions for the 6 points
// of a triangle).  Measured on B200: 1000 listeners x 5110 triangles x 1
// right-hand side 46 us, against 165 us with the densities interpolated onto
// the quadrature points by a pass of their own and 8 products per point and
// right-hand side.
template <int M>
__global__ void __launch_bounds__(kLsThreads)
    listen_few_kernel(GeomView g, const float* __restrict__ pts, int np, float k, const float2* __restrict__ neu,
                      const float2* __restrict__ dir, int nrhs, float2* __restrict__ out, int run) {
  __shared__ TriRec rec_s[kLsWarps][kLsChunk];
  __shared__ float4 dens_s[kLsWarps][kLsChunk][3][M];  // (neumann, dirichlet) at the triangle's vertices
  __shared__ float2 sum_s[kLsWarps][M][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
  TriRec* rec = rec_s[warp];
  float4(*dens)[3][M] = dens_s[warp];
  const float* x = pts + 3 * (size_t)min(p, np - 1);
  const float px = x[0], py = x[1], pz = x[2];
  const int part = (run + kLsWarps - 1) / kLsWarps, r0 = blockIdx.y * run;
  const int t0 = min(r0 + warp * part, g.nt), t1 = min(min(t0 + part, r0 + run), g.nt);
  ListenSums acc;
#pragma unroll
  for (int b = 0; b < 3; b++) acc.s[b] = acc.d[b] = make_float2(0.f, 0.f);
  float2 sum[M];
#pragma unroll
  for (int s = 0; s < M; s++) sum[s] = make_float2(0.f, 0.f);
  for (int c0 = t0; c0 < t1; c0 += kLsChunk) {
    const int n = min(kLsChunk, t1 - c0);
    __syncwarp();
    for (int e = lane; e < 8 * n; e += 32) ((float4*)rec)[e] = ((const float4*)&g.rec[c0])[e];
    for (int e = lane; e < 3 * M * n; e += 32) {
      const int t = e / (3 * M), b = (e / M) % 3, s = e % M;
      const size_t at = (size_t)g.rec[c0 + t].v[b] * nrhs + s;
      const float2 zero = make_float2(0.f, 0.f);
      const float2 a = neu && s < nrhs ? neu[at] : zero, u = dir && s < nrhs ? dir[at] : zero;
      dens[t][b][s] = make_float4(a.x, a.y, u.x, u.y);
    }
    __syncwarp();
#pragma unroll 1
    for (int t = 0; t < n; t++) {
      listen_triangle(rec[t], px, py, pz, k, acc);
      const int leave = c0 + t + 1 == t1 ? 7 : rec[t].leave;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        if (!((leave >> b) & 1)) continue;
        const float2 sv = acc.s[b], dv = acc.d[b];
#pragma unroll
        for (int s = 0; s < M; s++) {
          const float4 w = dens[t][b][s];
          sum[s].x -= sv.x * w.x - sv.y * w.y + dv.x * w.z - dv.y * w.w;
          sum[s].y -= sv.x * w.y + sv.y * w.x + dv.x * w.w + dv.y * w.z;
        }
        acc.s[b] = acc.d[b] = make_float2(0.f, 0.f);
      }
    }
  }
#pragma unroll
  for (int s = 0; s < M; s++) sum_s[warp][s][lane] = sum[s];
  __syncthreads();
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  if (cluster.num_blocks() == 1) {
    if (warp == 0 && p < np) {
#pragma unroll
      for (int s = 0; s < M; s++) {
        float2 t = sum_s[0][s][lane];
#pragma unroll
        for (int w = 1; w < kLsWarps; w++) t = f2_add(t, sum_s[w][s][lane]);
        if (s < nrhs) atomicAdd(&out[(size_t)p * nrhs + s], t);
      }
    }
    return;
  }
  for (int s = warp; s < M; s += kLsWarps) {  // right-hand side s of listener `lane`
    float2 t = sum_s[0][s][lane];
#pragma unroll
    for (int w = 1; w < kLsWarps; w++) t = f2_add(t, sum_s[w][s][lane]);
    sum_s[0][s][lane] = t;
  }
  cluster.sync();  // every CTA's sums are complete
  if (cluster.block_rank() == 0 && p < np)
    for (int s = warp; s < M && s < nrhs; s += kLsWarps) {
      double re = 0.0, im = 0.0;
      for (unsigned r = 0; r < cluster.num_blocks(); r++) {
        const float2 t = *cluster.map_shared_rank(&sum_s[0][s][lane], r);
        re += (double)t.x;
        im += (double)t.y;
      }
      atomicAdd(&out[(size_t)p * nrhs + s], make_float2((float)re, (float)im));
    }
  cluster.sync();  // the sums have been read
}

// The same for 8 J right-hand sides at a time (from rhs0 on): a thread writes
// its listener's path vertices as rows of a shared-memory tile; every
// kLsRows rows the CTA multiplies the tile (128 listeners x kLsRows vertices,
// S and D) with the densities of those vertices, a thread holding 8 listeners
// x J right-hand sides.  The densities of a row's vertex are copied
// asynchronously as soon as the vertex is known and arrive while the CTA walks
// on.  The tile stores Im also negated, as the packed arithmetic takes it.
//
// A product is four FMAs into one FP32 sum per row; after kLsChain rows or more
// the sums move on to second ones in shared memory (16 bytes per two outputs
// and thread, 4 J of them).  In one chain over the whole run, neighbouring
// vertices' like terms cost up to 2.9 times the error (33 right-hand sides, 4000
// listeners, 9800 triangles at 500 Hz: 8.0e-7 off 64 bits, 2.7e-7 so; one
// quadrature point after the other, in eight warps: 2.8e-7).  10 rows instead
// of 16 leave room for the second sums beside two CTAs per SM.
//
// Bound by the FP32 unit: per path vertex 16 operations per right-hand side
// and listener, besides the 125 instructions per triangle.  Measured on B200:
// 4096 listeners x 20 480 triangles x 64 right-hand sides 2.58 ms in one pass
// (FP32 pipe 68 % of its cycles; 2.47 ms in one chain per run, 2.81 ms moving on
// after 8 rows, 3.22 ms with 16 rows and one CTA per SM), against 21.1 ms with 8
// products per quadrature point and right-hand side in four passes.
constexpr int kLsRows = 10;
constexpr int kLsChain = 16;

template <int J>
struct ListenSmem {
  float w[kLsRows][6][kLsThreads];  // Re S, Im S, -Im S, Re D, Im D, -Im D
  float2 dens[kLsRows][2][8 * J];   // neumann and dirichlet
  TriRec rec[kBlock];
  float4 sum[4 * J][kLsThreads];    // (re, im) of a thread's listener pair l and right-hand side j at l J + j
};

// 8-byte asynchronous copy to shared memory; zeros if !in.
__device__ __forceinline__ void listen_copy(float2* dst, const float2* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}

template <int J>
__global__ void __launch_bounds__(kLsThreads, J == 8 ? 2 : 3)
    listen_many_kernel(GeomView g, const float* __restrict__ pts, int np, float k, const float2* __restrict__ neu,
                       const float2* __restrict__ dir, int nrhs, int rhs0, float2* __restrict__ out, int run) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ListenSmem<J>& sm = *reinterpret_cast<ListenSmem<J>*>(smem_raw);
  const int tid = threadIdx.x;
  const int cg = tid & 7, lg = tid >> 3;  // right-hand sides cg + 8 j, listeners 4 lg + 64 h + 0..3
  const float* x = pts + 3 * (size_t)min((int)blockIdx.x * kLsThreads + tid, np - 1);
  const float px = x[0], py = x[1], pz = x[2];
  const int t0 = blockIdx.y * run, t1 = min(t0 + run, g.nt);
  float2 ar[4][J], ai[4][J];  // listener pairs x right-hand sides
#pragma unroll
  for (int l = 0; l < 4; l++)
#pragma unroll
    for (int j = 0; j < J; j++) ar[l][j] = ai[l][j] = make_float2(0.f, 0.f);
  ListenSums acc;
#pragma unroll
  for (int b = 0; b < 3; b++) acc.s[b] = acc.d[b] = make_float2(0.f, 0.f);
  // the products so far move on to the thread's own sums
  bool first = true;
  auto fold = [&]() {
#pragma unroll
    for (int l = 0; l < 4; l++)
#pragma unroll
      for (int j = 0; j < J; j++) {
        float4& t = sm.sum[l * J + j][tid];
        float4 v = make_float4(ar[l][j].x, ai[l][j].x, ar[l][j].y, ai[l][j].y);
        if (!first) {
          const float4 old = t;
          v.x += old.x;
          v.y += old.y;
          v.z += old.z;
          v.w += old.w;
        }
        t = v;
        ar[l][j] = ai[l][j] = make_float2(0.f, 0.f);
      }
    first = false;
  };
  int rows = 0, chain = 0;
  for (int c0 = t0; c0 < t1; c0 += kBlock) {
    const int n = min(kBlock, t1 - c0);
    __syncthreads();  // everyone is done with the previous records
    for (int e = tid; e < 8 * n; e += kLsThreads) ((float4*)sm.rec)[e] = ((const float4*)&g.rec[c0])[e];
    __syncthreads();
    for (int t = 0; t < n;) {
      // ---- walk until the tile is full or the records end ----
#pragma unroll 1
      for (; t < n && rows + 3 <= kLsRows; t++) {
        const TriRec& r = sm.rec[t];
        listen_triangle(r, px, py, pz, k, acc);
        const int leave = c0 + t + 1 == t1 ? 7 : r.leave;
#pragma unroll
        for (int b = 0; b < 3; b++) {
          if (!((leave >> b) & 1)) continue;
          const float2 sv = acc.s[b], dv = acc.d[b];
          sm.w[rows][0][tid] = sv.x;
          sm.w[rows][1][tid] = sv.y;
          sm.w[rows][2][tid] = -sv.y;
          sm.w[rows][3][tid] = dv.x;
          sm.w[rows][4][tid] = dv.y;
          sm.w[rows][5][tid] = -dv.y;
          // 16 J densities: thread tid copies column tid of (neumann, dirichlet)
          for (int e = tid; e < 16 * J; e += kLsThreads) {
            const int layer = e / (8 * J), c = e - layer * 8 * J;
            const float2* src = layer ? dir : neu;
            const bool in = src && rhs0 + c < nrhs;
            listen_copy(&sm.dens[rows][layer][c], in ? src + (size_t)r.v[b] * nrhs + rhs0 + c : (const float2*)g.rec, in);
          }
          rows++;
          acc.s[b] = acc.d[b] = make_float2(0.f, 0.f);
        }
      }
      const bool last = t == n && c0 + n == t1;
      if (!last && rows + 3 <= kLsRows) continue;  // more records first
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      // ---- the product ----
#pragma unroll 1
      for (int row = 0; row < rows; row++) {
#pragma unroll
        for (int layer = 0; layer < 2; layer++) {
          float2 re[4], im[4], ni[4];
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const float4 a = *(const float4*)&sm.w[row][3 * layer][4 * lg + 64 * h];
            const float4 b = *(const float4*)&sm.w[row][3 * layer + 1][4 * lg + 64 * h];
            const float4 c = *(const float4*)&sm.w[row][3 * layer + 2][4 * lg + 64 * h];
            re[2 * h] = make_float2(a.x, a.y);
            re[2 * h + 1] = make_float2(a.z, a.w);
            im[2 * h] = make_float2(b.x, b.y);
            im[2 * h + 1] = make_float2(b.z, b.w);
            ni[2 * h] = make_float2(c.x, c.y);
            ni[2 * h + 1] = make_float2(c.z, c.w);
          }
#pragma unroll
          for (int j = 0; j < J; j++) {
            const float2 d = sm.dens[row][layer][cg + 8 * j], dr = f2(d.x), di = f2(d.y);
#pragma unroll
            for (int l = 0; l < 4; l++) {
              ar[l][j] = f2_fma(ni[l], di, f2_fma(re[l], dr, ar[l][j]));
              ai[l][j] = f2_fma(im[l], dr, f2_fma(re[l], di, ai[l][j]));
            }
          }
        }
      }
      chain += rows;
      rows = 0;
      if (chain >= kLsChain) {
        fold();
        chain = 0;
      }
      __syncthreads();  // the tile may be overwritten
    }
  }
  const int p = blockIdx.x * kLsThreads + 4 * lg;
  auto add_out = [&](int l, int j, const float4& t) {
    const int at = p + 64 * (l >> 1) + 2 * (l & 1), s = rhs0 + cg + 8 * j;
    if (s >= nrhs) return;
    if (at < np) atomicAdd(&out[(size_t)at * nrhs + s], make_float2(-t.x, -t.y));
    if (at + 1 < np) atomicAdd(&out[(size_t)(at + 1) * nrhs + s], make_float2(-t.z, -t.w));
  };
  fold();
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int ctas = (int)cluster.num_blocks();
  if (ctas == 1) {
#pragma unroll
    for (int l = 0; l < 4; l++)
#pragma unroll
      for (int j = 0; j < J; j++) add_out(l, j, sm.sum[l * J + j][tid]);
    return;
  }
  // the cluster's sums, a part of them per CTA
  cluster.sync();  // every CTA's sums are complete
  for (int q = (int)cluster.block_rank(); q < 4 * J; q += ctas) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int r = 0; r < ctas; r++) {
      const float4 v = *cluster.map_shared_rank(&sm.sum[q][tid], r);
      t[0] += (double)v.x;
      t[1] += (double)v.y;
      t[2] += (double)v.z;
      t[3] += (double)v.w;
    }
    add_out(q / J, q % J, make_float4((float)t[0], (float)t[1], (float)t[2], (float)t[3]));
  }
  cluster.sync();  // the sums have been read
}

__global__ void t2v_scatter_kernel(GeomView g, const float2* __restrict__ tv, float2* __restrict__ out,
                                   int* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.nt) return;
  const float2 v = tv[i];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int vid = g.triangles[3 * i + a];
    atomicAdd(&out[vid], v);
    atomicAdd(&cnt[vid], 1);
  }
}

__global__ void t2v_divide_kernel(int nv, float2* __restrict__ out, const int* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nv) return;
  // an isolated vertex gives 0/0 = NaN, as in the reference (bind.cu:46)
  const float c = (float)cnt[i];
  out[i] = make_float2(out[i].x / c, out[i].y / c);
}

}  // namespace

}  // namespace bemb

using namespace bemb;

extern "C" int bem_potential_matrix(const void* geom, int layer, const float* points, int np, float k, void* out,
                                    bem_stream_t stream) {
  GeomView g;
  int rc = geom_view(geom, &g, nullptr);
  if (rc) return rc;
  if (np < 0 || (np > 0 && (!points || !out))) return BEM_ERR_INVALID_ARGUMENT;
  if (layer != BEM_SINGLE_LAYER && layer != BEM_DOUBLE_LAYER) return BEM_ERR_UNSUPPORTED;
  if (np == 0) return BEM_OK;
  cudaStream_t s = (cudaStream_t)stream;
  BEM_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float2) * (size_t)np * g.nv, s));
  dim3 grid((g.nt + 127) / 128, np);
  if (layer == BEM_SINGLE_LAYER)
    (potential_matrix_kernel<BEM_SINGLE_LAYER><<<grid, 128, 0, s>>>(g, points, np, k, (float2*)out), count_launch());
  else
    (potential_matrix_kernel<BEM_DOUBLE_LAYER><<<grid, 128, 0, s>>>(g, points, np, k, (float2*)out), count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

extern "C" size_t bem_boundary2potential_scratch_bytes(int nt, int nrhs) {
  if (nt <= 0 || nrhs <= 0) return 0;
  return 2 * sizeof(float2) * (size_t)nt * 6 * (size_t)nrhs;
}

namespace bemb {
namespace {
// Runs of triangles: so many that the grid is a little below a whole number of
// waves of `slots` CTAs (as few waves as leave at most a tenth of the last one
// empty), of at least `least` triangles (each run loads its densities and adds
// its sums) and of at most 400, so that a listener's sums stay short (above,
// nothing is gained: 4096 listeners x 64 on 20 480 triangles 2.6 ms, with runs
// of 800 2.68 ms).
//
// An output takes one FP32 addition per run.  Where these are more than 64 (a
// fortieth of the triangles on small meshes, 8 at the least: as many as the
// chunks of 256 points that the point-by-point kernel added one by one), the
// runs of a cluster (up to 8 CTAs) are added up first, and there are
// no more than 512 runs while that leaves at most 400 triangles in each: 20
// listeners, one right-hand side, 20 480 triangles at 200 Hz 6.4e-7 -> 2.2e-7 off
// 64 bits, in the same time; 100 listeners x 5 on 1280 triangles 2.3e-7 -> 1.9e-7.
// Where they are fewer, a cluster gains nothing and costs 2 us of a 46 us call.
struct ListenRuns {
  int run, parts, cluster;
};

ListenRuns listen_runs(int groups, int nt, long long slots, int least) {
  long long splits = 1;
  for (int waves = 1; waves <= 64; waves++) {
    splits = std::max<long long>(1, waves * slots / groups);
    if (10 * splits * groups >= 9 * waves * slots && nt <= 400 * splits) break;
  }
  splits = std::min<long long>(splits, std::min(std::max(512, nt / 400), 65528));
  ListenRuns r;
  r.run = (int)std::max<long long>(least, (nt + splits - 1) / splits);
  r.parts = (nt + r.run - 1) / r.run;
  r.cluster = 1;
  const int limit = std::min(64, std::max(8, nt / 40));
  while (r.cluster < 8 && r.parts > limit * r.cluster) r.cluster *= 2;
  return r;
}

// Launch of a listener kernel with its runs as clusters along y; per_sm: CTAs
// that an SM holds; clusters: how many clusters of 2, 4 and 8 the GPU holds (0:
// not known yet).
template <typename Kernel, typename... Args>
int listen_launch(Kernel kernel, int groups, int nt, int sms, int per_sm, int least, size_t smem,
                  cudaStream_t s, std::atomic<int>* clusters, Args... args) {
  ListenRuns r = listen_runs(groups, nt, (long long)per_sm * sms, least);
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kLsThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = (unsigned)r.cluster;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = r.cluster > 1 ? 1 : 0;
  if (r.cluster > 1) {  // fewer CTAs fit as clusters
    std::atomic<int>& known = clusters[r.cluster == 2 ? 0 : (r.cluster == 4 ? 1 : 2)];
    int n = known.load(std::memory_order_relaxed);
    if (n == 0) {
      cfg.gridDim = dim3(1, (unsigned)r.cluster, 1);
      BEM_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
      if (n < 1) n = -1;  // none of this size
      known.store(n, std::memory_order_relaxed);
    }
    const int c = n > 0 ? r.cluster : 1;
    if (n > 0) r = listen_runs(groups, nt, (long long)n * c, least);
    r.cluster = c;
    r.parts = (r.parts + c - 1) / c * c;  // the last runs may be empty
    at[0].val.clusterDim.y = (unsigned)c;
    cfg.numAttrs = c > 1 ? 1 : 0;
  }
  cfg.gridDim = dim3((unsigned)groups, (unsigned)r.parts, 1);
  BEM_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args..., r.run));
  count_launch();
  return BEM_OK;
}

template <int M>
int listen_few(const GeomView& g, const float* pts, int np, float k, const float2* neu, const float2* dir, int nrhs,
               float2* out, int sms, cudaStream_t s) {
  static std::atomic<int> clusters[3];
  return listen_launch(listen_few_kernel<M>, (np + 31) / 32, g.nt, sms, 8, 16, 0, s, clusters, g, pts, np, k, neu, dir,
                       nrhs, out);
}

template <int J>
int listen_many(const GeomView& g, const float* pts, int np, float k, const float2* neu, const float2* dir, int nrhs,
                int rhs0, float2* out, int sms, cudaStream_t s) {
  const int smem = (int)sizeof(ListenSmem<J>);
  static std::atomic<int> clusters[3];
  static DeviceOnce once;
  if (const int rc = once.shared_memory(listen_many_kernel<J>, smem)) return rc;
  return listen_launch(listen_many_kernel<J>, (np + kLsThreads - 1) / kLsThreads, g.nt, sms, J == 8 ? 2 : 3, 12,
                       (size_t)smem, s, clusters, g, pts, np, k, neu, dir, nrhs, rhs0, out);
}
}  // namespace

// The work of bem_boundary2potential and bem_boundary2potential_noalloc.  Up
// to 4 right-hand sides multiply in the listener's registers; more go through
// the tiled product in passes of up to 64 (each pass evaluates the potentials
// again).
int b2p_enqueue(const GeomView& g, const float* points, int np, float k, const void* neumann, const void* dirichlet,
                int nrhs, void* out, cudaStream_t s) {
  const float2 *neu = (const float2*)neumann, *dir = (const float2*)dirichlet;
  float2* o = (float2*)out;
  BEM_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float2) * (size_t)np * nrhs, s));
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (nrhs <= 4) {
    const int rc = nrhs == 1   ? listen_few<1>(g, points, np, k, neu, dir, nrhs, o, sms, s)
                   : nrhs == 2 ? listen_few<2>(g, points, np, k, neu, dir, nrhs, o, sms, s)
                               : listen_few<4>(g, points, np, k, neu, dir, nrhs, o, sms, s);
    if (rc) return rc;
  } else {
    for (int r0 = 0; r0 < nrhs; r0 += 64) {
      const int left = nrhs - r0;
      const int rc = left > 32   ? listen_many<8>(g, points, np, k, neu, dir, nrhs, r0, o, sms, s)
                     : left > 16 ? listen_many<4>(g, points, np, k, neu, dir, nrhs, r0, o, sms, s)
                     : left > 8  ? listen_many<2>(g, points, np, k, neu, dir, nrhs, r0, o, sms, s)
                                 : listen_many<1>(g, points, np, k, neu, dir, nrhs, r0, o, sms, s);
      if (rc) return rc;
    }
  }
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}
}  // namespace bemb

extern "C" int bem_boundary2potential(const void* geom, const float* points, int np, float k, const void* neumann,
                                      const void* dirichlet, int nrhs, void* out, void* scratch, size_t scratch_bytes,
                                      bem_stream_t stream) {
  GeomView g;
  int rc = geom_view(geom, &g, nullptr);
  if (rc) return rc;
  if (np < 0 || nrhs <= 0 || (np > 0 && (!points || !out))) return BEM_ERR_INVALID_ARGUMENT;
  if (np == 0) return BEM_OK;
  // part of the contract, although the kernels sum in registers
  if (!scratch || scratch_bytes < bem_boundary2potential_scratch_bytes(g.nt, nrhs)) return BEM_ERR_WORKSPACE;
  return b2p_enqueue(g, points, np, k, neumann, dirichlet, nrhs, out, (cudaStream_t)stream);
}

extern "C" int bem_triangle2vertex(const void* geom, const void* tri_values, void* out, int* counts,
                                   bem_stream_t stream) {
  GeomView g;
  int rc = geom_view(geom, &g, nullptr);
  if (rc) return rc;
  if (!tri_values || !out || !counts) return BEM_ERR_INVALID_ARGUMENT;
  cudaStream_t s = (cudaStream_t)stream;
  BEM_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float2) * (size_t)g.nv, s));
  BEM_CUDA_TRY(cudaMemsetAsync(counts, 0, sizeof(int) * (size_t)g.nv, s));
  (t2v_scatter_kernel<<<(g.nt + 255) / 256, 256, 0, s>>>(g, (const float2*)tri_values, (float2*)out, counts), count_launch());
  (t2v_divide_kernel<<<(g.nv + 255) / 256, 256, 0, s>>>(g.nv, (float2*)out, counts), count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  return BEM_OK;
}

// ---------------------------------------------------------------------------
// Listener evaluation for callers that cannot allocate device memory.
//
// Some hosts of this library never call cudaMalloc while they run: real-time
// audio or rendering loops that synthesise sound from listener pressures
// must not block on the allocator (an allocation may synchronise the device
// and miss the callback deadline), and plug-ins embedded through a plain C
// FFI often have no device allocator of their own.  This entry point is the
// same computation as bem_boundary2potential without a scratch argument (the
// kernels keep their sums in registers and shared memory).
//
// Contract:
//  * requests with 6 * nt * nrhs > 2^20 are rejected with BEM_ERR_WORKSPACE
//    before any work is enqueued;
//  * calls may overlap (different streams, different host threads);
//  * no cudaMalloc, cudaFree or allocating library routine is called.
// ---------------------------------------------------------------------------
namespace bemb {
namespace {
constexpr long long kNoAllocQuadRhs = 1LL << 20;
}  // namespace
}  // namespace bemb

extern "C" long long bem_boundary2potential_noalloc_max(void) { return bemb::kNoAllocQuadRhs; }

extern "C" int bem_boundary2potential_noalloc(const void* geom, const float* points, int np, float k,
                                              const void* neumann, const void* dirichlet, int nrhs, void* out,
                                              bem_stream_t stream) {
  GeomView g;
  int rc = geom_view(geom, &g, nullptr);
  if (rc) return rc;
  if (np < 0 || nrhs <= 0 || (np > 0 && (!points || !out))) return BEM_ERR_INVALID_ARGUMENT;
  if ((long long)6 * g.nt * nrhs > kNoAllocQuadRhs) return BEM_ERR_WORKSPACE;
  if (np == 0) return BEM_OK;
  return b2p_enqueue(g, points, np, k, neumann, dirichlet, nrhs, out, (cudaStream_t)stream);
}
