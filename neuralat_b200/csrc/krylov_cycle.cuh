// GMRES with FP64 refinement for one right-hand side as ONE cooperative launch
// (included by linalg.cu after GmPtrs).
//
// A step per launch pair (matvec, Arnoldi kernel) leaves most of the chip idle
// for one right-hand side: the Arnoldi cluster is 16 CTAs, the matvec waits for
// it, launches and graph replays lie between, and about 25 small launches and
// copies start and end a solve.  Here a CTA owns rows of A and the same unknowns
// of every vector for the whole solve, and its slice of the basis never leaves
// shared memory.  Per step:
//   x = v_k (all of it, from L2);  w = A x on the CTA's rows: a warp sweeps 1, 2
//     or 4 rows at once, FP32 products, the lanes' sums added in FP64;
//   <v_j, w> and |w|^2 over the slice in FP64, added over the CTAs by FP64
//     atomics (8 copies, so that no address takes more than 19 additions);
//   == grid barrier ==
//   w' = w - sum_j v_j <v_j, w> / |v_j|^2;  v_{k+1} = fl32(c w'), |v_{k+1}|^2;
//   == grid barrier ==
// The basis vectors are orthogonal, not normalised: c is a power of two near
// 1 / |w'| (known before the second barrier from |w|^2 and the projections), so
// v_{k+1} is one rounding from w' and its norm, taken of the rounded vector, is
// exact to FP64.  The Hessenberg matrix of the normalised vectors follows by
// scaling.  A warp of CTA 0 of its own applies the Givens rotations of step k
// while step k + 1 multiplies, so every CTA learns one step late that the cycle
// is done.  Then CTA 0 solves the triangular system and every CTA adds V y to
// its unknowns.  Restarts, the FP64 residuals and the stopping tests follow the
// host loop of the other paths; every CTA takes the same decisions from the
// same sums.
//
// Bound by the matrix (8 n^2 bytes per step, from L2 up to about 3500 unknowns)
// and the latency of the two barriers (about 7 us per step).  Measured on B200, a
// whole solve, against a launch pair per step: 597 unknowns, 39 steps, 0.40 and
// 1.31 ms; 2487 unknowns, 46 steps, 0.81 and 1.97 ms; 5762 unknowns, 32 steps,
// 1.80 and 2.45 ms; 8412 unknowns, 32 steps, 3.81 and 3.79 ms; 10 242 unknowns,
// 32 steps, 7.4 and 5.1 ms (hence kCyMaxRows).
// Barrier waits are bounded (state.err on expiry, after which every CTA leaves).

constexpr int kCyWarps = 15;
constexpr int kCyCompute = 32 * kCyWarps;
constexpr int kCyThreads = kCyCompute + 32;  // + the Givens warp (512: 128 registers each)
constexpr int kCyCopies = 8;
constexpr int kCyMinRows = kCyWarps;  // unknowns per CTA: a row per warp at the least
constexpr int kCyMaxRows = 50;        // above, the matvec kernels stream the matrix faster

struct CyParams {
  double rtol, atol, inner_rtol;
  int max_iters, max_refine, use_x0;
};

// Global state of one solve, zeroed before the launch.
struct CyGlobal {
  GmState state;
  unsigned arrivals;  // of the grid barrier
  int done;           // basis size + 1, once the Givens warp has ended the cycle
  int kend;           // basis size of the last cycle
  int status, iterations, refinements, matvecs, pad;
  double resid;       // residual estimate of the last cycle
  double rel;         // FP64 residual / |b|
  // then double h[2][kCyCopies][2 (R + 2)] (by step parity), nu[2][kCyCopies], sum[4][kCyCopies]
};
__host__ __device__ inline size_t cy_sums(int R) { return (size_t)2 * kCyCopies * 2 * (R + 2); }
__host__ __device__ inline size_t cy_global_bytes(int R) {
  return sizeof(CyGlobal) + sizeof(double) * (cy_sums(R) + 6 * kCyCopies);
}

struct CyLayout {
  size_t x, basis, w, r, d, xs, coef, term, nu, sn, gs, hc, cs, part, total;
};
__host__ __device__ inline CyLayout cy_layout(int n, int rows, int R) {
  CyLayout L;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 15) / 16 * 16;
    return at;
  };
  L.x = take(sizeof(float2) * (size_t)n);
  L.basis = take(sizeof(float2) * (size_t)rows * (R + 1));
  L.w = take(sizeof(double2) * (size_t)rows);
  L.r = take(sizeof(double2) * (size_t)rows);
  L.d = take(sizeof(double2) * (size_t)rows);
  L.xs = take(sizeof(double2) * (size_t)rows);
  L.coef = take(sizeof(double2) * (R + 2));
  L.term = take(sizeof(double) * (R + 2));
  L.nu = take(sizeof(double) * (R + 2));
  L.sn = take(sizeof(double2) * R);
  L.gs = take(sizeof(double2) * (R + 2));
  L.hc = take(sizeof(double2) * (R + 2));
  L.cs = take(sizeof(double) * R);
  L.part = take(sizeof(double2) * kCyCompute);  // a double2 per thread
  L.total = o;
  return L;
}

__device__ __forceinline__ void cy_compute_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kCyCompute) : "memory"); }

// Grid barrier number `index` (from 1): all CTAs are resident.  False on every
// thread of the CTA if a wait expired anywhere.
__device__ __forceinline__ bool cy_grid_sync(CyGlobal* G, unsigned index) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int good = 1;
    __threadfence();  // this CTA's writes and atomics before the arrival
    const unsigned target = index * gridDim.x;
    if (atomicAdd(&G->arrivals, 1u) + 1 < target) {
      const unsigned long long t0 = globaltimer();
      for (unsigned it = 0; ld_acquire_u32(&G->arrivals) < target; it++) {
        if ((it & 63u) == 63u) {
          if (*(volatile int*)&G->state.err) {
            good = 0;
            break;
          }
          if (globaltimer() - t0 > kCoWaitNs) {
            atomicExch(&G->state.err, 1);
            good = 0;
            break;
          }
        }
      }
    }
    __threadfence();
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Rotations of column k (hc[0..k], subdiagonal hn): applies the earlier ones,
// adds the new one, advances g; returns the residual.  One lane.
__device__ __forceinline__ double cy_givens(double2* hc, int k, double hn, double* cs, double2* sn, double2* gs,
                                            bool* breakdown) {
  double2 a = hc[0];
  for (int l = 0; l < k; l++) {
    const double c = cs[l];
    const double2 s = sn[l], b = hc[l + 1];
    const double2 sb = cmul(s, b), t = cmul(make_double2(-s.x, s.y), a);  // -conj(s) a
    hc[l] = make_double2(c * a.x + sb.x, c * a.y + sb.y);
    a = make_double2(t.x + c * b.x, t.y + c * b.y);
  }
  const double na = sqrt(a.x * a.x + a.y * a.y), rho = sqrt(na * na + hn * hn);
  double c = 1.0;
  double2 s = make_double2(0.0, 0.0), d = a;
  if (rho != 0.0 && na == 0.0) {
    c = 0.0;
    s = make_double2(1.0, 0.0);
    d = make_double2(hn, 0.0);
  } else if (rho != 0.0) {
    c = na / rho;
    const double2 ph = make_double2(a.x / na, a.y / na);
    s = make_double2(ph.x * (hn / rho), ph.y * (hn / rho));
    d = make_double2(ph.x * rho, ph.y * rho);
  }
  hc[k] = d;
  cs[k] = c;
  sn[k] = s;
  const double2 gk = gs[k], g1 = cmul(make_double2(-s.x, s.y), gk);
  gs[k + 1] = g1;
  gs[k] = make_double2(c * gk.x, c * gk.y);
  *breakdown = !(hn > 1e-300) || !(hn > 1e-14 * rho);
  return sqrt(g1.x * g1.x + g1.y * g1.y);
}

// w = A x on the CTA's rows (compute warps): a warp sweeps RG rows at once, its
// lanes the columns, U columns in flight; passes of 15 RG rows.
template <int RG, int U, typename T2, typename T, typename X>
__device__ __forceinline__ void cy_sweep(const float2* __restrict__ A, int n, int i0, int rows, X&& x, double2* w) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int r0 = warp; r0 < rows; r0 += RG * kCyWarps) {
    const float2* row[RG];
    T2 acc[RG];
#pragma unroll
    for (int r = 0; r < RG; r++) {
      row[r] = A + (size_t)(i0 + min(r0 + r * kCyWarps, rows - 1)) * n;
      acc[r].x = 0;
      acc[r].y = 0;
    }
    int j = lane;
    for (; j + 32 * (U - 1) < n; j += 32 * U) {
      float2 a[U][RG];
#pragma unroll
      for (int u = 0; u < U; u++)
#pragma unroll
        for (int r = 0; r < RG; r++) a[u][r] = __ldcg(&row[r][j + 32 * u]);
#pragma unroll
      for (int u = 0; u < U; u++) {
        const T2 v = x(j + 32 * u);
#pragma unroll
        for (int r = 0; r < RG; r++) {
          acc[r].x = fma((T)a[u][r].x, v.x, fma((T)-a[u][r].y, v.y, acc[r].x));
          acc[r].y = fma((T)a[u][r].x, v.y, fma((T)a[u][r].y, v.x, acc[r].y));
        }
      }
    }
#pragma unroll 2
    for (; j < n; j += 32) {
      const T2 v = x(j);
#pragma unroll
      for (int r = 0; r < RG; r++) {
        const float2 a = __ldcg(&row[r][j]);
        acc[r].x = fma((T)a.x, v.x, fma((T)-a.y, v.y, acc[r].x));
        acc[r].y = fma((T)a.x, v.y, fma((T)a.y, v.x, acc[r].y));
      }
    }
#pragma unroll
    for (int r = 0; r < RG; r++) {
      double re = (double)acc[r].x, im = (double)acc[r].y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
      }
      if (lane == 0 && r0 + r * kCyWarps < rows) w[r0 + r * kCyWarps] = make_double2(re, im);
    }
  }
}

__global__ void __launch_bounds__(kCyThreads, 1)
    gm_single_kernel(GmPtrs P, const float2* __restrict__ A, const float2* __restrict__ B, float2* __restrict__ Xio,
                     CyGlobal* G, int rows_per_cta, CyParams prm) {
  extern __shared__ __align__(16) unsigned char cy_raw[];
  const int n = P.n, R = P.R, ldj = R + 1;
  const CyLayout L = cy_layout(n, rows_per_cta, R);
  float2* x = (float2*)(cy_raw + L.x);
  float2* basis = (float2*)(cy_raw + L.basis);  // [unknown][vector]
  double2* w = (double2*)(cy_raw + L.w);
  double2* rs = (double2*)(cy_raw + L.r);        // outer residual
  double2* d = (double2*)(cy_raw + L.d);         // correction of the current refinement
  double2* xs = (double2*)(cy_raw + L.xs);       // solution
  double2* coef = (double2*)(cy_raw + L.coef);   // <v_j, w> / |v_j|^2
  double* term = (double*)(cy_raw + L.term);
  double* nu = (double*)(cy_raw + L.nu);         // |v_j|
  double2* sn = (double2*)(cy_raw + L.sn);
  double2* gs = (double2*)(cy_raw + L.gs);
  double2* hc = (double2*)(cy_raw + L.hc);
  double* cs = (double*)(cy_raw + L.cs);
  double* part = (double*)(cy_raw + L.part);
  double2* part2 = (double2*)part;
  double* hsum = (double*)(G + 1);
  double* nsum = hsum + cy_sums(R);
  double* osum = nsum + 2 * kCyCopies;
  const size_t hstride = 2 * (size_t)(R + 2);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool compute = warp < kCyWarps, givens = blockIdx.x == 0 && warp == kCyWarps;
  const int copy = blockIdx.x % kCyCopies;
  const int i0 = blockIdx.x * rows_per_cta, rows = min(rows_per_cta, n - i0);
  unsigned bars = 0, sums = 0;
  __shared__ int s_done;
  __shared__ double s_sum;

  auto scale_of = [](double norm) -> double {  // a power of two near 1 / norm
    return norm > 0.0 && norm < INFINITY ? exp2(-rint(log2(norm))) : 1.0;
  };
  // CTA sum of the compute threads' values, added to *to by thread 0
  auto cta_add = [&](double v, double* to) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[warp] = v;
    cy_compute_sync();
    if (tid == 0) {
      double t = 0.0;
      for (int q = 0; q < kCyWarps; q++) t += part[q];
      atomicAdd(to, t);
    }
  };
  // sum over the grid (all threads call it, compute threads with their values);
  // a slot of `sum` is cleared two uses ahead, when everyone has read it
  auto grid_sum = [&](double v, double* out) -> bool {
    double* slot = osum + (sums & 3) * kCyCopies;
    if (compute) cta_add(v, slot + copy);
    if (!cy_grid_sync(G, ++bars)) return false;
    if (tid == 0) {
      double t = 0.0;
      for (int q = 0; q < kCyCopies; q++) t += __ldcg(&slot[q]);
      s_sum = t;
    }
    if (blockIdx.x == 0 && tid < kCyCopies) osum[((sums + 2) & 3) * kCyCopies + tid] = 0.0;
    sums++;
    __syncthreads();
    *out = s_sum;
    return true;
  };
  // fl32(c value) of unknown i into the basis and the exchange vector; |.|^2
  auto put = [&](int i, int j, double2 v, double c) -> double {
    const float2 f = make_float2((float)(v.x * c), (float)(v.y * c));
    basis[(size_t)i * ldj + j] = f;
    ((j & 1) ? P.Y : P.X)[i0 + i] = f;
    return (double)f.x * f.x + (double)f.y * f.y;
  };
  // compute threads: w = A v, FP32 products (v: all unknowns, complex64)
  auto product = [&](const float2* v) {
    for (int i = tid; i < n; i += kCyCompute) x[i] = __ldcg(&v[i]);
    cy_compute_sync();
    auto xv = [&](int j) { return x[j]; };
    if (rows_per_cta <= kCyWarps)
      cy_sweep<1, 8, float2, float>(A, n, i0, rows, xv, w);
    else if (rows_per_cta <= 2 * kCyWarps)
      cy_sweep<2, 8, float2, float>(A, n, i0, rows, xv, w);
    else if (rows_per_cta <= 3 * kCyWarps)
      cy_sweep<3, 6, float2, float>(A, n, i0, rows, xv, w);
    else
      cy_sweep<4, 4, float2, float>(A, n, i0, rows, xv, w);
    cy_compute_sync();
  };
  // compute threads: w = A x in FP64 (x: all unknowns, complex128)
  auto product64 = [&](const double2* v) {
    cy_sweep<2, 4, double2, double>(
        A, n, i0, rows, [&](int j) { return make_double2(__ldcg(&v[j].x), __ldcg(&v[j].y)); }, w);
    cy_compute_sync();
  };
  // column j's rotations (CTA 0's Givens warp)
  auto rotate = [&](int j, double hn, double tol, int max_steps) {
    for (int l = lane; l <= j; l += 32) {
      const double f = nu[l] / nu[j];
      hc[l] = make_double2(coef[l].x * f, coef[l].y * f);
    }
    __syncwarp();
    if (lane == 0) {
      bool breakdown;
      const double res = cy_givens(hc, j, hn, cs, sn, gs, &breakdown);
      G->resid = res;
      if (res <= tol || breakdown || j + 1 >= max_steps) *(volatile int*)&G->done = j + 2;
    }
    __syncwarp();
    double2* Hj = P.H + (size_t)j * (R + 1);
    for (int l = lane; l <= j; l += 32) Hj[l] = hc[l];
  };
  // sum over the basis, lanes over the vectors: sum_{l < count} v_l(i) coef_l, on every lane
  auto combine = [&](int i, int count) -> double2 {
    double2 t = make_double2(0.0, 0.0);
    for (int l = lane; l < count; l += 32) {
      const float2 v = basis[(size_t)i * ldj + l];
      const double2 p = cmul(make_double2(v.x, v.y), coef[l]);
      t.x += p.x;
      t.y += p.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
      t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
    }
    return t;
  };

  // ---- |b|, the start vector ----
  double n2 = 0.0, bn2, rn2;
  for (int i = tid; i < rows; i += kCyThreads) {
    const float2 b = B[i0 + i];
    rs[i] = make_double2(b.x, b.y);
    const float2 x0 = prm.use_x0 ? Xio[i0 + i] : make_float2(0.f, 0.f);
    xs[i] = make_double2(x0.x, x0.y);
    d[i] = make_double2(0.0, 0.0);
  }
  __syncthreads();
  if (compute)
    for (int i = tid; i < rows; i += kCyCompute) n2 += rs[i].x * rs[i].x + rs[i].y * rs[i].y;
  if (!grid_sum(n2, &bn2)) return;
  const double bn = sqrt(bn2);
  int status = BEM_ERR_NOT_CONVERGED, iterations = 0, refinements = 0, matvecs = 0;
  double rel = 0.0;
  bool x_nonzero = prm.use_x0 != 0;
  for (int outer = 0;; outer++) {
    // ---- FP64 residual, stopping tests ----
    rn2 = bn2;
    if (x_nonzero) {
      for (int i = tid; i < rows; i += kCyThreads) P.x[i0 + i] = xs[i];
      if (!cy_grid_sync(G, ++bars)) return;
      n2 = 0.0;
      if (compute) {
        product64(P.x);
        for (int i = tid; i < rows; i += kCyCompute) {
          const float2 b = B[i0 + i];
          const double2 r = make_double2(b.x - w[i].x, b.y - w[i].y);
          rs[i] = r;
          n2 += r.x * r.x + r.y * r.y;
        }
      }
      if (!grid_sum(n2, &rn2)) return;
      matvecs++;
    }
    const double rn = sqrt(rn2);
    rel = !(isfinite(bn) && isfinite(rn)) ? NAN : (bn > 0.0 ? rn / bn : (rn > 0.0 ? INFINITY : 0.0));
    if (!isfinite(rel)) {
      status = BEM_ERR_NONFINITE;
      break;
    }
    if (rn <= prm.rtol * bn || rn <= prm.atol) {
      status = BEM_OK;
      break;
    }
    if (outer == prm.max_refine || iterations >= prm.max_iters) break;
    refinements = outer + 1;
    const double tol = fmax(prm.inner_rtol * rn, 0.5 * prm.rtol * bn);

    // ---- restarted GMRES on A d = r ----
    bool first = true;
    while (iterations < prm.max_iters) {
      const int max_steps = min(R, prm.max_iters - iterations);
      double beta2 = rn2;
      if (!first) {  // r - A d, with A d in FP32
        for (int i = tid; i < rows; i += kCyThreads) P.X[i0 + i] = make_float2((float)d[i].x, (float)d[i].y);
        if (!cy_grid_sync(G, ++bars)) return;
        n2 = 0.0;
        if (compute) {
          product(P.X);
          for (int i = tid; i < rows; i += kCyCompute) {
            const double2 r = make_double2(rs[i].x - (float)w[i].x, rs[i].y - (float)w[i].y);
            w[i] = r;
            n2 += r.x * r.x + r.y * r.y;
          }
        }
        if (!grid_sum(n2, &beta2)) return;  // everyone is done with P.X
        matvecs++;
      }
      const double beta = sqrt(beta2);
      if (!(beta > tol)) break;  // the start residual meets the target (or is not finite)
      // v_0 = fl32(c r); sums of the last cycle are cleared before the barrier
      const double c0 = scale_of(beta);
      double nu2;
      n2 = 0.0;
      if (compute)
        for (int i = tid; i < rows; i += kCyCompute) n2 += put(i, 0, first ? rs[i] : w[i], c0);
      if (blockIdx.x == gridDim.x - 1)
        for (int e = tid; e < (int)(2 * kCyCopies * (hstride + 1)); e += kCyThreads) hsum[e] = 0.0;  // and nsum, behind it
      if (blockIdx.x == 0 && tid == 0) G->done = 0;
      if (!grid_sum(n2, &nu2)) return;
      first = false;
      if (tid == 0) {
        nu[0] = sqrt(nu2);
        gs[0] = make_double2(nu[0] / c0, 0.0);  // r = g_0 v_0 / |v_0|
      }
      __syncthreads();

      double c = 1.0;  // scale of v_k
      int k = 0;
      for (;; k++) {
        // ---- w = A v_k on the CTA's rows; meanwhile |v_k| and the rotations of column k - 1 ----
        if (compute) {
          product((k & 1) ? P.Y : P.X);
          // <v_j, w>, j <= k, and |w|^2 over the slice: a thread per (vector, part of the unknowns)
          int jw = 32;
          while (jw < k + 2) jw *= 2;
          const int j = tid & (jw - 1), s = tid / jw, S = kCyCompute / jw;
          double2 acc = make_double2(0.0, 0.0);
          if (s >= S) {  // a remainder of threads
          } else if (j <= k) {
            for (int i = s; i < rows; i += S) {
              const float2 v2 = basis[(size_t)i * ldj + j];
              const double2 wv = w[i];
              acc.x += (double)v2.x * wv.x + (double)v2.y * wv.y;
              acc.y += (double)v2.x * wv.y - (double)v2.y * wv.x;
            }
          } else if (j == k + 1) {
            for (int i = s; i < rows; i += S) acc.x += w[i].x * w[i].x + w[i].y * w[i].y;
          }
          part2[tid] = acc;
          cy_compute_sync();
          if (tid < jw && j <= k + 1) {
            for (int q = 1; q < S; q++) {
              acc.x += part2[q * jw + j].x;
              acc.y += part2[q * jw + j].y;
            }
            double* h = hsum + ((size_t)(k & 1) * kCyCopies + copy) * hstride + 2 * j;
            atomicAdd(h, acc.x);
            atomicAdd(h + 1, acc.y);
          }
        } else if (k > 0) {
          if (lane == 0) {
            double t = 0.0;
            for (int q = 0; q < kCyCopies; q++) t += __ldcg(&nsum[(k & 1) * kCyCopies + q]);
            nu[k] = sqrt(t);
          }
          __syncwarp();
          if (givens) rotate(k - 1, nu[k] / (c * nu[k - 1]), tol, max_steps);
        }
        if (!cy_grid_sync(G, ++bars)) return;

        // ---- w' = w - V h, v_{k+1}; the other parity's sums are cleared for the next step ----
        if (tid == 0) s_done = *(volatile int*)&G->done;
        if (tid <= k + 1) {
          double2 h = make_double2(0.0, 0.0);
          for (int q = 0; q < kCyCopies; q++) {
            const double* hq = hsum + ((size_t)(k & 1) * kCyCopies + q) * hstride + 2 * tid;
            h.x += __ldcg(hq);
            h.y += __ldcg(hq + 1);
          }
          const double inv = tid <= k ? 1.0 / (nu[tid] * nu[tid]) : 1.0;
          coef[tid] = make_double2(h.x * inv, h.y * inv);
          term[tid] = tid <= k ? -(h.x * h.x + h.y * h.y) * inv : h.x;
        }
        __syncthreads();
        if (s_done) break;  // with column k - 1
        {  // |w'|^2 = |w|^2 - sum |h_j|^2 / |v_j|^2, exact enough for a power of two
          double t = 0.0;
          for (int l = lane; l <= k + 1; l += 32) t += term[l];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          c = scale_of(sqrt(fmax(t, 1e-12 * term[k + 1])));
        }
        if (compute) {
          n2 = 0.0;
          for (int i = warp; i < rows; i += kCyWarps) {
            const double2 t = combine(i, k + 1);
            if (lane == 0) n2 += put(i, k + 1, make_double2(w[i].x - t.x, w[i].y - t.y), c);
          }
          cta_add(n2, &nsum[((k + 1) & 1) * kCyCopies + copy]);
          if (blockIdx.x == gridDim.x - 1) {
            double* h = hsum + (size_t)((k + 1) & 1) * kCyCopies * hstride;
            for (int e = tid; e < (int)(kCyCopies * hstride); e += kCyCompute) h[e] = 0.0;
          }
        }
        if (!cy_grid_sync(G, ++bars)) return;
        // |v_k| has been read by everyone: its sum is cleared for |v_{k+2}|
        if (blockIdx.x == 0 && tid < kCyCopies) nsum[(k & 1) * kCyCopies + tid] = 0.0;
        if (k + 1 == max_steps) {  // no further product: the last column's rotations now
          if (tid == kCyCompute) {
            double t = 0.0;
            for (int q = 0; q < kCyCopies; q++) t += __ldcg(&nsum[((k + 1) & 1) * kCyCopies + q]);
            nu[k + 1] = sqrt(t);
          }
          __syncwarp();
          if (givens) rotate(k, nu[k + 1] / (c * nu[k]), tol, max_steps);
          k++;
          break;
        }
      }
      // the basis has k vectors that count

      // ---- H y = g (CTA 0), then d += V y ----
      __syncthreads();
      if (blockIdx.x == 0 && compute) {
        double2 g = make_double2(0.0, 0.0), inv = g;
        if (tid < k) {
          g = gs[tid];
          const double2 dd = P.H[(size_t)tid * (R + 1) + tid];
          const double den = dd.x * dd.x + dd.y * dd.y;
          if (den > 0.0) inv = make_double2(dd.x / den, -dd.y / den);
        }
        constexpr int kAhead = 4;  // columns of H in registers, loaded that many steps ahead
        double2 col[kAhead];
        auto load = [&](int j) {
          return j >= 0 && tid < j ? P.H[(size_t)j * (R + 1) + tid] : make_double2(0.0, 0.0);
        };
#pragma unroll
        for (int q = 0; q < kAhead; q++) col[q] = load(k - 1 - q);
        for (int jb = k - 1; jb >= 0; jb -= kAhead) {
#pragma unroll
          for (int q = 0; q < kAhead; q++) {
            const int j = jb - q;  // uniform
            if (j < 0) break;
            if (tid == j) hc[j] = cmul(g, inv);
            cy_compute_sync();
            const double2 t = cmul(col[q], hc[j]);
            g.x -= t.x;
            g.y -= t.y;
            col[q] = load(j - kAhead);
          }
        }
        if (tid < k) {
          const double f = 1.0 / nu[tid];
          ((double2*)P.y)[tid] = make_double2(hc[tid].x * f, hc[tid].y * f);
        }
      }
      if (!cy_grid_sync(G, ++bars)) return;
      const double2* y = (const double2*)P.y;
      for (int l = tid; l < k; l += kCyThreads) coef[l] = make_double2(__ldcg(&y[l].x), __ldcg(&y[l].y));
      if (tid == 0) s_sum = __ldcg(&G->resid);
      __syncthreads();
      const double res = s_sum;
      if (compute)
        for (int i = warp; i < rows; i += kCyWarps) {
          const double2 t = combine(i, k);
          if (lane == 0) {
            d[i].x += t.x;
            d[i].y += t.y;
          }
        }
      __syncthreads();
      iterations += k;
      if (!(res > tol)) break;
    }
    for (int i = tid; i < rows; i += kCyThreads) {
      xs[i].x += d[i].x;
      xs[i].y += d[i].y;
      d[i] = make_double2(0.0, 0.0);
    }
    __syncthreads();
    x_nonzero = true;
  }
  for (int i = tid; i < rows; i += kCyThreads) Xio[i0 + i] = make_float2((float)xs[i].x, (float)xs[i].y);
  if (blockIdx.x == 0 && tid == 0) {
    G->status = status;
    G->iterations = iterations;
    G->refinements = refinements;
    G->matvecs = matvecs + iterations;
    G->rel = rel;
  }
}
