// Strip sweep of regular triangle pairs, shared by the V/K and the
// Burton-Miller assembly.
//
// The sorted triangles come in blocks of 32 whose members are ordered as
// paths over shared edges (geometry.cu).  A warp owns one test block (a test
// triangle per lane) and walks along a trial block: all lanes meet the same
// trial triangle at the same time, consecutive trial triangles keep their
// shared vertices in the same local slots, so the 3 x 3 blocks of a pair are
// summed in registers, by trial slot, until the slot's vertex leaves the path.
// Only then (about 1.2 columns per trial triangle instead of 3) the column is
// reduced over the block's test corners in the warp's own shared memory and
// added to the matrices.  Nothing is shared between warps: no block barrier,
// and a warp's reduction overlaps the other warps' arithmetic.
//
#pragma once

#include "async_copy.cuh"
#include "bem_common.cuh"

namespace bemb {

// Programmatic launch: lets the next kernel start as soon as every block of
// this one runs / waits for the kernels before this one to finish.
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch attributes of a kernel that may start while the one before it in the
// stream still runs (it calls wait_previous() before it ends).
struct EarlyLaunch {
  cudaLaunchAttribute attr{};
  cudaLaunchConfig_t cfg{};
  EarlyLaunch(unsigned blocks, int threads, size_t smem, cudaStream_t s) {
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
  }
};

constexpr int kStripThreads = 128;
constexpr int kStripWarps = kStripThreads / 32;
constexpr int kStripZero = kBlockCorners;  // index of a column entry that stays zero

// One warp's shared memory: the trial block being walked and the next one
// (bulk copies), ROWS values per test triangle (structure of arrays), and two
// columns of corner values (three complex numbers per test corner).
template <int ROWS, bool BM>
struct StripWarp {
  TriRec trial[2][kBlock];
  BmRec trial_bm[BM ? 2 : 1][BM ? kBlock : 1];
  float xs[ROWS][32];
  float4 col4[2][kBlockCorners + 1];
  float2 col2[2][kBlockCorners + 1];
  uint64_t full[2];
};

// The warp's position: test block `grp`, its lane's triangle and the lane's
// entry of the block's vertex table.
struct StripTest {
  int grp = -1;
  bool valid;
  float area, nx, ny, nz, cx, cy, cz;
  int v0, v1, v2;
  int nlv, most;   // distinct vertices of the block, most corners of one vertex
  int vid;         // vertex `lane` (or -1), its corners as bytes (8 at most), their number
  unsigned c_lo, c_hi;
  int corners;
};

__device__ __forceinline__ void strip_load_test(StripTest& t, const GeomView& g, int grp) {
  const int lane = threadIdx.x & 31;
  t.grp = grp;
  const int ti = grp * kBlock + lane;
  t.valid = ti < g.nt;
  const TriRec& r = g.rec[t.valid ? ti : g.nt - 1];
  t.area = r.area;
  t.nx = r.n[0];
  t.ny = r.n[1];
  t.nz = r.n[2];
  t.cx = r.c[0];
  t.cy = r.c[1];
  t.cz = r.c[2];
  t.v0 = r.v[0];
  t.v1 = r.v[1];
  t.v2 = r.v[2];
  const BlockRec& b = g.blocks[grp];
  t.nlv = b.nlv;
  t.most = b.most < 8 ? b.most : 8;
  t.vid = -1;
  t.corners = 0;
  t.c_lo = t.c_hi = kStripZero * 0x01010101u;
  if (lane < b.nlv) {
    const int p0 = b.ptr[lane];
    t.corners = b.ptr[lane + 1] - p0;
    t.vid = b.vid[lane];
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i < t.corners) {
        const unsigned c = b.corner[p0 + i];
        const int sh = 8 * (i & 3);
        if (i < 4)
          t.c_lo = (t.c_lo & ~(0xffu << sh)) | (c << sh);
        else
          t.c_hi = (t.c_hi & ~(0xffu << sh)) | (c << sh);
      }
  }
}

// Lane 0: bulk-copy trial block jb into buffer b.
template <int ROWS, bool BM>
__device__ __forceinline__ void strip_fetch(StripWarp<ROWS, BM>& sw, const GeomView& g, int jb, int b) {
  const int ntri = min(kBlock, g.nt - jb * kBlock);
  const uint32_t rb = (uint32_t)(ntri * sizeof(TriRec)), mb = BM ? (uint32_t)(ntri * sizeof(BmRec)) : 0u;
  mbar_expect_tx(&sw.full[b], rb + mb);
  bulk_load(sw.trial[b], &g.rec[jb * kBlock], rb, &sw.full[b]);
  if (BM) bulk_load(sw.trial_bm[BM ? b : 0], &g.bm[jb * kBlock], mb, &sw.full[b]);
}

template <int ROWS, bool BM>
__device__ __forceinline__ void strip_init(StripWarp<ROWS, BM>& sw) {
  if ((threadIdx.x & 31) == 0) {
    mbar_init(&sw.full[0], 1);
    mbar_init(&sw.full[1], 1);
    mbar_init_fence();
    for (int i = 0; i < 2; i++) {
      sw.col4[i][kStripZero] = make_float4(0.f, 0.f, 0.f, 0.f);
      sw.col2[i][kStripZero] = make_float2(0.f, 0.f);
    }
  }
  __syncwarp();
}

// The two columns in col4/col2 (corner a of lane t at 32 a + t; trial vertices
// b0 and b1, b1 < 0 if there is one column only) summed over the test corners
// of each distinct vertex A of the block, handed to store(A, b, sum4, sum2).
// Two at a time, since the sums are short chains of shared-memory loads.
// Lane l takes vertices l, l + 32, ...; the first 8 corners of vertex `lane`
// sit in registers, what lies beyond (blocks with more than 32 vertices,
// vertices with more than 8 corners in one block) is read from the block's
// table.
template <int ROWS, bool BM, typename F>
__device__ __forceinline__ void strip_reduce(StripWarp<ROWS, BM>& sw, const StripTest& t, const GeomView& g, int b0,
                                             int b1, F&& store) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the columns are complete
  float4 s4[2];
  float2 s2[2];
  auto clear = [&]() {
    s4[0] = s4[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    s2[0] = s2[1] = make_float2(0.f, 0.f);
  };
  auto add = [&](int c) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const float4 x = sw.col4[i][c];
      const float2 y = sw.col2[i][c];
      s4[i].x += x.x;
      s4[i].y += x.y;
      s4[i].z += x.z;
      s4[i].w += x.w;
      s2[i].x += y.x;
      s2[i].y += y.y;
    }
  };
  clear();
  unsigned lo = t.c_lo, hi = t.c_hi;
  for (int i = 0; i < t.most; i += 2) {  // unused places point at the zero entry
    add(lo & 0xff);
    add((lo >> 8) & 0xff);
    lo = __funnelshift_r(lo, hi, 16);
    hi >>= 16;
  }
  if (t.corners > 8) {
    const BlockRec& b = g.blocks[t.grp];
    for (int i = b.ptr[lane] + 8; i < b.ptr[lane + 1]; i++) add(b.corner[i]);
  }
  if (t.vid >= 0) {
    store(t.vid, b0, s4[0], s2[0]);
    if (b1 >= 0) store(t.vid, b1, s4[1], s2[1]);
  }
  for (int l = lane + 32; l < t.nlv; l += 32) {
    const BlockRec& b = g.blocks[t.grp];
    clear();
    for (int i = b.ptr[l]; i < b.ptr[l + 1]; i++) add(b.corner[i]);
    store(b.vid[l], b0, s4[0], s2[0]);
    if (b1 >= 0) store(b.vid[l], b1, s4[1], s2[1]);
  }
  __syncwarp();  // the columns may be overwritten
}

// Walks `steps` steps of one problem from trial triangle t0 of trial block jb on,
// for test block grp: a step is one trial triangle (blocks count 32, the last
// one too), after the last trial block comes the next test block's own.
// `uses` counts the trial blocks this warp has fetched (buffer uses & 1,
// mbarrier parity (uses >> 1) & 1).  Pol provides
//   load(sw, t, g, lane)                  the test block's rows of sw.xs,
//   pair(sw, t, rec, bm record, weight)   adds the pair's blocks,
//   take<B>(sw, i, lane)                  moves trial slot B's column into
//                                         sw.col4[i] / sw.col2[i] and clears it,
//   store(g, A, B, sum4, sum2)            adds the sums of vertices (A, B).
template <int ROWS, bool BM, typename Pol>
__device__ __forceinline__ void strip_walk(StripWarp<ROWS, BM>& sw, StripTest& test, const GeomView& g, Pol& pol,
                                           int grp, int jb, int t0, int steps, unsigned& uses,
                                           int* process_err) {
  const int lane = threadIdx.x & 31;
  if (steps <= 0) return;
  const int nb = g.nblocks;
  if (lane == 0) strip_fetch(sw, g, jb, uses & 1);
  for (; steps > 0; uses++) {
    const int t1 = min(32, t0 + steps);
    const int bf = uses & 1;
    steps -= t1 - t0;
    int next_grp = grp, next_jb = jb + 1;
    if (next_jb == nb) next_jb = ++next_grp;
    __syncwarp();  // every lane is done with buffer bf ^ 1 and with xs
    if (lane == 0 && steps > 0) strip_fetch(sw, g, next_jb, bf ^ 1);
    if (grp != test.grp) {
      strip_load_test(test, g, grp);
      pol.load(sw, test, g, lane);
    }
    if (!mbar_wait(&sw.full[bf], (uses >> 1) & 1u, g.err)) {
      // expired (this geometry's status word raised): record it process-wide
      // too, and let the copy land before the buffer is reused
      if (lane == 0) atomicExch(process_err, 1);
      mbar_wait_drain(&sw.full[bf], (uses >> 1) & 1u);
    }
    __syncwarp();  // xs is written
    const int stop = min(t1, g.nt - jb * kBlock);
    int waiting = -1;  // trial vertex of the column in col4[0], if one waits for the next
#pragma unroll 1
    for (int t = t0; t < stop; t++) {
      const TriRec& rj = sw.trial[bf][t];
      const int j0 = rj.v[0], j1 = rj.v[1], j2 = rj.v[2];
      const bool touching = (test.v0 == j0) | (test.v0 == j1) | (test.v0 == j2) | (test.v1 == j0) | (test.v1 == j1) |
                            (test.v1 == j2) | (test.v2 == j0) | (test.v2 == j1) | (test.v2 == j2);
      // on the test block itself each unordered pair once
      const bool once = jb > grp || t > lane;
      const float w = (test.valid && !touching && once) ? test.area * rj.area : 0.f;
      if (__any_sync(0xffffffffu, w != 0.f)) pol.pair(sw, test, rj, sw.trial_bm[BM ? bf : 0][BM ? t : 0], w, lane);
      const bool last = t + 1 == stop;
      const int leave = last ? 7 : rj.leave;  // slots whose vertex leaves the path
#pragma unroll 1
      for (int b = 0; b < 3; b++) {  // one copy of the reduction (instruction cache)
        if (!((leave >> b) & 1)) continue;
        const int at = waiting >= 0;
        if (b == 0)
          pol.template take<0>(sw, at, lane);
        else if (b == 1)
          pol.template take<1>(sw, at, lane);
        else
          pol.template take<2>(sw, at, lane);
        const int vertex = b == 0 ? j0 : (b == 1 ? j1 : j2);
        if (at || (last && b == 2)) {
          strip_reduce(sw, test, g, at ? waiting : vertex, at ? vertex : -1,
                       [&](int A, int B, const float4& s4, const float2& s2) { pol.store(g, A, B, s4, s2); });
          waiting = -1;
        } else {
          waiting = vertex;
        }
      }
    }
    grp = next_grp;
    jb = next_jb;
    t0 = 0;
  }
}

// Work items of one problem, in one of two orders.
//   panel == 0: runs of `chunk` steps, the block pairs taken test block by test
//     block.  Long items have fewer column flushes, but the warps then work all
//     over the matrices.
//   panel > 0 (Burton-Miller): an item is one test block against `panel` trial blocks, panel by
//     panel: at any time the warps work on a few columns of block pairs (and,
//     mirrored, rows), whose entries stay in L2 until their neighbours'
//     contributions have arrived.
struct StripItems {
  long long items, steps;
  int chunk, panel;
};

// Item `item` of P (all lanes).
template <int ROWS, bool BM, typename Pol>
__device__ __forceinline__ void strip_item(StripWarp<ROWS, BM>& sw, StripTest& test, const GeomView& g, Pol& pol,
                                           const StripItems& P, long long item, unsigned& uses, int* process_err) {
  const int nb = g.nblocks;
  int grp, jb, t0 = 0, steps;
  if (!BM || P.panel == 0) {
    const long long pos = item * P.chunk, unit = pos >> 5;
    grp = tile_group_of(unit, nb);
    jb = grp + (int)(unit - tile_units_before(grp, nb));
    t0 = (int)(pos & 31);
    steps = (int)(P.steps - pos < P.chunk ? P.steps - pos : P.chunk);
  } else {
    // panel c holds test blocks 0 .. panel (c + 1) - 1 (or nb - 1)
    const long long q = item / P.panel;
    long long c = (long long)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
    while (c > 0 && c * (c + 1) / 2 > q) c--;
    while ((c + 1) * (c + 2) / 2 <= q) c++;
    grp = (int)(item - P.panel * (c * (c + 1) / 2));
    const int first = (int)c * P.panel;
    jb = first > grp ? first : grp;
    steps = 32 * ((first + P.panel < nb ? first + P.panel : nb) - jb);
  }
  strip_walk(sw, test, g, pol, grp, jb, t0, steps, uses, process_err);  // one copy (instruction cache)
}

// Steps of a problem's walk.
inline long long strip_steps(int nblocks) { return 32LL * nblocks * (nblocks + 1) / 2; }

// Equal items go in `rounds` rounds over the warps that are resident, a CTA per
// four items, handed out in order: an SM that is ahead takes more of them, and
// what runs at one time writes neighbouring rows.  One item per warp left 10 %
// of the warp slots empty at the end.  Measured on B200, one round against many
// of at least 64 steps: V and K 20 480 triangles 14.1 and 13.5 ms, 8286
// triangles 2.63 and 2.48 ms, 5120 triangles 1.06 and 1.05 ms (16 steps 1.11);
// the Burton-Miller pair's panels 8.48 and 8.28 ms, with 6-point rules 20.2 and
// 18.6 ms.
constexpr int kStripRounds = 32, kStripRoundSteps = 64;

// Steps of an item, at most `most` rounds.
inline long long strip_part(long long steps, long long warps, int most) {
  long long rounds = steps / (warps * kStripRoundSteps);
  rounds = rounds < 1 ? 1 : (rounds < most ? rounds : most);
  return (steps + warps * rounds - 1) / (warps * rounds);
}

// The items for `warps` resident warps, at least `least` steps each; `blocks`
// trial blocks per item if that is not 0 (tuning).  Panels of `panel` blocks (0:
// never) are taken where the two matrices exceed the L2 cache by far (64 MB)
// and every warp gets `panel_items` of them, so that the uneven last round is
// small.  Measured on B200 for the Burton-Miller pair (at the 3-point rule a
// pair takes a third of the V/K pair's time, so that its atomics weigh more),
// contiguous items in one round against panels of 2: 20 480 triangles 11.8 and
// 8.5 ms, 8286 triangles 1.75 and 1.53 ms, 5120 triangles 0.66 and 0.68 ms.
// Against contiguous items in rounds, panels gain 2 % with the 6-point rules.  V
// and K take none: 81 920 triangles 206.4 ms in rounds, 207.0 ms in panels of 8.
inline StripItems strip_items(int nv, int nblocks, long long warps, int rounds, long long least, int blocks,
                              int panel, int panel_items) {
  StripItems P;
  P.steps = strip_steps(nblocks);
  const long long share = (P.steps + warps - 1) / warps;
  P.panel = blocks == 0 && 16.0 * nv * nv > 64e6 && share >= 32LL * panel * panel_items ? panel : 0;
  const long long part = strip_part(P.steps, warps, rounds);
  const long long chunk = blocks > 0 ? 32LL * blocks : (part > least ? part : least);
  P.chunk = (int)(chunk < (1 << 30) ? chunk : (1 << 30));
  if (P.panel) {
    const long long panels = (nblocks + P.panel - 1) / P.panel;
    P.items = P.panel * (panels * (panels - 1) / 2) + nblocks;
  } else {
    P.items = (P.steps + P.chunk - 1) / P.chunk;
  }
  return P;
}

}  // namespace bemb
