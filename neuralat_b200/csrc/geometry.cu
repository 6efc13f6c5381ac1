// Geometry set-up: validation, per-triangle quadrature records, locality
// sorted 16-triangle tiles and touching-pair lists.
//
// The reference recomputes everything per assembly call and discovers the
// touching pairs of every triangle with an O(T) scan per block
// (src/bem/cuda/bind.cu:81-97, capped at 64 neighbours by `adj[64]`).  Here
// the combinatorics are done once, exactly, on the host (no cap), and the
// floating-point records are computed on the device in FP64 and rounded.

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "bem_common.cuh"

namespace bemb {

namespace {

inline uint64_t align_up(uint64_t x, uint64_t a) { return (x + a - 1) / a * a; }

// Spread the low 10 bits of v so that there are two zero bits between each.
inline uint32_t part1by2(uint32_t v) {
  v &= 0x3ff;
  v = (v | (v << 16)) & 0x030000FF;
  v = (v | (v << 8)) & 0x0300F00F;
  v = (v | (v << 4)) & 0x030C30C3;
  v = (v | (v << 2)) & 0x09249249;
  return v;
}

struct HostGeom {
  int nv = 0, nt = 0, ntiles = 0, nblocks = 0;
  std::vector<float> vertices;
  std::vector<int> triangles;
  std::vector<int> perm;
  std::vector<int> slots;
  std::vector<TileRec> tiles;
  std::vector<BlockRec> blocks;
  std::vector<int2> edge_pairs, vert_pairs, vert_mirror;  // vert_pairs: test < trial, vert_mirror: test > trial
  int max_valence = 0;
  GeomHeader hdr{};
};

int analyse_host(HostGeom& g);

// The most recent analysis of this host thread: bem_geometry_bytes followed by
// bem_geometry_build on an unchanged mesh analyses it once, and a rebuild of
// an unchanged mesh re-uploads its staged integer tables.
thread_local HostGeom t_last;
thread_local bool t_last_valid = false;

// Pinned host buffer of this thread (grown on demand).
struct PinnedBuf {
  char* p = nullptr;
  size_t cap = 0;
  ~PinnedBuf() {
    if (p) cudaFreeHost(p);
  }
  int ensure(size_t n) {
    if (cap >= n) return BEM_OK;
    if (p) cudaFreeHost(p);
    p = nullptr;
    cap = 0;
    BEM_CUDA_TRY(cudaHostAlloc((void**)&p, n, cudaHostAllocDefault));
    cap = n;
    return BEM_OK;
  }
};
thread_local PinnedBuf t_download;  // the mesh read back for the comparison with t_last
thread_local PinnedBuf t_stage;     // t_last's integer tables as uploaded (valid if t_stage_ok)
thread_local bool t_stage_ok = false;

// Analysis of the mesh on the device (t_last; valid until the next call on
// this thread).
int analyse(const float* d_vertices, int nv, const int* d_triangles, int nt, cudaStream_t s, const HostGeom** out) {
  if (nv <= 0 || nt <= 0 || !d_vertices || !d_triangles) return BEM_ERR_INVALID_ARGUMENT;
  const size_t vb = sizeof(float) * 3 * (size_t)nv, tb = sizeof(int) * 3 * (size_t)nt;
  int rc = t_download.ensure(vb + tb);
  if (rc) return rc;
  BEM_CUDA_TRY(cudaMemcpyAsync(t_download.p, d_vertices, vb, cudaMemcpyDeviceToHost, s));
  BEM_CUDA_TRY(cudaMemcpyAsync(t_download.p + vb, d_triangles, tb, cudaMemcpyDeviceToHost, s));
  BEM_CUDA_TRY(cudaStreamSynchronize(s));
  if (t_last_valid && t_last.nv == nv && t_last.nt == nt && std::memcmp(t_last.vertices.data(), t_download.p, vb) == 0 &&
      std::memcmp(t_last.triangles.data(), t_download.p + vb, tb) == 0) {
    *out = &t_last;
    return BEM_OK;
  }
  t_last_valid = false;
  t_stage_ok = false;
  t_last.edge_pairs.clear();  // the vectors keep their capacity from mesh to mesh
  t_last.vert_pairs.clear();
  t_last.vert_mirror.clear();
  t_last.max_valence = 0;
  t_last.nv = nv;
  t_last.nt = nt;
  t_last.vertices.assign((const float*)t_download.p, (const float*)t_download.p + 3 * (size_t)nv);
  t_last.triangles.assign((const int*)(t_download.p + vb), (const int*)(t_download.p + vb) + 3 * (size_t)nt);
  rc = analyse_host(t_last);
  if (rc) return rc;
  t_last_valid = true;
  *out = &t_last;
  return BEM_OK;
}

// Vertex in slot a of the triangle at sorted position s.
inline int slot_vertex(const HostGeom& g, int s, int a) {
  return g.triangles[3 * (size_t)g.perm[s] + ((g.slots[s] >> (2 * a)) & 3)];
}

// Cuts the sorted triangles into blocks of 32 that share as many vertices as
// possible: a block grows from the first free triangle in Morton order, each
// time by the triangle across one of its edges that brings no new vertex, then
// by the one with the fewest free neighbours (so that no islands stay behind),
// the oldest first (so that it stays round).  Blocks of a closed mesh hold
// about 26 vertices (31 with plain runs of the Morton order), which is what a
// column flush of the strip kernels costs.
void grow_blocks(HostGeom& g, const std::vector<int>& nbr) {
  const int nt = g.nt;
  std::vector<int> order(g.perm), mark(g.nv, -1);
  std::vector<uint8_t> state(nt, 0);  // 0 free, 1 in the list of candidates, 2 taken
  std::vector<int> cand;
  int next = 0, done = 0;
  for (int blk = 0; done < nt; blk++) {
    cand.clear();
    for (int n = 0; n < kBlock && done < nt; n++) {
      int best = -1, best_score = -1;
      for (size_t c = 0; c < cand.size(); c++) {
        const int* v = &g.triangles[3 * (size_t)cand[c]];
        int score = (mark[v[0]] == blk) + (mark[v[1]] == blk) + (mark[v[2]] == blk);
        score *= 4;
        for (int e = 0; e < 3; e++) {
          const int j = nbr[3 * (size_t)cand[c] + e];
          score += j < 0 || state[j] == 2;
        }
        if (score > best_score) {
          best_score = score;
          best = (int)c;
        }
      }
      int tri;
      if (best >= 0) {
        tri = cand[best];
        cand.erase(cand.begin() + best);
      } else {
        while (state[order[next]] == 2) next++;
        tri = order[next];
      }
      state[tri] = 2;
      g.perm[done++] = tri;
      for (int a = 0; a < 3; a++) mark[g.triangles[3 * (size_t)tri + a]] = blk;
      for (int e = 0; e < 3; e++) {
        const int j = nbr[3 * (size_t)tri + e];
        if (j >= 0 && state[j] == 0) {
          state[j] = 1;
          cand.push_back(j);
        }
      }
    }
    for (int c : cand) state[c] = 0;
  }
}

// Orders the triangles of every 32-triangle block of the sorted order as
// paths over shared edges (nbr: up to three edge neighbours per triangle) and
// chooses the slots of each triangle's vertices and its leave bits (BlockRec).
// From a triangle the path goes on to the neighbour with the fewest
// neighbours left, so that few triangles end up alone.
void path_order(HostGeom& g, const std::vector<int>& nbr) {
  const int nt = g.nt;
  g.slots.assign(nt, 0);
  std::vector<int> place(nt);  // sorted position of a triangle
  for (int s = 0; s < nt; s++) place[g.perm[s]] = s;
  for (int b0 = 0; b0 < nt; b0 += kBlock) {
    const int n = std::min(kBlock, nt - b0);
    int tri[kBlock], left[kBlock], near[kBlock][3];
    bool used[kBlock];
    for (int i = 0; i < n; i++) {
      tri[i] = g.perm[b0 + i];
      used[i] = false;
      left[i] = 0;
      for (int e = 0; e < 3; e++) {
        const int j = nbr[3 * (size_t)tri[i] + e];
        const int p = j < 0 ? -1 : place[j] - b0;
        near[i][e] = p >= 0 && p < n ? p : -1;
        left[i] += near[i][e] >= 0;
      }
    }
    int last = -1, prev[3] = {-1, -1, -1};  // the path's last triangle, the vertices in its slots
    for (int s = 0; s < n; s++) {
      int best = -1;
      if (last >= 0)
        for (int e = 0; e < 3; e++) {
          const int i = near[last][e];
          if (i >= 0 && !used[i] && (best < 0 || left[i] < left[best] || (left[i] == left[best] && i < best))) best = i;
        }
      if (best < 0)  // a new path
        for (int i = 0; i < n; i++)
          if (!used[i] && (best < 0 || left[i] < left[best])) best = i;
      used[best] = true;
      for (int e = 0; e < 3; e++)
        if (near[best][e] >= 0) left[near[best][e]]--;
      // shared vertices keep their slots, the others fill the free ones in order
      const int* v = &g.triangles[3 * (size_t)tri[best]];
      int slot[3] = {-1, -1, -1};  // local vertex in each slot
      bool kept[3] = {false, false, false};
      for (int a = 0; a < 3; a++)
        for (int c = 0; c < 3; c++)
          if (prev[a] == v[c]) {
            slot[a] = c;
            kept[c] = true;
          }
      int leave = 0;
      for (int a = 0; a < 3; a++)
        if (slot[a] < 0) {
          leave |= 1 << a;
          int c = 0;
          while (kept[c]) c++;
          slot[a] = c;
          kept[c] = true;
        }
      if (s > 0) g.slots[b0 + s - 1] |= leave << 8;
      g.slots[b0 + s] = slot[0] | (slot[1] << 2) | (slot[2] << 4);
      g.perm[b0 + s] = tri[best];
      for (int a = 0; a < 3; a++) prev[a] = v[slot[a]];
      last = best;
    }
    g.slots[b0 + n - 1] |= 7 << 8;
  }
}

// Vertex table of `ntri` triangles from sorted position s0: the distinct
// vertices in order of appearance (vid, returns their number), the corners of
// each (ptr, corner; corner a of triangle t is st t + sa a) and, unless null,
// each corner's local vertex.  stamp / local: scratch, one entry per vertex
// (`tag` differs from call to call).
int local_vertices(const HostGeom& g, int s0, int ntri, int st, int sa, int tag, std::vector<int>& stamp,
                   std::vector<int>& local, int* vid, uint8_t* ptr, uint8_t* corner, uint8_t* corner_lv) {
  int n = 0, lv[kBlockCorners], fill[kBlockCorners + 1] = {0};
  for (int c = 0; c < 3 * ntri; c++) {
    const int v = slot_vertex(g, s0 + c / 3, c % 3);
    if (stamp[v] != tag) {
      stamp[v] = tag;
      local[v] = n;
      vid[n++] = v;
    }
    lv[c] = local[v];
    fill[lv[c] + 1]++;
  }
  for (int l = 0; l < n; l++) {
    fill[l + 1] += fill[l];
    ptr[l] = (uint8_t)fill[l];
  }
  ptr[n] = (uint8_t)(3 * ntri);
  for (int c = 0; c < 3 * ntri; c++) {
    const int at = st * (c / 3) + sa * (c % 3);
    corner[fill[lv[c]]++] = (uint8_t)at;
    if (corner_lv) corner_lv[at] = (uint8_t)lv[c];
  }
  return n;
}

int analyse_host(HostGeom& g) {
  const int nv = g.nv, nt = g.nt;

  for (size_t i = 0; i < g.vertices.size(); i++)
    if (!std::isfinite(g.vertices[i])) return BEM_ERR_NONFINITE;
  for (int i = 0; i < nt; i++) {
    const int* t = &g.triangles[3 * (size_t)i];
    for (int a = 0; a < 3; a++)
      if (t[a] < 0 || t[a] >= nv) return BEM_ERR_INDEX;
    if (t[0] == t[1] || t[1] == t[2] || t[0] == t[2]) return BEM_ERR_DEGENERATE;
    double p[3][3];
    for (int a = 0; a < 3; a++)
      for (int c = 0; c < 3; c++) p[a][c] = g.vertices[3 * (size_t)t[a] + c];
    double e1[3] = {p[1][0] - p[0][0], p[1][1] - p[0][1], p[1][2] - p[0][2]};
    double e2[3] = {p[2][0] - p[0][0], p[2][1] - p[0][1], p[2][2] - p[0][2]};
    double cx = e1[1] * e2[2] - e1[2] * e2[1], cy = e1[2] * e2[0] - e1[0] * e2[2], cz = e1[0] * e2[1] - e1[1] * e2[0];
    if (!(cx * cx + cy * cy + cz * cz > 0.0)) return BEM_ERR_DEGENERATE;
  }

  // Morton order of centroids (10 bits per axis over the bounding box).
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int v = 0; v < nv; v++)
    for (int c = 0; c < 3; c++) {
      lo[c] = std::min(lo[c], (double)g.vertices[3 * (size_t)v + c]);
      hi[c] = std::max(hi[c], (double)g.vertices[3 * (size_t)v + c]);
    }
  double ext = std::max({hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2], 1e-30});
  std::vector<uint64_t> key(nt);
  for (int i = 0; i < nt; i++) {
    uint32_t q[3];
    for (int c = 0; c < 3; c++) {
      double m = 0.0;
      for (int a = 0; a < 3; a++) m += g.vertices[3 * (size_t)g.triangles[3 * (size_t)i + a] + c];
      m = (m / 3.0 - lo[c]) / ext;
      q[c] = (uint32_t)std::min(1023.0, std::max(0.0, std::floor(m * 1024.0)));
    }
    uint64_t code = part1by2(q[0]) | (part1by2(q[1]) << 1) | (part1by2(q[2]) << 2);
    key[i] = (code << 32) | (uint32_t)i;
  }
  // three counting passes over the 30-bit code (stable: equal codes keep the input order)
  {
    std::vector<uint64_t> other(nt);
    for (int shift = 32; shift < 62; shift += 10) {
      int start[1025] = {0};
      for (int i = 0; i < nt; i++) start[((key[i] >> shift) & 1023) + 1]++;
      for (int d = 0; d < 1024; d++) start[d + 1] += start[d];
      for (int i = 0; i < nt; i++) other[start[(key[i] >> shift) & 1023]++] = key[i];
      key.swap(other);
    }
  }
  g.perm.resize(nt);
  for (int s2 = 0; s2 < nt; s2++) g.perm[s2] = (int)(key[s2] & 0xffffffffu);

  // Vertex stars and touching pairs (exact, no neighbour cap).
  std::vector<int> vptr(nv + 1, 0), vtri(3 * (size_t)nt);
  for (int i = 0; i < 3 * nt; i++) vptr[g.triangles[i] + 1]++;
  for (int v = 0; v < nv; v++) {
    g.max_valence = std::max(g.max_valence, vptr[v + 1]);
    vptr[v + 1] += vptr[v];
  }
  {
    std::vector<int> fill(vptr.begin(), vptr.end() - 1);
    for (int i = 0; i < nt; i++)
      for (int a = 0; a < 3; a++) vtri[fill[g.triangles[3 * (size_t)i + a]]++] = i;
  }
  std::vector<int> nbr(3 * (size_t)nt, -1);  // triangles across an edge (three at most are used)
  // triangles meeting i in the order of its stars; 4 i + vertices shared with i
  std::vector<int> touch;
  std::vector<long long> shared(nt, -1);
  g.edge_pairs.reserve(3 * (size_t)nt);
  g.vert_pairs.reserve(5 * (size_t)nt);
  g.vert_mirror.reserve(5 * (size_t)nt);
  for (int i = 0; i < nt; i++) {
    const int* ti = &g.triangles[3 * (size_t)i];
    touch.clear();
    const long long tag = 4LL * i;
    for (int a = 0; a < 3; a++)
      for (int p = vptr[ti[a]]; p < vptr[ti[a] + 1]; p++) {
        const int j = vtri[p];
        if (j == i) continue;
        if (shared[j] < tag) {
          shared[j] = tag;
          touch.push_back(j);
        }
        shared[j]++;
      }
    int edges = 0;
    for (int j : touch) {
      const int common = (int)(shared[j] - tag);
      if (common >= 3) return BEM_ERR_DEGENERATE;  // duplicated triangle
      if (common == 2) {
        g.edge_pairs.push_back(make_int2(i, j));
        if (edges < 3) nbr[3 * (size_t)i + edges++] = j;
      } else {
        (i < j ? g.vert_pairs : g.vert_mirror).push_back(make_int2(i, j));
      }
    }
  }

  grow_blocks(g, nbr);
  path_order(g, nbr);

  // 16-triangle tiles with local vertex tables.
  g.ntiles = (nt + kTile - 1) / kTile;
  g.tiles.assign(g.ntiles, TileRec{});
  std::vector<int> stamp(nv, -1), local(nv);
  for (int t = 0; t < g.ntiles; t++) {
    TileRec& tr = g.tiles[t];
    std::memset(&tr, 0, sizeof(TileRec));
    int ntri = std::min(kTile, nt - t * kTile);
    tr.ntri = ntri;
    tr.nlv = local_vertices(g, t * kTile, ntri, 3, 1, t, stamp, local, tr.vid, tr.lv_ptr, tr.lv_corner, tr.corner_lv);
  }
  // the same for the 32-triangle blocks (corner a of triangle t at 32 a + t)
  g.nblocks = (nt + kBlock - 1) / kBlock;
  g.blocks.assign(g.nblocks, BlockRec{});
  for (int t = 0; t < g.nblocks; t++) {
    BlockRec& br = g.blocks[t];
    const int ntri = std::min(kBlock, nt - t * kBlock);
    br.nlv = local_vertices(g, t * kBlock, ntri, 1, kBlock, g.ntiles + t, stamp, local, br.vid, br.ptr, br.corner,
                            nullptr);
    for (int l = 0; l < br.nlv; l++) br.most = std::max(br.most, br.ptr[l + 1] - br.ptr[l]);
  }

  // workspace layout
  GeomHeader& h = g.hdr;
  std::memset(&h, 0, sizeof(h));
  h.magic = kGeomMagic;
  h.nv = nv;
  h.nt = nt;
  h.ntiles = g.ntiles;
  h.n_edge = (int)g.edge_pairs.size();
  h.n_vert = (int)(g.vert_pairs.size() + g.vert_mirror.size());
  h.max_valence = g.max_valence;
  uint64_t off = align_up(sizeof(GeomHeader), 256);
  auto take = [&](uint64_t bytes) {
    uint64_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  // host-built tables first (one upload), device-computed records after
  h.off_vertices = take(sizeof(float) * 3 * (size_t)nv);
  h.off_triangles = take(sizeof(int) * 3 * (size_t)nt);
  h.off_perm = take(sizeof(int) * (size_t)nt);
  h.off_slots = take(sizeof(int) * (size_t)nt);
  h.off_tiles = take(sizeof(TileRec) * (size_t)g.ntiles);
  h.off_blocks = take(sizeof(BlockRec) * (size_t)g.nblocks);
  h.off_edge_pairs = take(sizeof(int2) * (size_t)std::max(1, h.n_edge));
  h.off_vert_pairs = take(sizeof(int2) * (size_t)std::max(1, h.n_vert));
  h.off_trirec = take(sizeof(TriRec) * (size_t)nt);
  h.off_trirec_orig = take(sizeof(TriRec) * (size_t)nt);
  h.off_normals = take(sizeof(float) * 3 * (size_t)nt);
  h.off_curls = take(sizeof(float) * 9 * (size_t)nt);
  h.off_bmrec = take(sizeof(BmRec) * (size_t)nt);
  h.bytes = off;
  return BEM_OK;
}

// FP64 per-triangle records; launched over sorted positions.
__global__ void geom_records_kernel(int nt, const float* __restrict__ verts, const int* __restrict__ tris,
                                    const int* __restrict__ perm, const int* __restrict__ slots,
                                    TriRec* __restrict__ rec_sorted,
                                    TriRec* __restrict__ rec_orig, float* __restrict__ normals,
                                    float* __restrict__ curls, BmRec* __restrict__ bm) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nt) return;
  int i = perm[s];
  int id[3];
  d3 p[3];
  for (int a = 0; a < 3; a++) {
    id[a] = tris[3 * i + a];
    p[a] = {(double)verts[3 * id[a]], (double)verts[3 * id[a] + 1], (double)verts[3 * id[a] + 2]};
  }
  d3 e1 = sub(p[1], p[0]), e2 = sub(p[2], p[0]);
  d3 cr = cross3(e1, e2);
  double J = sqrt(dot3(cr, cr));
  d3 n = {cr.x / J, cr.y / J, cr.z / J};
  TriRec r;
  for (int q = 0; q < 6; q++) {
    double x = 0, y = 0, z = 0;
    for (int b = 0; b < 3; b++) {
      double f = tri6_phi(q, b);
      x += f * p[b].x;
      y += f * p[b].y;
      z += f * p[b].z;
    }
    r.qp[3 * q] = (float)x;
    r.qp[3 * q + 1] = (float)y;
    r.qp[3 * q + 2] = (float)z;
  }
  r.n[0] = (float)n.x;
  r.n[1] = (float)n.y;
  r.n[2] = (float)n.z;
  r.c[0] = (float)((p[0].x + p[1].x + p[2].x) / 3.0);
  r.c[1] = (float)((p[0].y + p[1].y + p[2].y) / 3.0);
  r.c[2] = (float)((p[0].z + p[1].z + p[2].z) / 3.0);
  r.area = (float)(0.5 * J);
  r.v[0] = id[0];
  r.v[1] = id[1];
  r.v[2] = id[2];
  r.h = (float)dot3(n, p[0]);
  r.leave = 0;
  rec_orig[i] = r;
  // the sorted record holds local vertex slot[a] in slot a
  const int code = slots[s];
  const int slot[3] = {code & 3, (code >> 2) & 3, (code >> 4) & 3};
  TriRec rs = r;
  rs.leave = (code >> 8) & 7;
  for (int a = 0; a < 3; a++) {
    rs.v[a] = id[slot[a]];
    for (int c = 0; c < 3; c++) {
      rs.qp[3 * a + c] = r.qp[3 * slot[a] + c];
      rs.qp[9 + 3 * a + c] = r.qp[9 + 3 * slot[a] + c];
    }
  }
  rec_sorted[s] = rs;
  normals[3 * i] = r.n[0];
  normals[3 * i + 1] = r.n[1];
  normals[3 * i + 2] = r.n[2];
  // surface curls n x grad(phi_b) via (J^T J)^-1 (src/bem/solver.py:40-58)
  double g11 = dot3(e1, e1), g12 = dot3(e1, e2), g22 = dot3(e2, e2);
  double det = g11 * g22 - g12 * g12;
  double i11 = g22 / det, i12 = -g12 / det, i22 = g11 / det;
  d3 c1 = {i11 * e1.x + i12 * e2.x, i11 * e1.y + i12 * e2.y, i11 * e1.z + i12 * e2.z};
  d3 c2 = {i12 * e1.x + i22 * e2.x, i12 * e1.y + i22 * e2.y, i12 * e1.z + i22 * e2.z};
  d3 gr[3] = {{-(c1.x + c2.x), -(c1.y + c2.y), -(c1.z + c2.z)}, c1, c2};
  BmRec m;
  for (int b = 0; b < 3; b++) {
    d3 c = cross3(n, gr[b]);
    curls[9 * i + 3 * b] = (float)c.x;
    curls[9 * i + 3 * b + 1] = (float)c.y;
    curls[9 * i + 3 * b + 2] = (float)c.z;
  }
  for (int a = 0; a < 3; a++)
    for (int c = 0; c < 3; c++) m.curl[3 * a + c] = curls[9 * i + 3 * slot[a] + c];
  // 3-point degree-2 rule: point q = 2/3 vertex q + 1/6 (each other vertex)
  for (int q = 0; q < 3; q++) {
    const double own = 2.0 / 3.0 - 1.0 / 6.0, all = 1.0 / 6.0;
    const d3 pq = p[slot[q]];
    m.qp[3 * q] = (float)(all * (p[0].x + p[1].x + p[2].x) + own * pq.x);
    m.qp[3 * q + 1] = (float)(all * (p[0].y + p[1].y + p[2].y) + own * pq.y);
    m.qp[3 * q + 2] = (float)(all * (p[0].z + p[1].z + p[2].z) + own * pq.z);
  }
  m.pad[0] = m.pad[1] = 0.f;
  bm[s] = m;
}

}  // namespace

// Host-side copies of the headers of geometries built in this process, so
// that assembly calls need not read the header back from the device.
static std::mutex g_cache_mu;
static std::unordered_map<const void*, GeomHeader> g_cache;

static void cache_put(const void* geom, const GeomHeader& h) {
  std::lock_guard<std::mutex> lk(g_cache_mu);
  g_cache[geom] = h;
}

static void cache_drop(const void* geom) {
  std::lock_guard<std::mutex> lk(g_cache_mu);
  g_cache.erase(geom);
}

// Reads the header of a built geometry into a device view (host side).  A
// geometry built elsewhere (copied buffer) is read back with a blocking copy.
int geom_view(const void* geom, GeomView* v, GeomHeader* out_hdr) {
  if (!geom) return BEM_ERR_WORKSPACE;
  GeomHeader h;
  bool hit = false;
  {
    std::lock_guard<std::mutex> lk(g_cache_mu);
    auto it = g_cache.find(geom);
    if (it != g_cache.end()) {
      h = it->second;
      hit = true;
    }
  }
  if (!hit) {
    BEM_CUDA_TRY(cudaMemcpy(&h, geom, sizeof(h), cudaMemcpyDeviceToHost));
    if (h.magic == kGeomMagic) cache_put(geom, h);
  }
  if (h.magic != kGeomMagic) return BEM_ERR_WORKSPACE;
  const char* b = (const char*)geom;
  v->nv = h.nv;
  v->nt = h.nt;
  v->ntiles = h.ntiles;
  v->nblocks = (h.nt + kBlock - 1) / kBlock;
  v->n_edge = h.n_edge;
  v->n_vert = h.n_vert;
  v->vertices = (const float*)(b + h.off_vertices);
  v->triangles = (const int*)(b + h.off_triangles);
  v->perm = (const int*)(b + h.off_perm);
  v->slots = (const int*)(b + h.off_slots);
  v->rec = (const TriRec*)(b + h.off_trirec);
  v->rec_orig = (const TriRec*)(b + h.off_trirec_orig);
  v->tiles = (const TileRec*)(b + h.off_tiles);
  v->blocks = (const BlockRec*)(b + h.off_blocks);
  v->edge_pairs = (const int2*)(b + h.off_edge_pairs);
  v->vert_pairs = (const int2*)(b + h.off_vert_pairs);
  v->normals = (const float*)(b + h.off_normals);
  v->curls = (const float*)(b + h.off_curls);
  v->bm = (const BmRec*)(b + h.off_bmrec);
  v->err = (int*)((char*)geom + offsetof(GeomHeader, err));
  if (out_hdr) *out_hdr = h;
  return BEM_OK;
}

}  // namespace bemb

using namespace bemb;

extern "C" int bem_geometry_bytes(const float* vertices, int nv, const int* triangles, int nt, size_t* bytes,
                                  bem_stream_t stream) {
  if (!bytes) return BEM_ERR_INVALID_ARGUMENT;
  const HostGeom* g = nullptr;
  int rc = analyse(vertices, nv, triangles, nt, (cudaStream_t)stream, &g);
  if (rc) return rc;
  *bytes = (size_t)g->hdr.bytes;
  return BEM_OK;
}

extern "C" int bem_geometry_build(const float* vertices, int nv, const int* triangles, int nt, void* geom,
                                  size_t geom_bytes, bem_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const HostGeom* gp = nullptr;
  int rc = analyse(vertices, nv, triangles, nt, s, &gp);
  if (rc) return rc;
  const HostGeom& g = *gp;
  if (!geom || geom_bytes < g.hdr.bytes) return BEM_ERR_WORKSPACE;
  const GeomHeader& h = g.hdr;
  // the integer tables in one pinned staging buffer (kept while the mesh is
  // unchanged), then one upload
  const size_t nstage = h.off_trirec;
  if (!t_stage_ok) {
    if ((rc = t_stage.ensure(nstage))) return rc;
    char* st = t_stage.p;
    std::memset(st, 0, nstage);
    std::memcpy(st, &h, sizeof(h));
    std::memcpy(st + h.off_vertices, g.vertices.data(), sizeof(float) * 3 * (size_t)nv);
    std::memcpy(st + h.off_triangles, g.triangles.data(), sizeof(int) * 3 * (size_t)nt);
    std::memcpy(st + h.off_perm, g.perm.data(), sizeof(int) * (size_t)nt);
    std::memcpy(st + h.off_slots, g.slots.data(), sizeof(int) * (size_t)nt);
    std::memcpy(st + h.off_blocks, g.blocks.data(), sizeof(BlockRec) * (size_t)g.nblocks);
    std::memcpy(st + h.off_tiles, g.tiles.data(), sizeof(TileRec) * (size_t)g.ntiles);
    if (h.n_edge) std::memcpy(st + h.off_edge_pairs, g.edge_pairs.data(), sizeof(int2) * h.n_edge);
    if (h.n_vert) {
      const size_t half = sizeof(int2) * g.vert_pairs.size();
      std::memcpy(st + h.off_vert_pairs, g.vert_pairs.data(), half);
      std::memcpy(st + h.off_vert_pairs + half, g.vert_mirror.data(), sizeof(int2) * g.vert_mirror.size());
    }
    t_stage_ok = true;
  }
  BEM_CUDA_TRY(cudaMemcpyAsync(geom, t_stage.p, nstage, cudaMemcpyHostToDevice, s));
  char* b = (char*)geom;
  (geom_records_kernel<<<(nt + 127) / 128, 128, 0, s>>>(
      nt, (const float*)(b + h.off_vertices), (const int*)(b + h.off_triangles), (const int*)(b + h.off_perm),
      (const int*)(b + h.off_slots), (TriRec*)(b + h.off_trirec), (TriRec*)(b + h.off_trirec_orig), (float*)(b + h.off_normals),
      (float*)(b + h.off_curls), (BmRec*)(b + h.off_bmrec)), count_launch());
  BEM_CUDA_TRY(cudaGetLastError());
  BEM_CUDA_TRY(cudaStreamSynchronize(s));  // the staging buffer serves the next build of this thread
  cache_put(geom, h);
  return BEM_OK;
}

extern "C" int bem_geometry_status(const void* geom, bem_stream_t stream) {
  GeomView v;
  int rc = geom_view(geom, &v, nullptr);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  int err = 0;
  const int zero = 0;
  BEM_CUDA_TRY(cudaMemcpyAsync(&err, v.err, sizeof(int), cudaMemcpyDeviceToHost, s));
  BEM_CUDA_TRY(cudaStreamSynchronize(s));
  if (!err) return BEM_OK;
  BEM_CUDA_TRY(cudaMemcpyAsync(v.err, &zero, sizeof(int), cudaMemcpyHostToDevice, s));
  BEM_CUDA_TRY(cudaStreamSynchronize(s));
  return BEM_ERR_CUDA;
}

extern "C" int bem_geometry_release(const void* geom) {
  if (!geom) return BEM_ERR_INVALID_ARGUMENT;
  cache_drop(geom);
  return BEM_OK;
}

extern "C" int bem_geometry_normals(const void* geom, float* normals, float* curls, bem_stream_t stream) {
  GeomView v;
  int rc = geom_view(geom, &v, nullptr);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  if (normals)
    BEM_CUDA_TRY(cudaMemcpyAsync(normals, v.normals, sizeof(float) * 3 * (size_t)v.nt, cudaMemcpyDeviceToDevice, s));
  if (curls)
    BEM_CUDA_TRY(cudaMemcpyAsync(curls, v.curls, sizeof(float) * 9 * (size_t)v.nt, cudaMemcpyDeviceToDevice, s));
  return BEM_OK;
}
