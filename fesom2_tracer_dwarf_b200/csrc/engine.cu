// Engine: device memory, layout conversion, schedules, batching and
// dispatch to the per-precision kernel units (step_f64.cu, step_f32.cu).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <stdexcept>
#include <string>

#include "advect_fused.cuh"
#include "engine_impl.hpp"

namespace fesom {

namespace {
thread_local std::string g_err;
}
const char *last_error() { return g_err.c_str(); }
void set_last_error(const std::string &s) { g_err = s; }

namespace {

void build_sched(const std::vector<int> &counts, std::vector<int> &off, std::vector<int> &blk, int &max_items,
                 int cells_per_block) {
  const int n = (int)counts.size();
  off.assign(n + 1, 0);
  for (int i = 0; i < n; i++) off[i + 1] = off[i] + counts[i];
  blk.clear();
  blk.push_back(0);
  max_items = 1;
  // cells_per_block is a cap: a block takes whole items while its wet cells
  // stay within it, so that the 256 threads of a block walk its cells in at
  // most cap / 256 rounds (with a target instead, blocks overshooting 512
  // cells by a column gave a third round to a few threads, and the block's
  // time followed them: measured at 1000x1000x64, a 448 target was 6 %
  // faster than a 512 one).  A single item larger than the cap gets a block
  // of its own.
  const int cap = std::min(cells_per_block, kMaxCellsPerBlock);
  int start = 0, cells = 0;
  for (int i = 0; i < n; i++) {
    // close the block before an item that would overflow its capacity
    if (i > start && (cells + counts[i] > cap || i - start >= kMaxItemsPerBlock)) {
      blk.push_back(i);
      max_items = std::max(max_items, i - start);
      start = i;
      cells = 0;
    }
    cells += counts[i];
  }
  if (start < n || n == 0) {
    blk.push_back(n);
    max_items = std::max(max_items, n - start);
  }
  for (size_t b = 0; b + 1 < blk.size(); b++)
    if (off[blk[b + 1]] - off[blk[b]] > kMaxCellsPerBlock)
      throw std::runtime_error("a column or edge has more levels than a block holds");
}

// (ld, ncol) column-major host doubles -> device columns of stride S, type R
template <typename R>
R *upload_cols(EngineImpl &P, const double *h, int ld, int ncol, int nvalid) {
  std::vector<R> st((size_t)ncol * P.S, R(0));
  for (int c = 0; c < ncol; c++)
    for (int k = 0; k < nvalid; k++) st[(size_t)c * P.S + k] = (R)h[(size_t)c * ld + k];
  return P.upload(st);
}
template <typename R>
R *upload_conv(EngineImpl &P, const std::vector<double> &h) {
  std::vector<R> st(h.size());
  for (size_t i = 0; i < h.size(); i++) st[i] = (R)h[i];
  return P.upload(st);
}

// Work schedules (node and edge cells, of the learned flux alone) for a cap on the
// wet cells per block; the arrays of a previous tiling are released.
template <typename R>
void build_schedules(EngineImpl &P, DMeshT<R> &d, int cells_per_block) {
  const MeshHost &M = P.mesh;
  const int N = M.nod2D, E = M.edge2D;
  const std::vector<int> &slot_edge = P.slot_edge;
  for (const void *q : {(const void *)d.node_sched.cell_off, (const void *)d.node_sched.blk,
                        (const void *)d.edge_sched.cell_off, (const void *)d.edge_sched.blk})
    P.dfree(const_cast<void *>(q));
  std::vector<int> cnt(N), off, blk;
  for (int n = 0; n < N; n++) cnt[n] = M.nlev_node[n] - 1;
  build_sched(cnt, off, blk, d.node_sched.max_items, cells_per_block);
  d.node_sched.cell_off = P.upload(off);
  d.node_sched.blk = P.upload(blk);
  d.node_sched.nblk = (int)blk.size() - 1;
  cnt.assign(E, 0);
  for (int s = 0; s < E; s++) cnt[s] = M.edge_levels(slot_edge[s]);
  build_sched(cnt, off, blk, d.edge_sched.max_items, cells_per_block);
  d.edge_sched.cell_off = P.upload(off);
  d.edge_sched.blk = P.upload(blk);
  d.edge_sched.nblk = (int)blk.size() - 1;
}

// ---- records and pair schedules ------------------------------------------------
// Formed on the device from the mesh arrays already there.  On the host, and copied,
// they cost 0.75 of 5.7 s of an engine at 1000x1000x64 (FP64).

int blocks_for(long long threads) { return (int)std::max<long long>(1, std::min<long long>((threads + 255) / 256, 148 * 32)); }

// Levels of an edge whose up and down triangles are both there and wet.
template <typename R>
__device__ __forceinline__ int edge_tri_levels(const DMeshT<R> &m, int s) {
  const int2 ud = m.up_dn[s], nn = m.edge_nodes[s];
  if (ud.x < 0 || ud.y < 0) return 0;
  return max(0, min(m.nlev_node_min[nn.x], m.nlev_node_min[nn.y]) - 1);
}

// Per-edge records of k_edge (DMeshT::edge_idx, edge_geo).
template <typename R>
__global__ void k_edge_records(DMeshT<R> m, int4 *idx, R *geo) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.E; s += gridDim.x * blockDim.x) {
    const int2 nn = m.edge_nodes[s], ud = m.up_dn[s];
    const bool pair = ud.x >= 0 && ud.y >= 0;
    int un[3] = {nn.x, nn.x, nn.x}, dn[3] = {nn.y, nn.y, nn.y};
    R *g = geo + 16 * (size_t)s;
    for (int q = 0; q < 16; q++) g[q] = R(0);
    if (pair) {
      for (int q = 0; q < 3; q++) {
        un[q] = m.elem_nodes[3 * (size_t)ud.x + q];
        dn[q] = m.elem_nodes[3 * (size_t)ud.y + q];
      }
      for (int q = 0; q < 6; q++) {
        g[q] = m.grad_sca[6 * (size_t)ud.x + q];
        g[6 + q] = m.grad_sca[6 * (size_t)ud.y + q];
      }
    }
    g[12] = m.edge_dxdy[2 * (size_t)s] * m.edge_a[s];
    g[13] = m.edge_dxdy[2 * (size_t)s + 1] * (R)kREarthD;
    idx[3 * (size_t)s] = make_int4(nn.x * m.S, nn.y * m.S, un[0] * m.S, un[1] * m.S);
    idx[3 * (size_t)s + 1] = make_int4(un[2] * m.S, dn[0] * m.S, dn[1] * m.S, dn[2] * m.S);
    idx[3 * (size_t)s + 2] = make_int4(edge_tri_levels(m, s), m.nbl[nn.x], m.nbl[nn.y], m.edge_lev[s].y);
  }
}

// Element records of the ring means (DMeshT::elem_idx, elem_geo).
template <typename R>
__global__ void k_elem_records(DMeshT<R> m, int4 *idx, R *geo) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m.T; e += gridDim.x * blockDim.x) {
    const int *en = m.elem_nodes + 3 * (size_t)e;
    R *g = geo + 8 * (size_t)e;
    idx[e] = make_int4(en[0] * m.S, en[1] * m.S, en[2] * m.S, m.nlev_elem[e] - 1);
    for (int q = 0; q < 6; q++) g[q] = m.grad_sca[6 * (size_t)e + q];
    g[6] = m.elem_area[e];
    g[7] = R(0);
  }
}

// Node records of the column kernels (DMeshT::nrec, ne6); holds: elements of each node
template <typename R>
__global__ void k_holds(DMeshT<R> m, int *holds) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 3ll * m.T; i += (long long)gridDim.x * blockDim.x)
    atomicAdd(&holds[m.elem_nodes[i]], 1);
}
template <typename R>
__global__ void k_node_records(DMeshT<R> m, const int *holds, int4 *rec, int4 *ne) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < m.N; n += gridDim.x * blockDim.x) {
    const int p0 = m.ne_ptr[n], deg = m.ne_ptr[n + 1] - p0;
    const bool full = m.ring_ptr[n + 1] - m.ring_ptr[n] == holds[n];
    unsigned lev[2] = {0, 0}, r[12];
    for (int i = 0; i < 6; i++) {
      r[2 * i] = 0;
      r[2 * i + 1] = (unsigned)n * (unsigned)m.S;
      if (i >= deg) continue;
      const int4 q = m.ne4[p0 + i];
      r[2 * i] = (unsigned)(q.x >> 1) * (unsigned)m.S;
      r[2 * i + 1] = (unsigned)q.w | (unsigned)(q.x & 1) << 31;
      lev[i / 3] |= (unsigned)q.z << (10 * (i % 3));
    }
    rec[n] = make_int4(m.nlev_node[n] | deg << 16, (int)((unsigned)m.nlev_node_min[n] | (full ? 0x80000000u : 0u)), (int)lev[0],
                       (int)lev[1]);
    for (int i = 0; i < 3; i++)
      ne[3 * (size_t)n + i] = make_int4((int)r[4 * i], (int)r[4 * i + 1], (int)r[4 * i + 2], (int)r[4 * i + 3]);
  }
}

template <typename R>
void build_records(EngineImpl &P, DMeshT<R> &d) {
  const MeshHost &M = P.mesh;
  for (int n = 0; n < M.nod2D; n++)
    if (M.node_edge_ptr[n + 1] - M.node_edge_ptr[n] > 0xffff) throw std::invalid_argument("a node has more than 65535 edges");
  int4 *eidx = P.dalloc<int4>(3 * (size_t)d.E), *tidx = P.dalloc<int4>(d.T), *nrec = P.dalloc<int4>(d.N),
       *ne6 = P.dalloc<int4>(3 * (size_t)d.N);
  R *egeo = P.dalloc<R>(16 * (size_t)d.E), *tgeo = P.dalloc<R>(8 * (size_t)d.T);
  int *holds = P.dalloc<int>(d.N);
  k_edge_records<R><<<blocks_for(d.E), 256, 0, P.stream>>>(d, eidx, egeo);
  k_elem_records<R><<<blocks_for(d.T), 256, 0, P.stream>>>(d, tidx, tgeo);
  k_holds<R><<<blocks_for(3ll * d.T), 256, 0, P.stream>>>(d, holds);
  k_node_records<R><<<blocks_for(d.N), 256, 0, P.stream>>>(d, holds, nrec, ne6);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(P.stream));
  P.dfree(holds);
  P.bytes -= (size_t)d.N * sizeof(int);
  d.edge_idx = eidx;
  d.edge_geo = egeo;
  d.elem_idx = tidx;
  d.elem_geo = tgeo;
  d.nrec = nrec;
  d.ne6 = ne6;
}

// A schedule's arrays on the device: every lane without a pair, of item 0, until it
// is filled.
struct PairArrays {
  int *item;
  unsigned short *lev;
  PairArrays(EngineImpl &P, long long entries) {
    item = P.dalloc<int>(entries);
    lev = P.dalloc<unsigned short>(entries);
    if (entries) CK(cudaMemsetAsync(lev, 0xff, entries * sizeof(unsigned short), P.stream));
  }
  DPairs pairs(long long entries) const { return DPairs{item, lev, (int)(entries / 32)}; }
};

// Pair schedule of the edges, run by run of slots: the pairs with both triangles
// at every wet level, then the others.  A block takes a run: with `base` null it counts
// the pairs of both kinds, otherwise it writes them from base[2 run], base[2 run + 1].
constexpr int kPairRun = 2048, kPairThreads = 256, kPairEach = kPairRun / kPairThreads;
template <typename R>
__global__ void __launch_bounds__(kPairThreads) k_edge_pairs(DMeshT<R> m, const int *base, int *count, int *item,
                                                            unsigned short *lev) {
  __shared__ int off[kPairRun], part[kPairThreads];
  const int s0 = blockIdx.x * kPairRun, ns = min(m.E - s0, kPairRun), tid = threadIdx.x;
  // pairs of edge s with both triangles at every wet level, and the others
  auto pairs = [&](int s, int kind) {
    const int nl = m.edge_lev[s].y, tri = edge_tri_levels(m, s), all = (nl + 1) / 2, both = tri >= nl ? all : tri / 2;
    return kind == 0 ? both : all - both;
  };
  for (int kind = 0; kind < 2; kind++) {
    int c[kPairEach], sum = 0;
    for (int i = 0; i < kPairEach; i++) {
      const int j = tid * kPairEach + i;
      c[i] = j < ns ? pairs(s0 + j, kind) : 0;
      sum += c[i];
    }
    part[tid] = sum;
    __syncthreads();
    for (int w = 1; w < kPairThreads; w *= 2) {  // inclusive sums
      const int v = tid >= w ? part[tid - w] : 0;
      __syncthreads();
      part[tid] += v;
      __syncthreads();
    }
    const int total = part[kPairThreads - 1];
    if (!base) {
      if (tid == 0) count[2 * blockIdx.x + kind] = total;
      __syncthreads();
      continue;
    }
    int o = part[tid] - sum;
    for (int i = 0; i < kPairEach; i++) {
      off[tid * kPairEach + i] = o;
      o += c[i];
    }
    __syncthreads();
    const size_t b = base[2 * blockIdx.x + kind];
    for (int j = tid / 32; j < ns; j += kPairThreads / 32) {
      const int n = (j + 1 < ns ? off[j + 1] : total) - off[j], all = (m.edge_lev[s0 + j].y + 1) / 2;
      const int first = kind == 0 ? 0 : all - n;
      for (int q = tid % 32; q < n; q += 32) {
        item[b + off[j] + q] = s0 + j;
        lev[b + off[j] + q] = (unsigned short)((kind ? kPairRing : 0u) | (unsigned)(2 * (first + q)));
      }
    }
    // lanes without a pair hold the run's last edge
    if (total > 0 && tid < (32 - total % 32) % 32) item[b + total + tid] = s0 + ns - 1;
    __syncthreads();
  }
}
template <typename R>
DPairs build_edge_pairs(EngineImpl &P, const DMeshT<R> &d) {
  const int runs = (d.E + kPairRun - 1) / kPairRun;
  if (runs == 0) return DPairs{};
  int *dev = P.dalloc<int>(2 * (size_t)runs);
  std::vector<int> n(2 * (size_t)runs);
  k_edge_pairs<R><<<runs, kPairThreads, 0, P.stream>>>(d, nullptr, dev, nullptr, nullptr);
  CK(cudaGetLastError());
  P.d2h(n.data(), dev, n.size() * sizeof(int));
  long long total = 0;
  for (int &x : n) {
    const int c = (x + 31) / 32 * 32;
    x = (int)total;
    total += c;
  }
  const PairArrays a(P, total);
  P.h2d(dev, n.data(), n.size() * sizeof(int));
  k_edge_pairs<R><<<runs, kPairThreads, 0, P.stream>>>(d, dev, nullptr, a.item, a.lev);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(P.stream));
  P.dfree(dev);
  P.bytes -= n.size() * sizeof(int);
  return a.pairs(total);
}

// Pair schedule of the ring-mean gradients: an edge uses its nodes' ring means from
// level edge_tri_levels down.  first: each node's first such level.
template <typename R>
__global__ void k_grad_first(DMeshT<R> m, int *first) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < m.E; s += gridDim.x * blockDim.x) {
    const int2 nn = m.edge_nodes[s];
    const int tri = edge_tri_levels(m, s);
    atomicMin(&first[nn.x], tri);
    atomicMin(&first[nn.y], tri);
  }
}
__global__ void k_grad_pairs(int N, const int *first, const int *off, int *item, unsigned short *lev) {
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x)
    for (int i = off[n]; i < off[n + 1]; i++) {
      item[i] = n;
      lev[i] = (unsigned short)(first[n] / 2 * 2 + 2 * (i - off[n]));
    }
}
template <typename R>
DPairs build_grad_pairs(EngineImpl &P, const DMeshT<R> &d) {
  const MeshHost &M = P.mesh;
  const int N = M.nod2D;
  std::vector<int> first(N), off(N + 1, 0);
  for (int n = 0; n < N; n++) first[n] = std::max(0, M.nlev_node[n] - 1);
  int *df = P.upload(first);
  k_grad_first<R><<<blocks_for(d.E), 256, 0, P.stream>>>(d, df);
  CK(cudaGetLastError());
  P.d2h(first.data(), df, (size_t)N * sizeof(int));
  long long total = 0;
  for (int n = 0; n < N; n++) {
    const int last = M.nlev_node[n] - 1;
    if (first[n] < last) total += (last - first[n] / 2 * 2 + 1) / 2;
    off[n + 1] = (int)total;
  }
  total = (total + 31) / 32 * 32;
  const PairArrays a(P, total);
  int *doff = P.upload(off);
  k_grad_pairs<<<blocks_for(N), 256, 0, P.stream>>>(N, df, doff, a.item, a.lev);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(P.stream));
  P.dfree(df);
  P.dfree(doff);
  P.bytes -= (2 * (size_t)N + 1) * sizeof(int);
  return a.pairs(total);
}

// Pair schedule of the columns.  A warp takes whole columns, so that their
// vertical neighbours are the lanes beside; within a window of nodes they are
// placed largest first into the fullest warp that still holds them (windows of 32
// and 64 nodes leave more lanes idle: k_col1 5-10 % slower; a Morton order of the
// nodes instead of their own was slower too).  Columns
// of more than 32 pairs are cut into pieces that overlap by one pair at each cut
// (halo lanes: computed, not stored).
//
// A piece as the device fills it in: x node, y first entry, z first pair | pairs << 16,
// w 1: its first pair is a halo, 2: its last, 4: nothing follows it in its warp.
__global__ void k_node_pairs(int npieces, const int4 *pieces, int *item, unsigned short *lev) {
  const int lane = threadIdx.x & 31;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < npieces; i += (gridDim.x * blockDim.x) >> 5) {
    const int4 c = pieces[i];
    const int first = c.z & 0xffff, n = c.z >> 16, e = c.y + lane;
    if (lane < n) {
      const bool halo = ((c.w & 1) && lane == 0) || ((c.w & 2) && lane == n - 1);
      item[e] = c.x;
      lev[e] = (unsigned short)((halo ? kPairHalo : 0u) | (unsigned)(2 * (first + lane)));
    } else if ((c.w & 4) && e / 32 == c.y / 32) {
      item[e] = c.x;  // lanes without a pair
    }
  }
}
DPairs build_node_pairs(EngineImpl &P) {
  const MeshHost &M = P.mesh;
  const int N = M.nod2D, window = 256;
  std::vector<int4> pieces;  // in the order of the entries
  pieces.reserve(N);
  long long warps = 0;
  // one window: its pieces by length, the pieces of each warp, and the warps by free lanes
  struct Piece {
    int node, first, n, halo, next;
  };
  std::vector<Piece> w;
  std::vector<int> by_n[33], open[33], head, tail;
  for (int n0 = 0; n0 < N; n0 += window) {
    w.clear();
    head.clear();
    tail.clear();
    for (int i = 0; i <= 32; i++) {
      by_n[i].clear();
      open[i].clear();
    }
    for (int n = n0; n < std::min(N, n0 + window); n++) {
      const int np = M.nlev_node[n] / 2;  // pairs of nlev - 1 layers
      for (int p = 0; p < np;) {
        const bool lo = p > 0;
        const int left = np - p + (lo ? 1 : 0);  // with the leading halo
        const bool hi = left > 32;
        const Piece c{n, lo ? p - 1 : 0, std::min(left, 32), (lo ? 1 : 0) | (hi ? 2 : 0), -1};
        p = c.first + c.n - (hi ? 1 : 0);
        by_n[c.n].push_back((int)w.size());
        w.push_back(c);
      }
    }
    for (int n = 32; n >= 1; n--)
      for (int i : by_n[n]) {
        int r = n;
        while (r <= 32 && open[r].empty()) r++;
        int k;
        if (r > 32) {
          k = (int)head.size();
          head.push_back(i);
          tail.push_back(i);
          r = 32;
        } else {
          k = open[r].back();
          open[r].pop_back();
          w[tail[k]].next = i;
          tail[k] = i;
        }
        if (r - n > 0) open[r - n].push_back(k);
      }
    for (size_t k = 0; k < head.size(); k++) {
      int e = (int)(32 * (warps + (long long)k));
      for (int i = head[k]; i >= 0; i = w[i].next) {
        pieces.push_back(make_int4(w[i].node, e, w[i].first | w[i].n << 16, w[i].halo | (w[i].next < 0 ? 4 : 0)));
        e += w[i].n;
      }
    }
    warps += (long long)head.size();
  }
  const PairArrays a(P, 32 * warps);
  int4 *dp = P.upload(pieces);
  k_node_pairs<<<blocks_for(32ll * (long long)pieces.size()), 256, 0, P.stream>>>((int)pieces.size(), dp, a.item, a.lev);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(P.stream));
  P.dfree(dp);
  P.bytes -= pieces.size() * sizeof(int4);
  return a.pairs(32 * warps);
}

template <typename R>
void build_dmesh(EngineImpl &P, DMeshT<R> &d, const std::vector<int> &slot_edge, const std::vector<int> &edge_slot) {
  const MeshHost &M = P.mesh;
  const int N = M.nod2D, T = M.elem2D, E = M.edge2D, nl = M.nl, L = nl - 1;
  d.N = N; d.T = T; d.E = E; d.nl = nl; d.S = P.S;
  std::vector<int2> en(E), et(E), el(E), ud(E);
  std::vector<double> ecross(4 * (size_t)E), edxdy(2 * (size_t)E), ea(E);
  for (int n = 0; n < N; n++)
    if (M.nlev_node[n] - 1 > kMaxCellsPerBlock) throw std::runtime_error("a column or edge has more levels than a block holds");
  for (int s = 0; s < E; s++) {
    const int e = slot_edge[s];
    en[s] = make_int2(M.edge_nodes[2 * e], M.edge_nodes[2 * e + 1]);
    et[s] = make_int2(M.edge_tri[2 * e], M.edge_tri[2 * e + 1]);
    el[s] = make_int2(M.edge_shared_levels(e), M.edge_levels(e));
    ud[s] = make_int2(M.up_dn_tri[2 * e], M.up_dn_tri[2 * e + 1]);
    for (int q = 0; q < 4; q++) ecross[4 * (size_t)s + q] = M.edge_cross[4 * (size_t)e + q];
    for (int q = 0; q < 2; q++) edxdy[2 * (size_t)s + q] = M.edge_dxdy[2 * (size_t)e + q];
    ea[s] = M.edge_a[e];
  }
  d.edge_nodes = P.upload(en);
  d.edge_tri = P.upload(et);
  d.edge_lev = P.upload(el);
  d.up_dn = P.upload(ud);
  d.edge_cross = upload_conv<R>(P, ecross);
  d.edge_dxdy = upload_conv<R>(P, edxdy);
  d.edge_a = upload_conv<R>(P, ea);
  d.nlev_elem = P.upload(M.nlev_elem);
  d.nlev_node = P.upload(M.nlev_node);
  d.nlev_node_min = P.upload(M.nlev_node_min);
  d.nbl = P.upload(M.nboundary_lay);
  d.elem_nodes = P.upload(M.elem_nodes);
  d.grad_sca = upload_conv<R>(P, M.grad_sca);
  d.elem_area = upload_conv<R>(P, M.elem_area);
  d.ring_ptr = P.upload(M.ring_ptr);
  d.ring_elem = P.upload(M.ring_elem);
  d.ne_ptr = P.upload(M.node_edge_ptr);
  {
    std::vector<int4> ne4(M.node_edge.size());
    for (int n = 0; n < N; n++)
      for (int p = M.node_edge_ptr[n]; p < M.node_edge_ptr[n + 1]; p++) {
        const int code = M.node_edge[p], e = code >> 1, second = code & 1;
        const int other = M.edge_nodes[2 * e + (second ? 0 : 1)];
        ne4[p] = make_int4((edge_slot[e] << 1) | second, other, M.edge_levels(e), other * P.S);
      }
    d.ne4 = P.upload(ne4);
  }
  d.zbar = upload_conv<R>(P, M.zbar);
  d.Z = upload_conv<R>(P, M.Z);
  d.area = upload_cols<R>(P, M.area.data(), nl, N, nl);
  d.areasvol = upload_cols<R>(P, M.areasvol.data(), nl, N, nl);
  d.hnode = upload_cols<R>(P, M.hnode.data(), L, N, L);
  d.hnode_new = upload_cols<R>(P, M.hnode_new.data(), L, N, L);
  d.helem = upload_cols<R>(P, M.helem.data(), L, T, L);

  build_records(P, d);
  d.edge_pairs = build_edge_pairs(P, d);
  d.grad_pairs = build_grad_pairs(P, d);
  d.node_pairs = build_node_pairs(P);
}

// Patch plan of the fused step kernel: built on the host, uploaded, host
// lists released (the maxima stay for the shared-memory layout).
void build_tiles(EngineImpl &P, const std::vector<int> &edge_slot, int owned) {
  for (const void *q : {(const void *)P.tiles.cnt, (const void *)P.tiles.node_gid, (const void *)P.tiles.node_info,
                        (const void *)P.tiles.inc_ptr, (const void *)P.tiles.inc, (const void *)P.tiles.edge_slot,
                        (const void *)P.tiles.edge_nn, (const void *)P.tiles.edge_ud, (const void *)P.tiles.elem_gid,
                        (const void *)P.tiles.elem_nn, (const void *)P.tiles.ring_ptr, (const void *)P.tiles.ring})
    P.dfree(const_cast<void *>(q));
  P.tiles = DTiles{};
  P.tplan = TilePlanHost();
  if (P.mesh.nod2D <= 0 || P.mesh.nl > kTileMaxLevels) return;
  TilePlanHost &t = P.tplan;
  try {
    t = build_tile_plan(P.mesh, edge_slot, owned);
  } catch (const std::exception &) {
    t = TilePlanHost();  // no plan: the five-kernel path runs every scheme
    return;
  }
  DTiles &d = P.tiles;
  d.cnt = P.upload(t.cnt);
  d.node_gid = P.upload(t.node_gid);
  d.node_info = P.upload(t.node_info);
  d.inc_ptr = P.upload(t.inc_ptr);
  d.inc = P.upload(t.inc);
  d.edge_slot = P.upload(t.edge_slot);
  d.edge_nn = P.upload(t.edge_nn);
  d.edge_ud = P.upload(t.edge_ud);
  d.elem_gid = P.upload(t.elem_gid);
  d.elem_nn = P.upload(t.elem_nn);
  d.ring_ptr = P.upload(t.ring_ptr);
  d.ring = P.upload(t.ring);
  d.np = t.np;
  for (auto *v : {&t.node_gid, &t.inc_ptr, &t.edge_slot, &t.elem_gid, &t.ring_ptr}) std::vector<int>().swap(*v);
  for (auto *v : {&t.node_info, &t.inc, &t.edge_nn, &t.edge_ud, &t.elem_nn}) std::vector<uint32_t>().swap(*v);
  std::vector<uint16_t>().swap(t.ring);
  std::vector<TileCounts>().swap(t.cnt);
}

}  // namespace

static_assert(Engine::kDefaultCellsPerBlock == kCellsPerBlock, "one default schedule tile");

void learned_schedules(EngineImpl &P) {
  build_schedules(P, P.dm32, P.cells_per_block);
}

std::vector<int> edge_slot_order(const MeshHost &M) {
  // slot order: edges sorted by their smaller node id (stable in edge id)
  const int E = M.edge2D;
  std::vector<int> slot_edge(E), edge_slot(E);
  for (int e = 0; e < E; e++) slot_edge[e] = e;
  std::stable_sort(slot_edge.begin(), slot_edge.end(), [&](int a, int b) {
    return std::min(M.edge_nodes[2 * a], M.edge_nodes[2 * a + 1]) < std::min(M.edge_nodes[2 * b], M.edge_nodes[2 * b + 1]);
  });
  for (int s = 0; s < E; s++) edge_slot[slot_edge[s]] = s;
  return edge_slot;
}

Engine::Engine(const MeshHost &mesh, Precision prec) : p_(new EngineImpl) {
  EngineImpl &P = *p_;
  P.mesh = mesh;
  P.prec = prec;
  P.r_bytes = prec == Precision::FP64 ? 8 : 4;
  P.ts_bytes = prec == Precision::FP64 ? 8 : (prec == Precision::FP32 ? 4 : 2);
  const std::string bad = mesh.validate();
  if (!bad.empty()) throw std::invalid_argument("mesh: " + bad);
  const MeshHost &M = P.mesh;
  const int E = M.edge2D;
  // level stride: 32-byte aligned columns for FP64, 16-byte aligned ones (or
  // better) for the 4- and 2-byte types
  P.S = prec == Precision::FP64 ? (M.nl + 3) / 4 * 4 : (M.nl + 7) / 8 * 8;
  // the kernels index cells with 32-bit offsets (node column bases as int)
  if ((long long)M.nod2D * P.S >= (1ll << 31) || (long long)M.edge2D * P.S >= (1ll << 32))
    throw std::invalid_argument("mesh too large: nodes x level stride must stay below 2^31 and edges x level stride "
                                "below 2^32");
  CK(cudaGetDevice(&P.device));
  CK(cudaStreamCreateWithFlags(&P.stream, cudaStreamNonBlocking));
  const std::vector<int> edge_slot = edge_slot_order(M);
  std::vector<int> slot_edge(E);
  for (int e = 0; e < E; e++) slot_edge[edge_slot[e]] = e;
  P.slot_edge = slot_edge;
  if (prec == Precision::FP64) {
    build_dmesh<double>(P, P.dm64, slot_edge, edge_slot);
    build_rcp_f64(P);
  } else {
    build_dmesh<float>(P, P.dm32, slot_edge, edge_slot);
    build_rcp_f32(P);
  }
  build_tiles(P, edge_slot, kTileOwned);
  P.nonfinite_d = P.dalloc<unsigned long long>(1);
  P.vel = P.dalloc_bytes((size_t)2 * M.elem2D * P.S * P.r_bytes);
  P.W = P.dalloc_bytes((size_t)M.nod2D * P.S * P.r_bytes);
  CK(cudaStreamSynchronize(P.stream));
}

Engine::~Engine() {
  if (!p_) return;
  cudaStreamSynchronize(p_->stream);
  if (p_->io_h2d) {
    cudaStreamSynchronize(p_->io_h2d);
    cudaStreamSynchronize(p_->io_d2h);
    cudaStreamDestroy(p_->io_h2d);
    cudaStreamDestroy(p_->io_d2h);
  }
  for (cudaEvent_t e : p_->io_ev_in) cudaEventDestroy(e);
  for (cudaEvent_t e : p_->io_ev_out) cudaEventDestroy(e);
  release_ring(*p_);
  learned_release(*p_);
  for (void *a : p_->allocs) cudaFree(a);
  cudaStreamDestroy(p_->stream);
  delete p_;
}

const MeshHost &Engine::mesh() const { return p_->mesh; }
EngineImpl *Engine::impl() { return p_; }

void Engine::set_cells_per_block(int cells) {
  EngineImpl &P = *p_;
  if (cells < 32 || cells > kMaxCellsPerBlock) throw std::invalid_argument("cells per block must be in [32, 576]");
  CK(cudaStreamSynchronize(P.stream));
  P.cells_per_block = cells;
  if (P.learn) learned_schedules(P);  // otherwise set_learned builds them
}
int Engine::cells_per_block() const { return p_->cells_per_block; }
int Engine::level_stride() const { return p_->S; }
Precision Engine::precision() const { return p_->prec; }
void *Engine::stream() const { return (void *)p_->stream; }
int Engine::device() const { return p_->device; }
void Engine::set_fma64(bool on) { p_->fma64 = on; }
long long Engine::nonfinite_values(bool reset) {
  EngineImpl &P = *p_;
  unsigned long long n = 0;
  P.d2h(&n, P.nonfinite_d, sizeof(n));
  if (reset && n) {
    CK(cudaMemsetAsync(P.nonfinite_d, 0, sizeof(n), P.stream));
    CK(cudaStreamSynchronize(P.stream));
  }
  return (long long)n;
}
bool Engine::fma64() const { return p_->fma64; }
void Engine::synchronize() const { CK(cudaStreamSynchronize(p_->stream)); }
size_t Engine::device_bytes() const { return p_->bytes; }
int Engine::num_tracers() const { return (int)p_->tr.size(); }

void Engine::set_velocity(const double *uv, const double *w) {
  EngineImpl &P = *p_;
  P.vflux_valid = false;
  const MeshHost &M = P.mesh;
  const int L = M.nl - 1, T = M.elem2D, N = M.nod2D;
  std::vector<double> st((size_t)2 * T * P.S, 0.0), wst((size_t)N * P.S, 0.0);
  for (int e = 0; e < T; e++)
    for (int k = 0; k < L; k++) {
      st[2 * ((size_t)e * P.S + k)] = uv[2 * ((size_t)e * L + k)];
      st[2 * ((size_t)e * P.S + k) + 1] = uv[2 * ((size_t)e * L + k) + 1];
    }
  for (int n = 0; n < N; n++) std::memcpy(&wst[(size_t)n * P.S], w + (size_t)n * M.nl, sizeof(double) * M.nl);
  if (P.prec == Precision::FP64) {
    P.h2d(P.vel, st.data(), st.size() * sizeof(double));
    P.h2d(P.W, wst.data(), wst.size() * sizeof(double));
  } else {
    std::vector<float> f(st.begin(), st.end()), fw(wst.begin(), wst.end());
    P.h2d(P.vel, f.data(), f.size() * sizeof(float));
    P.h2d(P.W, fw.data(), fw.size() * sizeof(float));
  }
}

void Engine::set_velocity_zero() {
  EngineImpl &P = *p_;
  P.vflux_valid = false;
  CK(cudaMemsetAsync(P.vel, 0, P.r_bytes * 2 * P.mesh.elem2D * P.S, P.stream));
  CK(cudaMemsetAsync(P.W, 0, P.r_bytes * P.mesh.nod2D * P.S, P.stream));
  CK(cudaStreamSynchronize(P.stream));
}

void Engine::allocate_tracers(int ntr, bool with_ab) {
  EngineImpl &P = *p_;
  CK(cudaStreamSynchronize(P.stream));
  for (auto &t : P.tr) { P.dfree(t.T); P.dfree(t.Tout); P.dfree(t.TAB); }
  P.tr.assign(ntr, EngineImpl::Tracer{});
  const size_t n = (size_t)P.mesh.nod2D * P.S * P.ts_bytes;
  for (auto &t : P.tr) {
    t.T = P.dalloc_bytes(n);
    t.Tout = P.dalloc_bytes(n);
    t.TAB = with_ab ? P.dalloc_bytes(n) : nullptr;
  }
  CK(cudaStreamSynchronize(P.stream));
}

void Engine::release_work() {
  EngineImpl &P = *p_;
  CK(cudaStreamSynchronize(P.stream));
  for (void **q : {&P.adfh, &P.lo, &P.adfv}) {
    P.dfree(*q);
    *q = nullptr;
  }
  for (int t = 0; t < P.slots; t++) {
    for (void **q : {&P.rpm[t], &P.gradn[t]}) {
      P.dfree(*q);
      *q = nullptr;
    }
  }
  P.dfree(P.vflux);
  P.vflux = nullptr;
  P.vflux_valid = false;
  P.slots = 0;
}

static void check_id(const EngineImpl &P, int id) {
  if (id < 0 || id >= (int)P.tr.size()) throw std::out_of_range("invalid tracer id " + std::to_string(id + 1));
}

static bool storage16(const EngineImpl &P) { return P.prec == Precision::BF16 || P.prec == Precision::FP16; }

void Engine::set_values(int id, const double *v, bool also_ab) {
  EngineImpl &P = *p_;
  check_id(P, id);
  CK(cudaStreamSynchronize(P.stream));
  auto &tr = P.tr[id];
  stage_upload(P, v);
  // 16-bit storage offset: the wet-cell mean of this upload, rounded to FP32
  double off = 0.0;
  if (storage16(P)) {
    off = (double)(float)stage_wet_mean(P);
    if (!std::isfinite(off)) off = 0.0;
  }
  if (!also_ab && off != tr.off) storage_reoffset(P, tr.TAB, tr.off, off);  // valuesAB stays
  tr.off = off;
  stage_pack(P, off, tr.T, also_ab ? tr.TAB : nullptr, tr.Tout);
  CK(cudaStreamSynchronize(P.stream));
}

void Engine::set_values_ab(int id, const double *v) {
  EngineImpl &P = *p_;
  check_id(P, id);
  CK(cudaStreamSynchronize(P.stream));
  if (!P.tr[id].TAB) throw std::invalid_argument("tracer has no valuesAB array (valuesAB := values each step)");
  stage_upload(P, v);
  stage_pack(P, P.tr[id].off, P.tr[id].TAB, nullptr, nullptr);
  CK(cudaStreamSynchronize(P.stream));
}

void Engine::get_values(int id, double *out) const {
  EngineImpl &P = *p_;
  check_id(P, id);
  CK(cudaStreamSynchronize(P.stream));
  stage_unpack(P, P.tr[id].T, P.tr[id].off);
  stage_download(P, out);
}

void Engine::get_values_ab(int id, double *out) const {
  EngineImpl &P = *p_;
  check_id(P, id);
  CK(cudaStreamSynchronize(P.stream));
  stage_unpack(P, P.tr[id].TAB ? P.tr[id].TAB : P.tr[id].T, P.tr[id].off);
  stage_download(P, out);
}

void Engine::set_rounding(int mode) {
  if (mode < 0 || mode > 1) throw std::invalid_argument("rounding mode must be 0 (nearest) or 1 (stochastic)");
  p_->sround = mode;
}
int Engine::rounding() const { return p_->sround; }
double Engine::storage_offset(int id) const {
  check_id(*p_, id);
  return p_->tr[id].off;
}

// host copy of the kernels' mix32 (lowbias32)
static uint32_t mix32_host(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

void Engine::set_scheme(int id, const TracerScheme &s) {
  check_id(*p_, id);
  if (s.hor < 0 || s.hor > 2 || s.ver < 0 || s.ver > 3 || s.lim < 0 || s.lim > 1)
    throw std::invalid_argument("unknown advection scheme");
  p_->tr[id].sch = s;
}
TracerScheme Engine::scheme(int id) const {
  check_id(*p_, id);
  return p_->tr[id].sch;
}

static void ensure_slots(EngineImpl &P, int n) {
  if (n <= P.slots) return;
  const size_t ns = (size_t)P.mesh.nod2D * P.S * P.r_bytes, es = (size_t)P.mesh.edge2D * P.S * P.r_bytes;
  if (!P.vflux) P.vflux = P.dalloc_bytes(es);
  // adf_h, lo and adf_v hold a batch's tracers side by side: one array each,
  // reallocated for the larger batch
  CK(cudaStreamSynchronize(P.stream));
  P.dfree(P.adfh);
  P.dfree(P.lo);
  P.dfree(P.adfv);
  P.adfh = P.dalloc_bytes(n * es);
  P.lo = P.dalloc_bytes(n * ns);
  P.adfv = P.dalloc_bytes(n * ns);
  for (int t = P.slots; t < n; t++) {
    P.rpm[t] = P.dalloc_bytes(2 * ns);
    P.gradn[t] = P.dalloc_bytes(2 * ns);
  }
  P.slots = n;
}

bool fused_step(const EngineImpl &P, const TracerScheme &sc, bool learned) {
  if (P.step_path != 0 || P.tiles.np <= 0 || learned) return false;
  if (P.prec != Precision::FP64 && P.prec != Precision::FP32) return false;
  if (sc.ver != 0 && sc.ver != 1) return false;  // QR4C and CDIFF: five-kernel path
  const TileLayout L = tile_layout(P.tplan, (unsigned)P.r_bytes, false, sc.hor != 0, sc.lim == 1);
  return L.bytes <= (unsigned)kTileSmemMax;
}

static void dispatch(EngineImpl &P, const TracerScheme &sc, int nt, const BatchPtrs &b, double dt) {
  if (P.mesh.nod2D <= 0) return;
  if (P.prec == Precision::FP64) (P.fma64 ? launch_batch_f64fma : launch_batch_f64)(P, sc, nt, b, dt);
  else launch_batch_f32(P, sc, nt, b, dt);
  CK(cudaGetLastError());
}

// Tracers are advanced in batches of up to kBatchMax consecutive tracers with
// the same scheme; a batch shares the edge volume fluxes, the geometry loads
// and every geometry-only division.
static void run_batch(EngineImpl &P, int first, int nt, double dt, bool refresh_ab) {
  ensure_slots(P, nt);
  BatchPtrs b;
  for (int t = 0; t < nt; t++) {
    auto &tr = P.tr[first + t];
    b.T[t] = tr.T;
    if (!refresh_ab && !tr.TAB) throw std::invalid_argument("tracer has no valuesAB array: advance with valuesAB := values");
    b.TAB[t] = refresh_ab ? tr.T : tr.TAB;
    b.T_out[t] = tr.Tout;
    b.rpm[t] = P.rpm[t];
    b.gradn[t] = P.gradn[t];
    if (learned_active(P) && tr.sch.hor == 1) learned_slot_buffers(P, t, &b.feat[t], &b.fscale[t]);
    b.off[t] = tr.off;
    b.seed[t] = mix32_host(P.sround_seed ^ mix32_host((uint32_t)(first + t) * 0x9e3779b9u + tr.nstep));
    tr.nstep++;
  }
  b.adf_h = P.adfh;
  b.adf_v = P.adfv;
  b.lo = P.lo;
  b.sround = storage16(P) ? P.sround : 0;
  // the velocity only changes through set_velocity: the first launch after it
  // stores the edge volume fluxes, later ones load them
  b.vflux = P.vflux;
  b.vflux_mode = P.vflux_valid ? 2 : 1;
  dispatch(P, P.tr[first].sch, nt, b, dt);
  P.vflux_valid = true;
  for (int t = 0; t < nt; t++) std::swap(P.tr[first + t].T, P.tr[first + t].Tout);
}

static bool same_scheme(const TracerScheme &a, const TracerScheme &b) {
  return a.hor == b.hor && a.ver == b.ver && a.lim == b.lim && a.ph == b.ph && a.pv == b.pv;
}

// batch sizes the engine launches: 4, 2 or 1 tracers
static int batch_size(const EngineImpl &P, int first) {
  int run = 1;
  while (first + run < (int)P.tr.size() && run < kBatchMax && same_scheme(P.tr[first].sch, P.tr[first + run].sch)) run++;
  return run >= 4 ? 4 : (run >= 2 ? 2 : 1);
}

int Engine::launches_per_step() const {
  const EngineImpl &P = *p_;
  int n = 0;
  for (int i = 0; i < (int)P.tr.size();) {
    const int nt = batch_size(P, i);
    if (fused_step(P, P.tr[i].sch, learned_active(P) && P.tr[i].sch.hor == 1)) n += nt;
    else n += (P.tr[i].sch.lim == 1 ? 4 : 3) + (P.tr[i].sch.hor != 0 ? 1 : 0);
    i += nt;
  }
  return n;
}

void Engine::set_step_path(int path) {
  if (path < 0 || path > 1) throw std::invalid_argument("step path must be 0 (fused where possible) or 1 (five kernels)");
  p_->step_path = path;
}
int Engine::step_path() const { return p_->step_path; }
bool Engine::fused(int id) const {
  check_id(*p_, id);
  return fused_step(*p_, p_->tr[id].sch, learned_active(*p_) && p_->tr[id].sch.hor == 1);
}
int Engine::tile_count() const { return p_->tiles.np; }
void Engine::set_patch_size(int owned) {
  if (owned < 1) throw std::invalid_argument("patch size must be at least one owned node");
  CK(cudaStreamSynchronize(p_->stream));
  build_tiles(*p_, edge_slot_order(p_->mesh), owned);
  CK(cudaStreamSynchronize(p_->stream));
}
double Engine::tile_node_ratio() const { return p_->tplan.node_ratio; }

bool Engine::step_io(double dt, bool refresh_ab, const double *const *in, double *const *out) {
  EngineImpl &P = *p_;
  const int ntr = (int)P.tr.size();
  const size_t bytes = sizeof(double) * (size_t)(P.mesh.nl - 1) * P.mesh.nod2D;
  if (P.prec != Precision::FP64 && P.prec != Precision::FP32) return false;
  for (int t = 0; t < ntr; t++) {
    if (in && in[t] && !host_range_pinned(in[t], bytes)) return false;
    if (out && out[t] && !host_range_pinned(out[t], bytes)) return false;
    if (!refresh_ab && !P.tr[t].TAB) return false;
  }
  CK(cudaStreamSynchronize(P.stream));
  if (!P.io_h2d) {
    CK(cudaStreamCreateWithFlags(&P.io_h2d, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&P.io_d2h, cudaStreamNonBlocking));
  }
  while ((int)P.io_in.size() < ntr) {
    P.io_in.push_back(P.dalloc<double>(bytes / sizeof(double)));
    P.io_out.push_back(P.dalloc<double>(bytes / sizeof(double)));
    cudaEvent_t a, b;
    CK(cudaEventCreateWithFlags(&a, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&b, cudaEventDisableTiming));
    P.io_ev_in.push_back(a);
    P.io_ev_out.push_back(b);
  }
  // every input copy is queued at once on the H2D stream; the compute stream
  // takes each tracer as soon as its copy lands, and the D2H stream takes
  // each new field as soon as its step is done
  for (int t = 0; t < ntr; t++)
    if (in && in[t]) {
      CK(cudaMemcpyAsync(P.io_in[t], in[t], bytes, cudaMemcpyHostToDevice, P.io_h2d));
      CK(cudaEventRecord(P.io_ev_in[t], P.io_h2d));
    }
  for (int t = 0; t < ntr; t++) {
    auto &tr = P.tr[t];
    if (in && in[t]) {
      CK(cudaStreamWaitEvent(P.stream, P.io_ev_in[t], 0));
      pack_from(P, P.io_in[t], P.stream, tr.T, tr.TAB, tr.Tout);
    }
    run_batch(P, t, 1, dt, refresh_ab);
    if (out && out[t]) {
      unpack_to(P, tr.T, P.io_out[t], P.stream);
      CK(cudaEventRecord(P.io_ev_out[t], P.stream));
      CK(cudaStreamWaitEvent(P.io_d2h, P.io_ev_out[t], 0));
      CK(cudaMemcpyAsync(out[t], P.io_out[t], bytes, cudaMemcpyDeviceToHost, P.io_d2h));
    }
  }
  CK(cudaStreamSynchronize(P.stream));
  CK(cudaStreamSynchronize(P.io_d2h));
  CK(cudaStreamSynchronize(P.io_h2d));
  return true;
}

void Engine::step_tracer(int id, double dt, bool refresh_ab) {
  check_id(*p_, id);
  run_batch(*p_, id, 1, dt, refresh_ab);
}

void Engine::step(double dt, bool refresh_ab) {
  for (int i = 0; i < (int)p_->tr.size();) {
    const int nt = batch_size(*p_, i);
    run_batch(*p_, i, nt, dt, refresh_ab);
    i += nt;
  }
}

size_t Engine::step_scratch_doubles() const {
  const EngineImpl &P = *p_;
  auto up = [](size_t n) { return (n + 31) / 32 * 32; };  // 256-byte pieces
  const size_t es = up((size_t)P.mesh.edge2D * P.S), ns = up((size_t)P.mesh.nod2D * P.S);
  return 2 * es + 6 * ns;
}

void Engine::step_with_scratch(int id, const double *T, const double *TAB, double *T_out, double dt, double *scratch,
                               size_t scratch_doubles) {
  EngineImpl &P = *p_;
  check_id(P, id);
  if (P.prec != Precision::FP64) throw std::invalid_argument("the allocation-free step runs the FP64 engine only");
  if (scratch_doubles < step_scratch_doubles()) throw std::length_error("scratch too small for this mesh");
  auto up = [](size_t n) { return (n + 31) / 32 * 32; };
  const size_t es = up((size_t)P.mesh.edge2D * P.S), ns = up((size_t)P.mesh.nod2D * P.S);
  BatchPtrs b;
  b.T[0] = T;
  b.TAB[0] = TAB;
  b.T_out[0] = T_out;
  b.vflux = scratch;
  b.adf_h = scratch + es;
  b.adf_v = scratch + 2 * es;
  b.lo = scratch + 2 * es + ns;
  b.rpm[0] = scratch + 2 * es + 2 * ns;  // 2 ns
  b.gradn[0] = scratch + 2 * es + 4 * ns;
  dispatch(P, P.tr[id].sch, 1, b, dt);
  CK(cudaStreamSynchronize(P.stream));
}

const char *const *Engine::kernel_kind_names(int *n) {
  static const char *const names[KK_COUNT] = {"k_edge", "k_col1", "k_col2", "k_col3", "k_grad", "k_tile", "k_vflux"};
  *n = KK_COUNT;
  return names;
}

int Engine::profile_steps(int nsteps, double dt, bool refresh_ab, double *ms, int nkinds) {
  EngineImpl &P = *p_;
  std::vector<EngineImpl::ProfRec> recs;
  P.prof = &recs;
  try {
    for (int s = 0; s < nsteps; s++) step(dt, refresh_ab);
  } catch (...) {
    P.prof = nullptr;
    throw;
  }
  P.prof = nullptr;
  CK(cudaStreamSynchronize(P.stream));
  for (int k = 0; k < nkinds; k++) ms[k] = 0.0;
  for (auto &r : recs) {
    float t = 0.f;
    CK(cudaEventElapsedTime(&t, r.a, r.b));
    if (r.kind < nkinds) ms[r.kind] += t;
    cudaEventDestroy(r.a);
    cudaEventDestroy(r.b);
  }
  return (int)recs.size();
}

void Engine::volume_sum(int id, double out[2]) const {
  EngineImpl &P = *p_;
  check_id(P, id);
  CK(cudaStreamSynchronize(P.stream));
  if (P.prec == Precision::FP64) volume_sum_f64(P, P.tr[id].T, out);
  else volume_sum_f32(P, P.tr[id].T, P.tr[id].off, out);
}

void Engine::stats(int id, double out[4]) const {
  EngineImpl &P = *p_;
  check_id(P, id);
  tracer_stats(P, P.tr[id].T, P.tr[id].off, out);
}

}  // namespace fesom
