// Device-resident mesh tables and work schedules.
//
// Edge arrays are stored in "slot" order -- edges sorted by their first node,
// so the edges of neighbouring nodes sit next to each other -- while every
// node-side gather still walks its edges in ascending edge id, the order of
// the reference's serial scatters.
//
// HBM layout: every 3D field is column-major per node (or element, or edge)
// with the level index fastest and a padded level stride S (multiple of 4
// levels, so every column starts on a 32-byte sector for FP64).  A cell
// (column c, level k, 0-based) lives at c*S + k.  The 2D tables are
// structure-of-arrays in int2/double2/double4 records so one vector load
// fetches an edge's nodes, elements or cross distances.
//
// Work is scheduled over wet level pairs only: a lane's entry names its column or
// edge and the first of its two levels (DPairs), so every lane has work even where
// the bathymetry leaves most of a column dry.  The learned flux's training kernels
// walk single wet cells by prefix sums of the wet-level counts (DSched).
#pragma once
#include <cuda_runtime.h>

namespace fesom {

// Schedule over "items" (nodes or edges) with a variable number of levels.
struct DSched {
  const int *cell_off;  // (n_items + 1) prefix sums of wet levels
  const int *blk;       // (nblk + 1) first item of each block
  int nblk;
  int max_items;        // largest item count in one block
};

// Schedule of level pairs over items (nodes or edges): lane i of warp w takes
// the pair of item[32 w + i] whose first level is lev & kPairLevel, or none where
// lev is kPairNone.  Items follow one another in the order of their slots or
// (within windows of 256) nodes, so that a block's pairs share their neighbours'
// columns in L1.  Edge pairs whose
// levels all have both an up and a down triangle and those that have not
// (kPairRing) are kept in warps apart, so that no warp mixes the two forms of
// the MUSCL gradient.  kPairHalo: computed, stored by another warp.
struct DPairs {
  const int *item;
  const unsigned short *lev;
  int nwarps;
};
// blocks of `threads` threads that hold the schedule's warps, `per` to a warp
inline int pair_blocks(const DPairs &s, int threads, int per) {
  const int n = threads / 32 * per;
  return (s.nwarps + n - 1) / n;
}
// Warps of a schedule that a warp takes one after the other, its loads running
// ahead from one to the next: at most `most`.  Measured at 1000x1000x64: edges 1 / 2 /
// 4 / 8: FP64 2.28 / 1.94 / 1.83 / 1.83 ms; columns (k_col1 + k_col2 + k_col3) 4.77 / 4.28 /
// 4.62 / 4.87 ms.  A run also divides the warps launched, and with them the waves that
// the last one is a part of: fewer where less than 40 warps per SM would be left, 1.1
// to 2.5 waves of the kernels' 16 to 36.  A step with column runs of 1 / 2: at 9,510
// warps (150x150x64) FP64, two tracers 0.155 / 0.163 ms, FP32, one 0.057 / 0.061; at
// 5,072 0.092 / 0.102, 0.033 / 0.044; at 13,773 (FP64, one) 0.133 / 0.128; with edge runs
// of 1 / 2 / 4 (FP64, two): at 11,415 0.088 / 0.088 / 0.092, at 31,025 0.217 / 0.212 /
// 0.216, at 59,943 0.407 / 0.396 / 0.398.  Engines that share the device (a batch's
// members on their streams) fill it together, so their runs are cut at 16 warps per
// SM: three members of 194x194x36, 213x213x29 and 188x188x26, 8 tracers: 0.904 ms a
// step at 16, 0.920 at 40.
constexpr int kEdgeRun = 4, kColRun = 2, kRunAlone = 40, kRunShared = 16;
inline int pair_run(const DPairs &s, int most, int warps_per_sm) {
  const int n = s.nwarps / (148 * warps_per_sm);
  return n < 1 ? 1 : (n > most ? most : n);
}
constexpr unsigned kPairNone = 0xffffu, kPairHalo = 0x8000u, kPairRing = 0x4000u, kPairLevel = 0x3fffu;

template <typename R>
struct DMeshT {
  int N, T, E, nl, S;
  // 2D tables
  const int2 *edge_nodes;   // (n1, n2)
  const int2 *edge_tri;     // (el1, el2), el2 = -1 on boundary edges
  const int2 *edge_lev;     // (shared levels = min(nl1, nl2), edge levels = max(nl1, nl2))
  const R *edge_cross;      // (4, E): dX1, dY1, dX2, dY2
  const R *edge_dxdy;       // (2, E)
  const R *edge_a;          // (E)
  const int2 *up_dn;        // (up, dn) triangles, -1 = none
  const int *nlev_elem;     // nlevels(elem)
  const int *nlev_node;     // nlevels_nod2D
  const int *nlev_node_min; // nlevels_nod2D_min
  const int *nbl;           // nboundary_lay
  const int *elem_nodes;    // (3, T)
  const R *grad_sca;        // (6, T)
  const R *elem_area;       // (T)
  const int *ring_ptr;      // (N+1)
  const int *ring_elem;
  const int *ne_ptr;        // (N+1)
  const int4 *ne4;          // per incidence, in ascending edge id:
                            // (slot << 1 | node is the edge's 2nd node, other node, edge levels,
                            //  other node x S: its column base)
  const R *zbar;            // (nl)
  const R *Z;               // (nl-1)
  // 3D geometry, stride S
  const R *area;            // node, nl levels
  const R *areasvol;        // node
  const R *hnode;           // node
  const R *hnode_new;       // node
  const R *helem;           // element
  // reciprocals 1/areasvol (plane 0) and 1/hnode_new (plane 1) of the wet
  // cells, S x N each, computed once per mesh (k_rcp_planes)
  const R *rcp;
  size_t rcp_plane;         // S * N
  // Per-edge record of k_edge (slot order), read as vectors.  edge_idx: three
  // int4, {n1 S, n2 S, u0 S, u1 S}, {u2 S, d0 S, d1 S, d2 S} (column bases of the
  // edge's nodes and of its up and down triangles' nodes) and {levels with both
  // triangles wet, levels where c_lo is 1 at n1, at n2, edge levels}.
  // edge_geo: 16 reals, the up and down triangles' gradient_sca, edge_dxdy(1)
  // * edge_a, edge_dxdy(2) * r_earth and two unused.
  const int4 *edge_idx;
  const R *edge_geo;
  DPairs edge_pairs;        // items = edges
  // Node records of the column kernels: nrec {nlevels | incident edges << 16,
  // nlevels_nod2D_min | complete ring << 31, levels of the first three incident
  // edges and of the next three in 10 bits each}; ne6: {slot x S, other node x
  // S | node is the edge's second << 31} of the first six incident edges in
  // ascending edge id (fewer: entries without levels).
  const int4 *nrec;
  const int4 *ne6;          // three int4 per node
  DPairs node_pairs;        // items = nodes; whole columns, or overlapping pieces of
                            // those deeper than a warp
  // thicknesses and 1/hnode_new of cell (n, k) at [n hS + k]: the full arrays,
  // or one column (hS = 0) where every node has the same at each wet level
  const R *hT, *hnT, *yhnT;
  int hS;
  int uniform_h;            // the latter holds; ltab has the PPM weights
  const R *ltab;            // level tables (advect_fused.cuh)
  DSched node_sched;        // items = nodes, levels = nlev_node - 1
  DSched edge_sched;        // items = edges, levels = edge levels
  // Element record of the ring means: {column bases (node x S) of its nodes,
  // layers} and 8 reals, gradient_sca, area and one unused.
  const int4 *elem_idx;
  const R *elem_geo;
  DPairs grad_pairs;        // node-level pairs some incident edge takes the ring mean of
};

}  // namespace fesom
