// Kernels of the tracer advection step (do_oce_adv_tra,
// lib/oce_adv_tra_driver.F90:23-294, FCT of lib/oce_adv_tra_fct.F90), fused
// into four passes and batched over up to NTMAX tracers that share a mesh,
// a flow and a scheme.
//
//   k_edge  [edge pairs]  volume flux of every edge level (stored once for all
//                         tracers) and, per tracer, the antidiffusive flux
//                         HO(T_AB) - LO(T) (MUSCL/MFCT/UPW1), or HO alone
//                         without FCT
//   k_col1  [node pairs]  horizontal LO gather, vertical LO and HO fluxes
//                         (PPM slopes and interface values of the neighbouring
//                         levels by shuffle, geometry coefficients shared by the
//                         tracers), LO solution
//   k_col2  [node pairs]  FCT cluster bounds (a1-a3), antidiffusive in/out
//                         sums (b1) and limiter ratios (b2)
//   k_col3  [node pairs]  limiting (b3), flux2dtracer, T += del / h_new
//
// A lane advances a pair of levels (2j+1, 2j+2) of its column or edge for every
// tracer of its group; warps are packed with whole columns (pairs.cuh).
//
// Edge scatters of the reference become node-centric gathers over the
// node's incident edges in ascending edge id: every node sums its
// contributions in the order of the reference's serial edge loop, with no
// float atomics.  The FP64 build has no FMA contraction and keeps every
// operation of the reference in its order; divisions multiply by a reciprocal (a
// table's for static geometry, formed on the spot otherwise) and correct the product
// after Markstein, which gives the correctly rounded quotient, i.e. the bits of a
// division.  They are straight-line: operands outside the range where that is exact
// set a flag, and the lane repeats its pair with plain divisions (div_fast, div_any,
// div_3k below; div_rcp, which branches, is left to the fused patch kernel).
#pragma once
#include <cstdint>

#include "pairs.cuh"

namespace fesom {
FESOM_VARIANT_BEGIN

constexpr int NTMAX = 4;
constexpr int kThreads = 256;
constexpr int kEdgeThreads = 128, kColThreads = 128;

// Programmatic dependent launch: each step kernel lets the next one start as soon
// as its own blocks run, and waits, after reading its schedule and tables, for
// the kernel before it to be complete.  Both are no-ops in a kernel launched without
// the attribute.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void prefetch(const void *p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
// Resident 128-thread blocks per SM that each step kernel's register budget is
// cut for.  The kernels are bound by the latency of their gathers; a lane issues the
// loads of its whole stencil before it uses the first, so what hides the latency
// is the loads in flight per warp: 16 warps of 128 registers per SM beat 20-24
// with fewer (FP64, 400x400x64, two tracers: k_edge 0.30 ms at 4 blocks, 0.33 at 3; k_col1
// 0.225 at 4, 0.256 / 0.30 at 3 / 5; k_col3 0.236 at 4, 0.237 / 0.32; FP32 k_edge 0.184 at 5, 0.193
// / 0.188 at 4 / 6; k_col1 0.133 at 7, 0.141 at 5, and with BF16 storage at 500x500x48
// 0.152, 0.172; k_col2 0.138 at 6, 0.148 at 8: as measured when each budget was chosen.
// The present build: FP64 k_edge 0.301, k_col1 0.240, k_col2 0.255, k_col3 0.205 ms, FP32
// 0.162, 0.132, 0.137, 0.126).  Build-time knobs.
#ifndef FESOM_MINB_EDGE
#define FESOM_MINB_EDGE 4
#endif
#ifndef FESOM_MINB_COL1
#define FESOM_MINB_COL1 4
#endif
#ifndef FESOM_MINB_COL2
#define FESOM_MINB_COL2 4
#endif
#ifndef FESOM_MINB_COL3
#define FESOM_MINB_COL3 4
#endif
#ifndef FESOM_MINB_GRAD
#define FESOM_MINB_GRAD 7
#endif
#ifndef FESOM_MINB32_GRAD
#define FESOM_MINB32_GRAD 9
#endif
#ifndef FESOM_MINB32_EDGE
#define FESOM_MINB32_EDGE 5
#endif
#ifndef FESOM_MINB32_FEAT
#define FESOM_MINB32_FEAT 4
#endif
#ifndef FESOM_MINB32_COL1
#define FESOM_MINB32_COL1 7
#endif
#ifndef FESOM_MINB32_COL2
#define FESOM_MINB32_COL2 6
#endif
#ifndef FESOM_MINB32_COL3
#define FESOM_MINB32_COL3 7
#endif
template <typename R, int NT>
struct StepBlocks {
  // (k_col1 of one tracer: 6 blocks 0.148, 4 blocks 0.161 ms)
  static constexpr int grad = FESOM_MINB_GRAD, edge = FESOM_MINB_EDGE, feat = edge, col1 = NT == 1 ? 6 : FESOM_MINB_COL1,
                       col2 = FESOM_MINB_COL2, col3 = FESOM_MINB_COL3;
};
template <int NT>
struct StepBlocks<float, NT> {
  // four tracers a lane: 128 registers; one: more blocks (k_col1 0.093 ms at 9, 0.105
  // at 5; BF16 storage 0.105, 0.138)
  static constexpr int pick(int n1, int n2) { return NT == 4 ? 4 : (NT == 1 ? n1 : n2); }
  // k_edge with the learned flux's features of two tracers: 0.666 ms at 4, 0.784 at 5,
  // 0.726 at 3 (500x500x64); of one: 0.418 at 6, 0.437 at 4
  static constexpr int feat = pick(6, FESOM_MINB32_FEAT);
  static constexpr int grad = FESOM_MINB32_GRAD, edge = pick(6, FESOM_MINB32_EDGE), col1 = pick(9, FESOM_MINB32_COL1),
                       col2 = pick(8, FESOM_MINB32_COL2), col3 = pick(7, FESOM_MINB32_COL3);
};
// Tracers of a batch of NT that a lane advances together; it takes the groups one
// after the other.  Two FP64 tracers share a column's records and geometry
// (400x400x64: k_col1 0.240 ms against 2 x 0.154 for one at a time, k_col3 0.205 against
// 2 x 0.133), except in k_col2, whose sums and bounds of two do not fit the registers
// (one after the other 0.267, both at once 0.363, when it was chosen; 0.255 now).
template <typename R, int NT>
struct LaneTracers {
  static constexpr int cap(int g) { return g < NT ? g : NT; }
  static constexpr int col1 = cap(sizeof(R) == 8 ? 2 : 4), col2 = cap(sizeof(R) == 8 ? 1 : 4), col3 = col1,
                       grad = cap(sizeof(R) == 8 ? 2 : 4);
};
constexpr int kCellsPerBlock = 512;      // cell maps (learned flux): wet cells per block, two per thread
constexpr int kMaxCellsPerBlock = 576;   // upper bound (target + deepest column)
constexpr int kMaxItemsPerBlock = 512;

// ---------------------------------------------------------------------------
// Correctly rounded division a / b given y = RN(1/b).
//
// Markstein's theorem (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; see also
// Muller et al., Handbook of Floating-Point Arithmetic, Sec. 4.7): if y is
// within half an ulp of 1/b and q is a faithful approximation of a/b, then
// r = a - b q is exact when computed with one FMA and RN(q + r y) = RN(a/b).
// q0 = RN(a y) can be 1.5 ulp off, so one correction first makes it faithful,
// the second rounds correctly.  Zero and extreme magnitudes (where r could
// underflow or overflow) take the plain division.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double div_rcp(double a, double b, double y) {
  const double aa = fabs(a);
  if (!(aa > 0x1p-900 && aa < 0x1p900)) return a / b;
  double q = a * y;
  double r = __fma_rn(-b, q, a);
  if (r == 0.0) return q;
  q = __fma_rn(r, y, q);
  r = __fma_rn(-b, q, a);
  return __fma_rn(r, y, q);
}
__device__ __forceinline__ float div_rcp(float a, float b, float y) {
  const float aa = fabsf(a);
  if (!(aa > 0x1p-100f && aa < 0x1p100f)) return a / b;
  float q = a * y;
  float r = __fmaf_rn(-b, q, a);
  if (r == 0.0f) return q;
  q = __fmaf_rn(r, y, q);
  r = __fmaf_rn(-b, q, a);
  return __fmaf_rn(r, y, q);
}

// R: compute and geometry type; TS: tracer storage type (R itself, or a
// 16-bit float with R = float)
template <typename R, typename TS>
struct FusedArgs {
  const TS *T[NTMAX];     // values
  const TS *TAB[NTMAX];   // valuesAB (high-order fluxes)
  TS *T_out[NTMAX];
  R *adf_h;               // (S, edge) pairs of every tracer side by side (pairs.cuh, il_at)
  R *adf_v;               // (S, node) interfaces, likewise
  R *lo;                  // (S, node), likewise
  R *rpm[NTMAX];          // (2, S, node): limiter ratios R+ and R- of each cell side by side
  R *vflux;               // (S, edge), shared by the tracers
  R *gradn[NTMAX];        // (2, S, node): ring-mean gradient (gx, gy) of valuesAB
  const R *vel;           // (2, S, elem)
  const R *W;             // (S, node) interfaces
  R dt, ph, pv;
  // learned flux (FP32 only): when feat[t] is set the edge kernel writes 16
  // BF16 features and the correction scale of every MUSCL edge cell (dense
  // edge-schedule index)
  __nv_bfloat16 *feat[NTMAX];
  float *fscale[NTMAX];
  R off[NTMAX];           // storage offsets (16-bit storage)
  uint32_t seed[NTMAX];   // per-step random stream of each tracer (stochastic rounding)
  int sround;             // 1: stochastic rounding of 16-bit stores
  // edge volume fluxes: 0, 1 computed from the velocity and stored, 2 loaded
  // from vflux (stored by an earlier launch with the same velocity)
  int vflux_mode;
  // failure detection: count of non-finite new values (nullptr: not counted)
  unsigned long long *nonfinite;
};

// ---------------------------------------------------------------------------
// block cell maps: a block owns a range of items (nodes or edges); every wet
// cell of those items gets the local item index in shared memory
// ---------------------------------------------------------------------------
struct CellMap {
  int i0, ni, c0, nc;
};

__device__ __forceinline__ CellMap map_cells(const DSched &sc, int blk, int *s_off, int *s_item) {
  CellMap cm;
  cm.i0 = sc.blk[blk];
  cm.ni = sc.blk[blk + 1] - cm.i0;
  for (int t = threadIdx.x; t <= cm.ni; t += blockDim.x) s_off[t] = sc.cell_off[cm.i0 + t];
  __syncthreads();
  cm.c0 = s_off[0];
  cm.nc = s_off[cm.ni] - cm.c0;
  for (int j = threadIdx.x; j < cm.ni; j += blockDim.x) {
    const int a = s_off[j] - cm.c0, b = s_off[j + 1] - cm.c0;
    for (int q = a; q < b; q++) s_item[q] = j;
  }
  __syncthreads();
  return cm;
}

// ---------------------------------------------------------------------------
// k_grad: ring-mean gradients of valuesAB (lib/oce_muscl_adv.F90:400-450:
// the mean of tr_xy over the node's ring, weighted by element area), for the
// node-levels where some incident edge lacks a shared up/down pair
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ld_pair(const double *p, double &x, double &y) {
  const double2 v = *reinterpret_cast<const double2 *>(p);
  x = v.x;
  y = v.y;
}
__device__ __forceinline__ void ld_pair(const float *p, float &x, float &y) {
  const float2 v = *reinterpret_cast<const float2 *>(p);
  x = v.x;
  y = v.y;
}
__device__ __forceinline__ void st_pair(double *p, double x, double y) {
  *reinterpret_cast<double2 *>(p) = make_double2(x, y);
}
__device__ __forceinline__ void st_pair(float *p, float x, float y) {
  *reinterpret_cast<float2 *>(p) = make_float2(x, y);
}

// Whether a is not a zero, given u = 2 x its high word: subnormals below 2^-1042
// have a high word of zero and a low word that is not.
__device__ __forceinline__ bool not_zero(double a, unsigned u) { return (u | (unsigned)__double2loint(a)) != 0u; }

// a / b given y = RN(1 / b), correctly rounded (see div_rcp), straight-line:
// numerators outside [2^-900, 2^900] other than zero set `bad` and the caller
// divides again.  The sign of a zero result is not kept (no output of the step
// depends on the sign of a zero quotient).
__device__ __forceinline__ double div_near(double a, double b, double y) {  // numerator known to be in range
  double q = a * y;
  q = __fma_rn(__fma_rn(-b, q, a), y, q);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
__device__ __forceinline__ double div_fast(double a, double b, double y, bool &bad) {
  const unsigned u = 2u * (unsigned)__double2hiint(a);
  bad |= (u - 0x0f600000u > 0xf0800000u - 0x0f600000u) && not_zero(a, u);
  return div_near(a, b, y);
}
__device__ __forceinline__ float div_near(float a, float b, float y) {
  float q = a * y;
  q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
__device__ __forceinline__ float div_fast(float a, float b, float y, bool &bad) {
  const unsigned u = 2u * __float_as_uint(a);
  bad |= (u - 0x1b000000u > 0xe3000000u - 0x1b000000u) && u != 0u;
  return div_near(a, b, y);
}

// RN(1 / b), straight-line: the hardware's approximate reciprocal refined by
// Newton steps y += y (1 - b y), the last of which rounds correctly unless b's
// significand is all ones (Markstein).  That significand, and magnitudes outside
// [2^-500, 2^500] (FP32: [2^-EXP, 2^EXP]: 2^60 where quotients are formed with it),
// set `bad`.
__device__ __forceinline__ double rcp_newton(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));  // about 2^-20
  y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  return __fma_rn(__fma_rn(-b, y, 1.0), y, y);
}
__device__ __forceinline__ double rcp_exact(double b, bool &bad) {
  const double y = rcp_newton(b);
  const unsigned u = 2u * (unsigned)__double2hiint(b);
  bad |= u - 0x41600000u > 0xbe600000u - 0x41600000u || ((unsigned)__double2hiint(b) | 0xfff00000u) == 0xffffffffu;
  return __fma_rn(__fma_rn(-b, y, 1.0), y, y);
}
template <int EXP = 60>
__device__ __forceinline__ float rcp_exact(float b, bool &bad) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));  // within a unit in the last place
  constexpr unsigned lo = (unsigned)(127 - EXP) << 24, hi = (unsigned)(127 + EXP) << 24;
  const unsigned u = 2u * __float_as_uint(b);
  bad |= u - lo > hi - lo || (__float_as_uint(b) | 0xff800000u) == 0xffffffffu;
  return __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
}
// a / b for any divisor, given y = RN(1 / b) of rcp_exact: the limiter ratios and the
// ring means.  Numerators other than zero outside [2^-500, 2^900] (FP32: [2^-60,
// 2^100]) set `bad`, so that no quotient underflows.
__device__ __forceinline__ double div_any(double a, double b, double y, bool &bad) {
  const unsigned u = 2u * (unsigned)__double2hiint(a);
  bad |= (u - 0x41600000u > 0xf0800000u - 0x41600000u) && not_zero(a, u);
  return div_near(a, b, y);
}
__device__ __forceinline__ float div_any(float a, float b, float y, bool &bad) {
  const unsigned u = 2u * __float_as_uint(a);
  bad |= (u - 0x43000000u > 0xe3000000u - 0x43000000u) && u != 0u;
  return div_near(a, b, y);
}
template <typename R>
__device__ __forceinline__ R div_any(R a, R b, bool &bad) {
  return div_any(a, b, rcp_exact(b, bad), bad);
}

// The flag of a pair's divisions: pb[q] takes those of level q, and a dry second
// level's has no say, whatever its cells hold.
struct PairBad {
  bool wet1;  // the second level is wet
  bool any = false;
  struct Level {
    PairBad &p;
    int q;
    bool b = false;
    __device__ __forceinline__ Level(PairBad &p, int q) : p(p), q(q) {}
    __device__ __forceinline__ ~Level() { p.any |= b && (q == 0 || p.wet1); }
    __device__ __forceinline__ operator bool &() { return b; }
  };
  __device__ __forceinline__ explicit PairBad(bool wet1) : wet1(wet1) {}
  __device__ __forceinline__ Level operator[](int q) { return Level(*this, q); }
};

// One pair of node levels: the ring's elements one after the other (a level an
// element does not reach adds nothing).  The pairs are the few bottom levels of
// each column, so every load of a warp touches as many lines as it has nodes:
// the kernel is bound by those lines, and more resident warps hide more of them
// than more loads per warp (400x400x64: one element at a time in 56-72 registers
// FP64 0.088, FP32 0.059 ms; two in 78-120 0.095, 0.062; three 0.098, 0.062; the cell-mapped
// kernel before 0.091, 0.071).
template <typename R, typename TS, int NT>
__device__ __forceinline__ void grad_pair(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int n, int k) {
  const int p0 = m.ring_ptr[n], p1 = m.ring_ptr[n + 1], nln = m.nlev_node[n] - 1;
  R vol[2] = {R(0), R(0)}, sx[NT][2], sy[NT][2];
#pragma unroll
  for (int t = 0; t < NT; t++) sx[t][0] = sx[t][1] = sy[t][0] = sy[t][1] = R(0);
#pragma unroll 1
  for (int p = p0; p < p1; p++) {
    const int el = m.ring_elem[p];
    const int4 r = m.elem_idx[el];
    R g[8], v[NT][3][2];
    ldv8(m.elem_geo + 8 * (size_t)el, g);
#pragma unroll
    for (int t = 0; t < NT; t++) {
      ld_pair_T(a.TAB[t], (cix)r.x + k, a.off[t], v[t][0]);
      ld_pair_T(a.TAB[t], (cix)r.y + k, a.off[t], v[t][1]);
      ld_pair_T(a.TAB[t], (cix)r.z + k, a.off[t], v[t][2]);
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const bool wet = k + q < r.w;
      vol[q] = wet ? vol[q] + g[6] : vol[q];
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const R gx = (g[0] * v[t][0][q] + g[1] * v[t][1][q]) + g[2] * v[t][2][q];
        const R gy = (g[3] * v[t][0][q] + g[4] * v[t][1][q]) + g[5] * v[t][2][q];
        sx[t][q] = wet ? sx[t][q] + gx * g[6] : sx[t][q];
        sy[t][q] = wet ? sy[t][q] + gy * g[6] : sy[t][q];
      }
    }
  }
  const cix o = (cix)n * m.S + k;
  if (k + 1 >= nln) vol[1] = R(1);  // dry
  bool bad = false;
  const R y[2] = {rcp_exact(vol[0], bad), rcp_exact(vol[1], bad)};
#pragma unroll
  for (int t = 0; t < NT; t++) {
    R out[4];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      out[2 * q] = div_any(sx[t][q], vol[q], y[q], bad);
      out[2 * q + 1] = div_any(sy[t][q], vol[q], y[q], bad);
    }
    if (bad)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        out[2 * q] = sx[t][q] / vol[q];
        out[2 * q + 1] = sy[t][q] / vol[q];
      }
    stv4(a.gradn[t] + 2 * (size_t)o, out);
  }
}

template <typename R, typename TS, int NT>
__device__ __forceinline__ void grad_block(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int blk) {
  const int warp = blk * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5);
  if (warp >= m.grad_pairs.nwarps) return;
  const PairLane l = pair_lane(m.grad_pairs, warp);
  if (l.on()) prefetch(m.ring_elem + m.ring_ptr[l.item]);
  pdl_wait();
  if (!l.on()) return;
  constexpr int G = LaneTracers<R, NT>::grad;
  if constexpr (G == NT) {
    grad_pair<R, TS, NT>(m, a, l.item, l.k());
  } else {
    FusedArgs<R, TS> b;  // the pointers grad_pair reads, of one group of tracers at a time
#pragma unroll
    for (int t0 = 0; t0 < NT; t0 += G) {
#pragma unroll
      for (int t = 0; t < G; t++) {
        b.TAB[t] = a.TAB[t0 + t];
        b.off[t] = a.off[t0 + t];
        b.gradn[t] = a.gradn[t0 + t];
      }
      grad_pair<R, TS, G>(m, b, l.item, l.k());
    }
  }
}

template <typename R, typename TS, int NT>
__global__ void __launch_bounds__(kColThreads, StepBlocks<R, NT>::grad)
    k_grad(const __grid_constant__ DMeshT<R> m, const __grid_constant__ FusedArgs<R, TS> a) {
  pdl_launch();
  grad_block<R, TS, NT>(m, a, blockIdx.x);
}

// ---------------------------------------------------------------------------
// k_edge
// ---------------------------------------------------------------------------
// x / 6 and x / 3, correctly rounded.  The reciprocals of 3 and 6 round with a
// relative error of 2^-54 (FP32: 2^-25), so q = RN(x y) is already a faithful
// quotient and one Markstein correction rounds it (div_rcp needs two).  The
// sign of a zero is not kept.  Straight-line: extreme magnitudes (nonzero below
// 2^-900, or not finite), for which the remainder may be inexact, set `bad`, and the
// caller computes that lane again with plain divisions.
template <int B>  // B = 3 or 6
__device__ __forceinline__ double div_3k(double x, bool &bad) {
  const double y = 1.0 / B;
  const double q = x * y;
  const unsigned u = 2u * (unsigned)__double2hiint(x);
  bad |= (u - 0x0f600000u >= 0xffe00000u - 0x0f600000u) && not_zero(x, u);
  return __fma_rn(__fma_rn(-(double)B, q, x), y, q);
}
template <int B>
__device__ __forceinline__ float div_3k(float x, bool &bad) {
  const float y = 1.0f / B;
  const float q = x * y;
  const unsigned u = 2u * __float_as_uint(x);
  bad |= (u - 0x1b000000u >= 0xff000000u - 0x1b000000u) && u != 0u;  // 2^-100
  return __fmaf_rn(__fmaf_rn(-(float)B, q, x), y, q);
}
template <typename R>
__device__ __forceinline__ R div6(R x, bool &bad) { return div_3k<6>(x, bad); }
template <typename R>
__device__ __forceinline__ R div3(R x, bool &bad) { return div_3k<3>(x, bad); }

// Divisions of the learned flux's features, correctly rounded: straight-line, or
// plain again for the lanes that set `bad`.
struct FeatFast {
  bool &bad;
  __device__ __forceinline__ float rcp(float x) { return rcp_exact<100>(x, bad); }
  __device__ __forceinline__ float div(float a, float b) { return div_fast(a, b, rcp_exact(b, bad), bad); }
};
struct FeatPlain {
  __device__ __forceinline__ float rcp(float x) { return 1.0f / x; }
  __device__ __forceinline__ float div(float a, float b) { return a / b; }
};
// Courant number of an edge level's volume flux in the upwind node's cell, of
// volume vol; the same for every tracer.
template <typename D>
__device__ __forceinline__ float edge_courant(float vflux, float dt, float vol, D d) {
  return fminf(d.div(fabsf(vflux) * dt, vol), 4.0f);
}

// learned flux: 16 features of one MUSCL edge level in the flow's frame, in
// units of the local variation sig, and the scale of the network's output
template <typename TS, typename D>
__device__ __forceinline__ void edge_features(const DMeshT<float> &m, const FusedArgs<float, TS> &a, D d, int t, int cell,
                                              int k, float vflux, float cour, float t1, float t2, float x1, float x2, float Tmean1,
                                              float Tmean2, float gux, float guy, float gdx, float gdy, float exa,
                                              float eyr, float c_lo1, float c_lo2, bool shared) {
  const float sixth = 1.0f / 6.0f;
  const bool fwd = vflux >= 0.0f;
  const float tu = fwd ? t1 : t2, td = fwd ? t2 : t1;
  const float xu = fwd ? x1 : -x2, xd = fwd ? x2 : -x1;
  const float face = 0.5f * (Tmean1 + Tmean2);
  const float sig = fabsf(td - tu) + (fabsf(xu) + fabsf(xd)) * sixth + 1e-6f * (fabsf(tu) + fabsf(td)) + 1e-20f;
  const float inv = d.rcp(sig);
  const float gx = fwd ? gux : gdx, gy = fwd ? guy : gdy;
  const float trans = (-eyr * gx + exa * gy) * inv;
  float f[16];
  f[0] = (td - tu) * inv;
  f[1] = xu * sixth * inv;
  f[2] = xd * sixth * inv;
  f[3] = (face - tu) * inv;
  f[4] = cour;
  f[5] = cour * cour;
  f[6] = fwd ? c_lo1 : c_lo2;
  f[7] = fwd ? c_lo2 : c_lo1;
  f[8] = (float)k / (float)max(1, m.nl - 2);
  f[9] = shared ? 1.0f : 0.0f;
  f[10] = fabsf(f[0]);
  f[11] = f[1] - f[2];
  f[12] = (xu * xd > 0.0f) ? 1.0f : -1.0f;
  f[13] = fminf(fabsf(f[1]), fabsf(f[2]));
  f[14] = fmaxf(-8.0f, fminf(8.0f, trans));
  f[15] = 1.0f;
  __align__(16) __nv_bfloat16 h[16];
  for (int q = 0; q < 16; q++) h[q] = __float2bfloat16_rn(f[q]);
  uint4 *dst = reinterpret_cast<uint4 *>(a.feat[t] + (size_t)cell * 16);
  dst[0] = reinterpret_cast<const uint4 *>(h)[0];
  dst[1] = reinterpret_cast<const uint4 *>(h)[1];
  a.fscale[t][cell] = -vflux * sig;
}

// Record of an edge: the column bases of its nodes and its triangles' nodes,
// and its level limits (DMeshT::edge_idx).
struct EdgeIdx {
  int4 a, b, c;
  __device__ __forceinline__ int tri_levels() const { return c.x; }
  __device__ __forceinline__ int c1_levels() const { return c.y; }
  __device__ __forceinline__ int c2_levels() const { return c.z; }
  __device__ __forceinline__ int levels() const { return c.w; }
};
template <typename R>
__device__ __forceinline__ EdgeIdx edge_idx(const DMeshT<R> &m, int e) {
  const int4 *p = m.edge_idx + 3 * (size_t)e;
  return EdgeIdx{p[0], p[1], p[2]};
}

// Both levels of an edge pair once more, with plain divisions: the lanes whose
// operands lie outside div6's range.
template <typename R, typename TS, int NT, int HOR, int LIM>
__device__ __noinline__ void edge_pair_slow(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int e, int k0) {
  const EdgeIdx x = edge_idx(m, e);
  const R *g = m.edge_geo + 16 * (size_t)e;
#pragma unroll 1
  for (int k = k0; k < min(k0 + 2, x.levels()); k++) {
    const cix o = (cix)e * m.S + k, o1 = (cix)x.a.x + k, o2 = (cix)x.a.y + k;
    const R vf = a.vflux[o];
    const R c1 = HOR == HOR_MFCT || k < x.c1_levels() ? R(1) : R(0), c2 = HOR == HOR_MFCT || k < x.c2_levels() ? R(1) : R(0);
#pragma unroll 1
    for (int t = 0; t < NT; t++) {
      auto B = [&](int base) { return ldT<R>(a.TAB[t], (cix)base + k, a.off[t]); };
      R gux, guy, gdx, gdy;
      if (k < x.tri_levels()) {
        const R u0 = B(x.a.z), u1 = B(x.a.w), u2 = B(x.b.x), d0 = B(x.b.y), d1 = B(x.b.z), d2 = B(x.b.w);
        gux = (g[0] * u0 + g[1] * u1) + g[2] * u2;
        guy = (g[3] * u0 + g[4] * u1) + g[5] * u2;
        gdx = (g[6] * d0 + g[7] * d1) + g[8] * d2;
        gdy = (g[9] * d0 + g[10] * d1) + g[11] * d2;
      } else {
        ld_pair(a.gradn[t] + 2 * (size_t)o1, gux, guy);
        ld_pair(a.gradn[t] + 2 * (size_t)o2, gdx, gdy);
      }
      const R b1 = B(x.a.x), b2 = B(x.a.y);
      const R x2 = R(2) * (b2 - b1) + g[12] * gdx + g[13] * gdy;
      const R x1 = R(2) * (b2 - b1) + g[12] * gux + g[13] * guy;
      const R Tmean2 = b2 - x2 / R(6) * c2, Tmean1 = b1 + x1 / R(6) * c1;
      const R cHO = (vf + fabs(vf)) * Tmean1 + (vf - fabs(vf)) * Tmean2;
      const R ho = -(R(0.5) * (R(1) - a.ph) * cHO) - vf * a.ph * R(0.5) * (Tmean1 + Tmean2);
      const R flo = (LIM == LIM_FCT) ? upw1_flux(vf, ldT<R>(a.T[t], o1, a.off[t]), ldT<R>(a.T[t], o2, a.off[t])) : R(0);
      il<NT>(a.adf_h, t, o) = ho - flo;
      if constexpr (HOR == HOR_MUSCL_FEAT) {
        const cix ou = vf >= R(0) ? o1 : o2;
        edge_features(m, a, FeatPlain{}, t, m.edge_sched.cell_off[e] + k, k, vf,
                      edge_courant(vf, a.dt, m.areasvol[ou] * m.hnode_new[ou], FeatPlain{}), b1, b2, x1, x2, Tmean1, Tmean2, gux, guy,
                      gdx, gdy, g[12], g[13], c1, c2, k < x.tri_levels());
      }
    }
  }
}

// One edge pair.  RING: some lane of the warp has a level without both
// triangles (the schedule groups such pairs into warps of their own), which
// takes the node ring means of k_grad instead.  LOADV: the edge volume fluxes
// are stored (vflux_mode 2); otherwise they are computed here and stored.
template <typename R, typename TS, int NT, int HOR, int LIM, bool LOADV, bool RING>
__device__ __forceinline__ void edge_pair(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int e, int k, const EdgeIdx &x) {
  const cix o = (cix)e * m.S + k;
  R vf[2];
  if constexpr (LOADV) {
    ldv2(a.vflux + o, vf);
  } else {
    const EdgeCtx<R> c = edge_ctx(m, e);
    vf[0] = edge_vflux(m, c, a.vel, k);
    vf[1] = k + 1 < c.levels ? edge_vflux(m, c, a.vel, k + 1) : R(0);
    stv2(a.vflux + o, vf);
  }
  const cix o1 = (cix)x.a.x + k, o2 = (cix)x.a.y + k;
  if constexpr (HOR == HOR_UPW1) {
    const R vp[2] = {vf[0] + fabs(vf[0]), vf[1] + fabs(vf[1])}, vm[2] = {vf[0] - fabs(vf[0]), vf[1] - fabs(vf[1])};
#pragma unroll
    for (int t = 0; t < NT; t++) {
      R b1[2], b2[2];
      ld_pair_T(a.TAB[t], o1, a.off[t], b1);
      ld_pair_T(a.TAB[t], o2, a.off[t], b2);
      R t1[2] = {b1[0], b1[1]}, t2[2] = {b2[0], b2[1]};
      if (LIM == LIM_FCT && a.T[t] != a.TAB[t]) {
        ld_pair_T(a.T[t], o1, a.off[t], t1);
        ld_pair_T(a.T[t], o2, a.off[t], t2);
      }
      R out[2];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const R flo = (LIM == LIM_FCT) ? R(-0.5) * (t1[q] * vp[q] + t2[q] * vm[q]) : R(0);
        out[q] = R(-0.5) * (b1[q] * vp[q] + b2[q] * vm[q]) - flo;
      }
      if (k + 1 >= x.levels()) out[1] = R(0);
      st_pair_il<NT, 1>(a.adf_h, t, o, out);
    }
  } else {
    PairBad bad(k + 1 < x.levels());
    // the loads of G tracers are all issued before the first is used
    constexpr int G = NT > 2 ? 2 : NT;
    [[maybe_unused]] int cell = 0;
    [[maybe_unused]] R vol[2] = {R(1), R(1)};
    if constexpr (HOR == HOR_MUSCL_FEAT) {
      cell = m.edge_sched.cell_off[e] + k;
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const cix ou = (vf[q] >= R(0) ? o1 : o2) + q;
        vol[q] = m.areasvol[ou] * m.hnode_new[ou];
      }
    }
#pragma unroll
    for (int t0 = 0; t0 < NT; t0 += G) {
      R b1[G][2], b2[G][2], u[G][3][2], d[G][3][2], p1[G][4], p2[G][4];
#pragma unroll
      for (int i = 0; i < G; i++) {
        const TS *B = a.TAB[t0 + i];
        const R off = a.off[t0 + i];
        ld_pair_T(B, o1, off, b1[i]);
        ld_pair_T(B, o2, off, b2[i]);
        ld_pair_T(B, (cix)x.a.z + k, off, u[i][0]);
        ld_pair_T(B, (cix)x.a.w + k, off, u[i][1]);
        ld_pair_T(B, (cix)x.b.x + k, off, u[i][2]);
        ld_pair_T(B, (cix)x.b.y + k, off, d[i][0]);
        ld_pair_T(B, (cix)x.b.z + k, off, d[i][1]);
        ld_pair_T(B, (cix)x.b.w + k, off, d[i][2]);
        if constexpr (RING) {
          ldv4(a.gradn[t0 + i] + 2 * (size_t)o1, p1[i]);
          ldv4(a.gradn[t0 + i] + 2 * (size_t)o2, p2[i]);
        }
      }
      R g[16];
      {
        const R *ge = m.edge_geo + 16 * (size_t)e;
        ldv4(ge, g);
        ldv4(ge + 4, g + 4);
        ldv4(ge + 8, g + 8);
        ldv2(ge + 12, g + 12);
      }
      const R exa = g[12], eyr = g[13];
      const R hph = R(0.5) * (R(1) - a.ph);
      [[maybe_unused]] R cour[2];
      if constexpr (HOR == HOR_MUSCL_FEAT) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
          auto b = bad[q];
          cour[q] = edge_courant(vf[q], a.dt, vol[q], FeatFast{b});
        }
      }
      R out[2 * G];
#pragma unroll
      for (int i = 0; i < G; i++) {
        const int t = t0 + i;
        R t1[2] = {b1[i][0], b1[i][1]}, t2[2] = {b2[i][0], b2[i][1]};
        if (LIM == LIM_FCT && a.T[t] != a.TAB[t]) {
          ld_pair_T(a.T[t], o1, a.off[t], t1);
          ld_pair_T(a.T[t], o2, a.off[t], t2);
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const bool sh = !RING || k + q < x.tri_levels();
          const R c1 = k + q < x.c1_levels() ? R(1) : R(0), c2 = k + q < x.c2_levels() ? R(1) : R(0);
          // edge_up_dn_grad (lib/oce_muscl_adv.F90:383-527)
          R gux = (g[0] * u[i][0][q] + g[1] * u[i][1][q]) + g[2] * u[i][2][q];
          R guy = (g[3] * u[i][0][q] + g[4] * u[i][1][q]) + g[5] * u[i][2][q];
          R gdx = (g[6] * d[i][0][q] + g[7] * d[i][1][q]) + g[8] * d[i][2][q];
          R gdy = (g[9] * d[i][0][q] + g[10] * d[i][1][q]) + g[11] * d[i][2][q];
          if (RING && !sh) {
            gux = p1[i][2 * q]; guy = p1[i][2 * q + 1];
            gdx = p2[i][2 * q]; gdy = p2[i][2 * q + 1];
          }
          // lib/oce_adv_tra_hor.F90:454-469 (MUSCL), :743-753 (MFCT, no c_lo)
          const R x2 = R(2) * (b2[i][q] - b1[i][q]) + exa * gdx + eyr * gdy;
          const R x1 = R(2) * (b2[i][q] - b1[i][q]) + exa * gux + eyr * guy;
          R Tmean2, Tmean1;
          if (HOR != HOR_MFCT) {
            Tmean2 = b2[i][q] - div6(x2, bad[q]) * c2;
            Tmean1 = b1[i][q] + div6(x1, bad[q]) * c1;
          } else {
            Tmean2 = b2[i][q] - div6(x2, bad[q]);
            Tmean1 = b1[i][q] + div6(x1, bad[q]);
          }
          const R vp = vf[q] + fabs(vf[q]), vm = vf[q] - fabs(vf[q]);
          const R cHO = vp * Tmean1 + vm * Tmean2;
          const R ho = -(hph * cHO) - vf[q] * a.ph * R(0.5) * (Tmean1 + Tmean2);
          const R flo = (LIM == LIM_FCT) ? R(-0.5) * (t1[q] * vp + t2[q] * vm) : R(0);
          out[2 * i + q] = ho - flo;
          if constexpr (HOR == HOR_MUSCL_FEAT) {
            if (k + q < x.levels())
              edge_features(m, a, FeatFast{bad.any}, t, cell + q, k + q, vf[q], cour[q], b1[i][q], b2[i][q], x1, x2, Tmean1, Tmean2, gux,
                            guy, gdx, gdy, exa, eyr, c1, c2, sh);
          }
        }
      }
      // a dry second level holds zero: the node kernels add it without a test
      if (k + 1 >= x.levels())
#pragma unroll
        for (int i = 0; i < G; i++) out[2 * i + 1] = R(0);
      st_pair_il<NT, G>(a.adf_h, t0, o, out);
    }
    if (bad.any) edge_pair_slow<R, TS, NT, HOR, LIM>(m, a, e, k);
  }
}

// The edge pairs of `per` consecutive warps of the schedule; the records of
// the next pair and the map entry of the one after it are loaded ahead of the
// current pair's arithmetic, so that a pair costs one memory latency instead of
// three dependent ones.
template <typename R, typename TS, int NT, int HOR, int LIM, bool LOADV>
__device__ __forceinline__ void edge_block(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int blk, int per) {
  const DPairs &s = m.edge_pairs;
  int warp = (blk * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5)) * per;
  const int end = min(warp + per, s.nwarps);
  if (warp >= end) return;
  PairLane nxt = pair_lane(s, warp);
  EdgeIdx idx = edge_idx(m, nxt.item);
  PairLane nn = warp + 1 < end ? pair_lane(s, warp + 1) : nxt;
  pdl_wait();
  do {
    const PairLane c = nxt;
    const EdgeIdx x = idx;
    if (++warp < end) {
      nxt = nn;
      idx = edge_idx(m, nxt.item);
      if (warp + 1 < end) nn = pair_lane(s, warp + 1);
    }
    if (c.on()) {
      if (HOR != HOR_UPW1 && c.ring()) edge_pair<R, TS, NT, HOR, LIM, LOADV, true>(m, a, c.item, c.k(), x);
      else edge_pair<R, TS, NT, HOR, LIM, LOADV, false>(m, a, c.item, c.k(), x);
    }
  } while (warp < end);
}

template <typename R, typename TS, int NT, int HOR, int LIM, bool LOADV>
__global__ void __launch_bounds__(kEdgeThreads, HOR == HOR_MUSCL_FEAT ? StepBlocks<R, NT>::feat : StepBlocks<R, NT>::edge)
    k_edge(const __grid_constant__ DMeshT<R> m, const __grid_constant__ FusedArgs<R, TS> a, int per) {
  pdl_launch();
  edge_block<R, TS, NT, HOR, LIM, LOADV>(m, a, blockIdx.x, per);
}

// ---------------------------------------------------------------------------
// Node columns: lanes hold level pairs, columns are packed whole into warps
// (DMeshT::node_pairs), so the vertical stencils exchange values by shuffles and
// the kernels need neither shared memory nor block barriers.
// ---------------------------------------------------------------------------
constexpr unsigned kFull = 0xffffffffu;

// Node record (DMeshT::nrec, ne6): levels, the first six incident edges in
// ascending edge id, and how many there are.
struct NodeRec {
  int4 h;
  int4 e[3];
  __device__ __forceinline__ int nlev() const { return h.x & 0xffff; }
  __device__ __forceinline__ int degree() const { return (int)((unsigned)h.x >> 16); }
  __device__ __forceinline__ int nlev_min() const { return h.y & 0x7fffffff; }
  __device__ __forceinline__ bool ring_full() const { return h.y < 0; }
  __device__ __forceinline__ int levels(int i) const { return ((i < 3 ? h.z : h.w) >> (10 * (i % 3))) & 1023; }
  __device__ __forceinline__ unsigned edge(int i) const { return (unsigned)(i % 2 ? e[i / 2].z : e[i / 2].x); }
  __device__ __forceinline__ unsigned other(int i) const { return (unsigned)(i % 2 ? e[i / 2].w : e[i / 2].y); }
};
template <typename R>
__device__ __forceinline__ NodeRec node_rec(const DMeshT<R> &m, int n) {
  NodeRec r;
  r.h = m.nrec[n];
  const int4 *p = m.ne6 + 3 * (size_t)n;
  r.e[0] = p[0];
  r.e[1] = p[1];
  r.e[2] = p[2];
  return r;
}
// f(cell of the edge, cell of the other node, node is the edge's second, edge
// levels) for every incident edge in ascending edge id: the six of the record
// unrolled (fewer: the rest have no levels), those beyond from the lists.
template <typename R, typename F>
__device__ __forceinline__ void for_edges(const DMeshT<R> &m, int n, int k, const NodeRec &rec, F f) {
#pragma unroll
  for (int i = 0; i < 6; i++)
    f((cix)rec.edge(i) + k, (cix)(rec.other(i) & 0x7fffffffu) + k, (rec.other(i) >> 31) != 0, rec.levels(i));
  if (rec.degree() > 6) {
    const int p0 = m.ne_ptr[n];
    for (int p = p0 + 6; p < p0 + rec.degree(); p++) {
      const int4 q = m.ne4[p];
      f((cix)(q.x >> 1) * m.S + k, (cix)q.w + k, (q.x & 1) != 0, q.z);
    }
  }
}

// PPM weights of one column level (lib/oce_adv_tra_ver.F90:525-553): c1, c2, c3
// of layer k's slope, and A .. E of the value at interface k (between layers
// k - 1 and k) from the thicknesses h[-2 .. 1] around it.
template <typename R>
__device__ __forceinline__ void ppm_slope_weights(R hm, R h, R hp, R *c) {
  c[0] = h / (hm + h + hp);
  c[1] = (R(2) * hm + h) / (hp + h);
  c[2] = (h + R(2) * hp) / (hm + h);
}
template <typename R>
__device__ __forceinline__ void ppm_face_weights(R dzjm1, R dzj, R dzjp1, R dzjp2, R *c) {
  c[0] = dzj / (dzj + dzjp1);
  c[1] = R(1) / (dzjm1 + dzj + dzjp1 + dzjp2);
  c[2] = (R(2) * dzjp1 * dzj) / (dzj + dzjp1) *
         ((dzjm1 + dzj) / (R(2) * dzj + dzjp1) - (dzjp2 + dzjp1) / (R(2) * dzjp1 + dzj));
  c[3] = dzj * (dzjm1 + dzj) / (R(2) * dzj + dzjp1);
  c[4] = dzjp1 * (dzjp1 + dzjp2) / (dzj + R(2) * dzjp1);
}

// Level tables (DMeshT::ltab), S entries each, where every column has the same
// thicknesses (uniform z levels): the PPM weights, 1/hnode, and for any mesh
// QR4C's level distances, their reciprocal and its two offsets.
enum { LT_C1 = 0, LT_C2, LT_C3, LT_A, LT_B, LT_C, LT_D, LT_E, LT_YH, LT_ZD, LT_YZD, LT_ZA, LT_ZB, LT_COUNT };
template <typename R>
__global__ void k_level_tables(DMeshT<R> m, int n, R *t) {
  const int S = m.S;
  const R *HN = m.hnode_new + (size_t)n * S, *H = m.hnode + (size_t)n * S;
  const int nln = m.nlev_node[n] - 1;
  for (int k = threadIdx.x; k < S; k += blockDim.x) {
    R c[3] = {0, 0, 0}, f[5] = {0, 0, 0, 0, 0};
    if (m.uniform_h && k >= 1 && k <= nln - 2) ppm_slope_weights(HN[k - 1], HN[k], HN[k + 1], c);
    if (m.uniform_h && k >= 2 && k <= nln - 2) ppm_face_weights(HN[k - 2], HN[k - 1], HN[k], HN[k + 1], f);
    for (int i = 0; i < 3; i++) t[(LT_C1 + i) * S + k] = c[i];
    for (int i = 0; i < 5; i++) t[(LT_A + i) * S + k] = f[i];
    // NaN: a thickness that div_fast has no quotient for (k_col1 divides again)
    constexpr R big = sizeof(R) == 8 ? R(0x1p500) : R(0x1p60f);
    const R h = m.uniform_h && k < nln ? H[k] : R(1);
    t[LT_YH * S + k] = fabs(h) >= 1 / big && fabs(h) <= big ? (k < nln ? R(1) / h : R(0)) : R(NAN);
    const bool in = k >= 1 && k < m.nl - 1;
    const R zd = in ? m.Z[k - 1] - m.Z[k] : R(1);
    t[LT_ZD * S + k] = zd;
    t[LT_YZD * S + k] = R(1) / zd;
    t[LT_ZA * S + k] = in ? m.zbar[k] - m.Z[k] : R(0);
    t[LT_ZB * S + k] = in ? m.zbar[k] - m.Z[k - 1] : R(0);
  }
}

// PPM slope of layer j (1-based) with the limiter of lib/oce_adv_tra_ver.F90:
// 525-540; c1, c2, c3 are the geometric factors of that layer.
template <typename R>
__device__ __forceinline__ R ppm_slope(R Tm1, R T0, R Tp1, R c1, R c2, R c3) {
  R d = c1 * (c2 * (Tp1 - T0) + c3 * (T0 - Tm1));
  if ((Tp1 - T0) * (T0 - Tm1) > R(0))
    d = fmin3(fabs(d), R(2) * fabs(Tp1 - T0), R(2) * fabs(T0 - Tm1)) * sgn1(d);
  else
    d = R(0);
  return d;
}
// PPM flux through an interface with velocity w (not zero) out of the layer of
// value Tc with face values aL, aR and Courant number x (lib/oce_adv_tra_ver.F90:
// 597-639); D divides by 6.
template <typename R, typename D>
__device__ __forceinline__ R ppm_face(R w, R Tc, R aL, R aR, R x, D div) {
  const R two3 = R(2.0 / 3.0);
  if ((aR - Tc) * (Tc - aL) <= R(0)) { aL = Tc; aR = Tc; }
  if ((aR - aL) * (Tc - R(0.5) * (aL + aR)) > div((aR - aL) * (aR - aL))) aL = R(3) * Tc - R(2) * aR;
  if ((aR - aL) * (Tc - R(0.5) * (aR + aL)) < -div((aR - aL) * (aR - aL))) aR = R(3) * Tc - R(2) * aL;
  const R aj = R(6) * (Tc - R(0.5) * (aL + aR));
  const R dn = (-aL - R(0.5) * x * (aR - aL + (R(1) - two3 * x) * aj));
  const R up = (-aR + R(0.5) * x * (aR - aL - (R(1) - two3 * x) * aj));
  return w > R(0) ? dn : up;
}

// vertical LO flux at interface k (0-based: top of layer k) of values Tk (layer
// k) and Tm (layer k - 1); adv_tra_ver_upw1 (lib/oce_adv_tra_ver.F90:300-327)
template <typename R>
__device__ __forceinline__ R upw_v(R Tk, R Tm, R w, R A, int k, int nln) {
  const R top = -(w * Tk * A);
  const R in = -(R(0.5) * (Tk * (w + fabs(w)) + Tm * (w - fabs(w))) * A);
  return k == 0 ? top : (k >= nln ? R(0) : in);
}

// The antidiffusive vertical fluxes of a pair's interfaces once more, level by
// level from memory with plain divisions (operands outside the fast divisions'
// range).
template <typename R, typename TS, int NT, int G, int VER, int LIM>
__device__ __noinline__ void col1_vert_slow(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t0, int n, int k0) {
  const cix col = (cix)n * m.S;
  const int nlev = m.nlev_node[n], nln = nlev - 1;
  const R *W = a.W + col, *A = m.area + col, *H = m.hnode + col, *HN = m.hnode_new + col;
#pragma unroll 1
  for (int k = k0; k < min(k0 + 2, nln); k++)
#pragma unroll 1
    for (int t = t0; t < t0 + G; t++) {
      auto T = [&](int j) { return ldT<R>(a.T[t], col + j, a.off[t]); };
      auto B = [&](int j) { return ldT<R>(a.TAB[t], col + j, a.off[t]); };
      const R lov = LIM == LIM_FCT ? upw_v(T(k), T(max(k - 1, 0)), W[k], A[k], k, nln) : R(0);
      R hov;
      if (VER == VER_PPM) {
        auto slope = [&](int j) {
          R c[3];
          ppm_slope_weights(HN[j - 1], HN[j], HN[j + 1], c);
          return ppm_slope(B(j - 1), B(j), B(j + 1), c[0], c[1], c[2]);
        };
        auto tv = [&](int j) {
          if (j == 0) return B(0);
          if (j == nln) return B(nln - 1);
          if (j == nln - 1) {
            const R s = sgn1(W[j]);
            return -B(j - 1) * fmin2(s, R(0)) + B(j) * fmax2(s, R(0));
          }
          if (j == 1) return R(0.5) * (B(0) + B(1));
          R c[5];
          ppm_face_weights(HN[j - 2], HN[j - 1], HN[j], HN[j + 1], c);
          const R T0 = B(j - 1), T1 = B(j);
          return T0 + c[0] * (T1 - T0) + c[1] * (c[2] * (T1 - T0) - c[3] * slope(j) + c[4] * slope(j - 1));
        };
        const R w = W[k];
        if (k == 0) {
          hov = -(tv(0) * w * A[0]) - lov;
        } else if (!(w > R(0)) && !(w < R(0))) {
          hov = R(0) - lov;
        } else {
          const int j = w > R(0) ? k : k - 1;
          const R d = w * a.dt / H[j];
          const R x = w > R(0) ? fmin2(d, R(1)) : fmin2(-d, R(1));
          hov = ppm_face(w, B(j), tv(j), tv(j + 1), x, [](R z) { return z / R(6); }) * A[k] * w - lov;
        }
      } else {
        Col<R, TS> c;
        c.T = a.TAB[t] + col; c.W = W; c.A = A; c.nlev = nlev; c.off = a.off[t];
        hov = VER == VER_QR4C ? ver_qr4c(c, m.zbar, m.Z, k + 1, a.pv, lov)
                              : (VER == VER_CDIFF ? ver_cdiff(c, k + 1, lov) : ver_upw1(c, k + 1) - lov);
      }
      il<NT>(a.adf_v, t, col + k) = hov;
    }
}

// ---------------------------------------------------------------------------
// k_col1: LO solution and vertical fluxes
// ---------------------------------------------------------------------------
// UNI: the mesh has uniform z levels and the level tables hold the PPM weights
// and reciprocal thicknesses; otherwise they are formed here.
template <typename R, typename TS, int NT, int G, int VER, int LIM, bool UNI>
__device__ __forceinline__ void col1_pair(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t0, const PairLane &l) {
  const int n = l.item, k = l.k(), S = m.S;
  const cix col = (cix)n * S, o = col + k;
  const NodeRec rec = node_rec(m, n);
  const int nln = rec.nlev() - 1;
  const int km = max(k - 1, 0), kp = min(k + 2, S - 1);
  R W[2], A[2];
  ldv2(a.W + o, W);
  ldv2(m.area + o, A);
  // values k - 1 .. k + 2 of valuesAB, and k - 1 .. k + 1 of the values
  R x[G][4], ts[G][3] = {};
#pragma unroll
  for (int t = 0; t < G; t++) {
    x[t][0] = ldT<R>(a.TAB[t0 + t], col + km, a.off[t0 + t]);
    ld_pair_T(a.TAB[t0 + t], o, a.off[t0 + t], x[t] + 1);
    x[t][3] = ldT<R>(a.TAB[t0 + t], col + kp, a.off[t0 + t]);
    if (LIM == LIM_FCT) {
      ts[t][0] = x[t][0];
      ts[t][1] = x[t][1];
      ts[t][2] = x[t][2];
      if (a.T[t0 + t] != a.TAB[t0 + t]) {
        ts[t][0] = ldT<R>(a.T[t0 + t], col + km, a.off[t0 + t]);
        ld_pair_T(a.T[t0 + t], o, a.off[t0 + t], ts[t] + 1);
      }
    }
  }
  if (k + 1 >= nln)  // the second level is dry, whatever its cell holds
#pragma unroll
    for (int t = 0; t < G; t++) x[t][2] = ts[t][2] = R(0);
  // horizontal LO gather (lib/oce_adv_tra_driver.F90:122-181): with the edge
  // flux's sign turned to point out of this node, both ends' contributions are
  // the same expression
  R acc[G][2];
  if (LIM == LIM_FCT) {
#pragma unroll
    for (int t = 0; t < G; t++) acc[t][0] = acc[t][1] = R(0);
    for_edges(m, n, k, rec, [&](cix oe, cix oo, bool second, int lev) {
      const bool w0 = k < lev, w1 = k + 1 < lev;
      R v[2], to[G][2];
      ldv2_if(a.vflux + oe, w0, v);
#pragma unroll
      for (int t = 0; t < G; t++) ld_pair_T_if(a.T[t0 + t], oo, a.off[t0 + t], w0, to[t]);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const R vo = second ? -v[q] : v[q];
        const R vp = vo + fabs(vo), vm = vo - fabs(vo);
#pragma unroll
        for (int t = 0; t < G; t++) {
          const R F = R(-0.5) * (ts[t][1 + q] * vp + to[t][q] * vm);
          acc[t][q] = acc[t][q] + (q == 0 ? F : (w1 ? F : R(0)));
        }
      }
    });
  }

  PairBad bad(k + 1 < nln);
  R hov[2 * G], lov[G][2];
#pragma unroll
  for (int t = 0; t < G; t++)
#pragma unroll
    for (int q = 0; q < 2; q++)
      lov[t][q] = LIM == LIM_FCT ? upw_v(ts[t][1 + q], ts[t][q], W[q], A[q], k + q, nln) : R(0);
  if constexpr (VER == VER_PPM) {
    R c1[2], c2[2], c3[2], fA[2], fB[2], fC[2], fD[2], fE[2], h[3], yh[3];
    if constexpr (UNI) {
      const R *lt = m.ltab + k;
      ldv2(lt + LT_C1 * S, c1); ldv2(lt + LT_C2 * S, c2); ldv2(lt + LT_C3 * S, c3);
      ldv2(lt + LT_A * S, fA); ldv2(lt + LT_B * S, fB); ldv2(lt + LT_C * S, fC);
      ldv2(lt + LT_D * S, fD); ldv2(lt + LT_E * S, fE);
      h[0] = m.hT[km]; ldv2(m.hT + k, h + 1);
      yh[0] = m.ltab[LT_YH * S + km]; ldv2(lt + LT_YH * S, yh + 1);
      bad.any = yh[0] != yh[0] || yh[1] != yh[1] || yh[2] != yh[2];
    } else {
      const R *HN = m.hnode_new + col, *H = m.hnode + col;
      const R z[5] = {HN[max(k - 2, 0)], HN[km], HN[k], HN[k + 1], HN[kp]};
#pragma unroll
      for (int q = 0; q < 2; q++) {
        R c[3], f[5];
        ppm_slope_weights(z[1 + q], z[2 + q], z[3 + q], c);
        ppm_face_weights(z[q], z[1 + q], z[2 + q], z[3 + q], f);
        c1[q] = c[0]; c2[q] = c[1]; c3[q] = c[2];
        fA[q] = f[0]; fB[q] = f[1]; fC[q] = f[2]; fD[q] = f[3]; fE[q] = f[4];
      }
      h[0] = H[km]; h[1] = H[k]; h[2] = H[k + 1];
    }
#pragma unroll
    for (int t = 0; t < G; t++) {
      R s[2], tv[4];
#pragma unroll
      for (int q = 0; q < 2; q++) s[q] = ppm_slope(x[t][q], x[t][q + 1], x[t][q + 2], c1[q], c2[q], c3[q]);
      const R sm = __shfl_up_sync(kFull, s[1], 1);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        // interface values (lib/oce_adv_tra_ver.F90:545-553 with nz = k + q)
        const int kk = k + q;
        const R T0 = x[t][q], T1 = x[t][q + 1];
        R v = T0 + fA[q] * (T1 - T0) + fB[q] * (fC[q] * (T1 - T0) - fD[q] * s[q] + fE[q] * (q == 0 ? sm : s[0]));
        if (kk == 1) v = R(0.5) * (T0 + T1);
        const R sg = sgn1(W[q]);
        if (kk == nln - 1) v = -T0 * fmin2(sg, R(0)) + T1 * fmax2(sg, R(0));
        if (kk == 0) v = T1;
        tv[1 + q] = v;
      }
      tv[0] = __shfl_up_sync(kFull, tv[2], 1);
      tv[3] = __shfl_down_sync(kFull, tv[1], 1);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int kk = k + q;
        const R w = W[q];
        const bool pos = w > R(0);
        const R Tc = pos ? x[t][q + 1] : x[t][q];
        const R aL = pos ? tv[q + 1] : tv[q];
        const R aR = pos ? (kk == nln - 1 ? x[t][q + 1] : tv[q + 2]) : tv[q + 1];
        R d;
        if constexpr (UNI) d = div_fast(w * a.dt, pos ? h[q + 1] : h[q], pos ? yh[q + 1] : yh[q], bad[q]);
        else d = w * a.dt / (pos ? h[q + 1] : h[q]);
        const R cx = pos ? fmin2(d, R(1)) : fmin2(-d, R(1));
        const R f = ppm_face(w, Tc, aL, aR, cx, [&](R z) { return div6(z, bad[q]); });
        R v = f * A[q] * w - lov[t][q];
        if (!pos && !(w < R(0))) v = R(0) - lov[t][q];
        if (kk == 0) v = -(tv[1 + q] * w * A[q]) - lov[t][q];
        hov[2 * t + q] = kk >= nln ? R(0) : v;
      }
    }
  } else if constexpr (VER == VER_QR4C) {
    // lib/oce_adv_tra_ver.F90:397-436, the reference's assignments in order
    R zd[2], yz[2], za[2], zb[2];
    const R *lt = m.ltab + k;
    ldv2(lt + LT_ZD * S, zd); ldv2(lt + LT_YZD * S, yz); ldv2(lt + LT_ZA * S, za); ldv2(lt + LT_ZB * S, zb);
#pragma unroll
    for (int t = 0; t < G; t++) {
      R g[4];
#pragma unroll
      for (int q = 0; q < 2; q++) g[1 + q] = div_fast(x[t][q] - x[t][q + 1], zd[q], yz[q], bad[q]);
      g[0] = __shfl_up_sync(kFull, g[2], 1);
      g[3] = __shfl_down_sync(kFull, g[1], 1);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int kk = k + q;
        const R w = W[q], T0 = x[t][q], T1 = x[t][q + 1];
        R v = lov[t][q];
        const R mid = -(R(0.5) * (T0 + T1) * w * A[q]);
        if (kk == 0) v = -(T1 * w * A[q]) - v;
        if (kk == 1) v = mid - v;
        if (kk == nln - 1) v = mid - v;
        const R m1 = T1 + div3((R(2) * g[1 + q] + g[2 + q]) * za[q], bad[q]);
        const R m2 = T0 + div3((R(2) * g[1 + q] + g[q]) * zb[q], bad[q]);
        const R tm = (w + fabs(w)) * m1 + (w - fabs(w)) * m2;
        const R f = (-(R(0.5) * (R(1) - a.pv) * tm) - a.pv * (R(0.5) * (m1 + m2)) * w) * A[q] - v;
        if (kk >= 2 && kk <= nln - 2) v = f;
        hov[2 * t + q] = kk >= nln ? R(0) : v;
      }
    }
  } else {
#pragma unroll
    for (int t = 0; t < G; t++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int kk = k + q;
        const R T0 = x[t][q], T1 = x[t][q + 1];
        R v;
        if constexpr (VER == VER_CDIFF) {
          const R c = R(0.5) * (T0 + T1);
          v = (kk == 0 ? -(W[q] * T1 * A[q]) : -(c * W[q] * A[q])) - lov[t][q];
        } else {
          v = upw_v(T1, T0, W[q], A[q], kk, nln) - lov[t][q];
        }
        hov[2 * t + q] = kk >= nln ? R(0) : v;
      }
  }
  const bool st = l.stores();
  if (st) {
    st_pair_il<NT, G>(a.adf_v, t0, o, hov);
    if (k + 2 == nln)  // the bottom interface of a column of whole pairs
      for (int t = 0; t < G; t++) il<NT>(a.adf_v, t0 + t, o + 2) = R(0);
  }
  if constexpr (LIM == LIM_FCT) {
    // LO solution (lib/oce_adv_tra_driver.F90:202-211)
    R asv[2], yas[2], hn[2], yhn[2], h[2], out[2 * G];
    const cix oh = (cix)n * m.hS + k;
    ldv2(m.areasvol + o, asv);
    ldv2(m.rcp + o, yas);
    ldv2(m.hnT + oh, hn);
    ldv2(m.yhnT + oh, yhn);
    ldv2(m.hT + oh, h);
    PairBad badl(k + 1 < nln);
#pragma unroll
    for (int t = 0; t < G; t++) {
      const R dn = __shfl_down_sync(kFull, lov[t][0], 1);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const R f1 = q == 0 ? lov[t][1] : (k + 2 >= nln ? R(0) : dn);
        acc[t][q] = (acc[t][q] + (lov[t][q] - f1)) * a.dt;
        const R num = ts[t][1 + q] * h[q] + div_fast(acc[t][q], asv[q], yas[q], badl[q]);
        out[2 * t + q] = div_fast(num, hn[q], yhn[q], badl[q]);
      }
    }
    if (badl.any) {
      for (int t = 0; t < G; t++)
        for (int q = 0; q < 2; q++) out[2 * t + q] = (ts[t][1 + q] * h[q] + acc[t][q] / asv[q]) / hn[q];
    }
    if (st) st_pair_il<NT, G>(a.lo, t0, o, out);
  }
  if (st && bad.any) col1_vert_slow<R, TS, NT, G, VER, LIM>(m, a, t0, n, k);
}

// The column pairs of `per` consecutive warps of the schedule, one after the
// other; the next pair's map entry is loaded ahead.
template <typename R, typename F>
__device__ __forceinline__ void col_warps(const DMeshT<R> &m, int blk, int per, F f) {
  const DPairs &s = m.node_pairs;
  int warp = (blk * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5)) * per;
  const int end = min(warp + per, s.nwarps);
  if (warp >= end) return;
  PairLane nxt = pair_lane(s, warp);
  prefetch(m.nrec + nxt.item);
  prefetch(m.ne6 + 3 * (size_t)nxt.item);
  pdl_wait();
  do {
    const PairLane c = nxt;
    if (++warp < end) nxt = pair_lane(s, warp);
    f(c);
  } while (warp < end);
}

template <typename R, typename TS, int NT, int VER, int LIM, bool UNI>
__device__ __forceinline__ void col1_block(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int blk, int per) {
  constexpr int G = LaneTracers<R, NT>::col1;
  col_warps(m, blk, per, [&](const PairLane &l) {
#pragma unroll
    for (int t0 = 0; t0 < NT; t0 += G) col1_pair<R, TS, NT, G, VER, LIM, UNI>(m, a, t0, l);
  });
}
template <typename R, typename TS, int NT, int VER, int LIM, bool UNI>
__global__ void __launch_bounds__(kColThreads, StepBlocks<R, NT>::col1)
    k_col1(const __grid_constant__ DMeshT<R> m, const __grid_constant__ FusedArgs<R, TS> a, int per) {
  pdl_launch();
  col1_block<R, TS, NT, VER, LIM, UNI>(m, a, blockIdx.x, per);
}

// ---------------------------------------------------------------------------
// k_col2: bounds, in/out sums, ratios (lib/oce_adv_tra_fct.F90:105-374)
// ---------------------------------------------------------------------------
// Limiter ratios min(1, q / (P dt / V +- eps)), formed in FP64 in every precision:
// scale() once per cell, den() per sum, ratio() per bound.
//
// FP64: IEEE quotients, y the plane's RN(1 / V).
// FP32: the FP32 value nearest to the FP64 quotient's.  Reciprocals of two Newton steps
// and four roundings leave less than 2^-50 of relative error, so the FP32 rounding is
// the quotient's own unless the result lies within 64 ulp (2^-46) of the middle of two
// FP32 values: one in 2^22, which sets `bad` like results below 2^-126 and, through NaN,
// operands that are not finite.  (All quotients exact before their rounding: 3 % of a
// step of four tracers.)
template <typename R>
struct Ratio;
template <>
struct Ratio<double> {
  static __device__ __forceinline__ double scale(double, double, double y) { return y; }
  static __device__ __forceinline__ double den(double P, double dt, double V, double y, double eps, bool &bad) {
    return div_fast(P * dt, V, y, bad) + eps;
  }
  static __device__ __forceinline__ double ratio(double q, double den, bool &bad) { return fmin2(1.0, div_any(q, den, bad)); }
};
template <>
struct Ratio<float> {
  static __device__ __forceinline__ double scale(float dt, float V, float) { return (double)dt * rcp_newton((double)V); }
  static __device__ __forceinline__ double den(float P, float, float, double y, double eps, bool &) {
    return __fma_rn((double)P, y, eps);
  }
  static __device__ __forceinline__ float ratio(float q, double den, bool &bad) {
    const double r = (double)q * rcp_newton(den);
    const unsigned u = 2u * (unsigned)__double2hiint(r), lo = (unsigned)__double2loint(r);
    bad |= ((u - 0x70200000u > 0xffa00000u - 0x70200000u) && not_zero(r, u)) || (lo & 0x1fffffffu) - (0x10000000u - 64u) < 128u;
    return fmin2(1.0f, (float)r);
  }
};

// FCT bounds of one cell from the ring elements, for nodes whose ring list is
// incomplete (lib/oce_adv_tra_fct.F90:105-181).
template <typename R>
struct Bounds {
  R mx, mn;
};
template <typename R, typename TS, int NT>
__device__ __noinline__ Bounds<R> ring_bounds(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t, int n, int k) {
  const R big = R(1e3);
  Bounds<R> b{R(0), R(0)};
  const int p0 = m.ring_ptr[n], p1 = m.ring_ptr[n + 1];
#pragma unroll 1
  for (int p = p0; p < p1; p++) {
    const int el = m.ring_elem[p];
    R hi = -big, lw = big;
    if (k < m.nlev_elem[el] - 1) {
      const int *en = m.elem_nodes + 3 * (size_t)el;
      R h[3], l[3];
      for (int q = 0; q < 3; q++) {
        const cix o = (cix)en[q] * m.S + k;
        const R lv = il<NT>(a.lo, t, o), tv = ldT<R>(a.T[t], o, a.off[t]);
        h[q] = fmax2(lv, tv);
        l[q] = fmin2(lv, tv);
      }
      hi = fmax3(h[0], h[1], h[2]);
      lw = fmin3(l[0], l[1], l[2]);
    }
    b.mx = p == p0 ? hi : fmax2(b.mx, hi);
    b.mn = p == p0 ? lw : fmin2(b.mn, lw);
  }
  return b;
}

template <typename R, typename TS, int NT, int G>
__device__ __forceinline__ void col2_pair(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t0, const PairLane &l) {
  const int n = l.item, k = l.k(), S = m.S;
  const cix o = (cix)n * S + k;
  const NodeRec rec = node_rec(m, n);
  const int nln = rec.nlev() - 1;
  const R big = R(1e3);
  R lo[2 * G], av[2 * G], mx[2 * G], mn[2 * G], fp[2 * G], fm[2 * G];
  ld_pair_il<NT, G>(a.lo, t0, o, lo);
  ld_pair_il<NT, G>(a.adf_v, t0, o, av);
#pragma unroll
  for (int t = 0; t < G; t++) {
    R tt[2];
    ld_pair_T(a.T[t0 + t], o, a.off[t0 + t], tt);
    // interface k + 2 (zero at the column's bottom)
    const R a2 = k + 2 < nln ? il<NT>(a.adf_v, t0 + t, o + 2) : R(0);
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = 2 * t + q;
      mx[i] = fmax2(lo[i], tt[q]);
      mn[i] = fmin2(lo[i], tt[q]);
      const R v0 = av[i], v1 = q == 0 ? av[i + 1] : a2;
      fp[i] = R(0) + (fmax2(R(0), v0) + fmax2(R(0), -v1));
      fm[i] = R(0) + (fmin2(R(0), v0) + fmin2(R(0), -v1));
    }
  }
  // in/out sums over the incident edges and, with a complete ring, the bounds:
  // the nodes of the ring elements wet at a level are the node itself and the
  // far ends of its edges wet there (each such edge has a wet triangle holding
  // both ends); max and min are exact, so these equal the per-element ones
  for_edges(m, n, k, rec, [&](cix oe, cix oo, bool second, int lev) {
    const bool w0 = k < lev, w1 = k + 1 < lev;
    R f[2 * G], l1[2 * G], t1[2 * G];
    ld_pair_il_if<NT, G>(a.adf_h, t0, oe, w0, f);
    ld_pair_il_if<NT, G>(a.lo, t0, oo, w0, l1);
#pragma unroll
    for (int t = 0; t < G; t++) ld_pair_T_if(a.T[t0 + t], oo, a.off[t0 + t], w0, t1 + 2 * t);
#pragma unroll
    for (int i = 0; i < 2 * G; i++) {
      const bool w = i % 2 == 0 ? w0 : w1;
      const R hi = fmax2(l1[i], t1[i]), lw = fmin2(l1[i], t1[i]);
      mx[i] = (w && hi > mx[i]) ? hi : mx[i];
      mn[i] = (w && lw < mn[i]) ? lw : mn[i];
      const R g = second ? -f[i] : f[i];  // zero where the edge is dry
      fp[i] = fp[i] + fmax2(R(0), g);
      fm[i] = fm[i] + fmin2(R(0), g);
    }
  });
  if (!rec.ring_full()) {
#pragma unroll
    for (int i = 0; i < 2 * G; i++) {
      const Bounds<R> b = ring_bounds<R, TS, NT>(m, a, t0 + i / 2, n, k + i % 2);
      mx[i] = b.mx;
      mn[i] = b.mn;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 2 * G; i++)
      if (k + i % 2 + 1 > rec.nlev_min() - 1) {  // a ring element is dry here: +-big enter the bounds
        mx[i] = fmax2(mx[i], -big);
        mn[i] = fmin2(mn[i], big);
      }
  }
  R asv[2], yas[2];
  ldv2(m.areasvol + o, asv);
  ldv2(m.rcp + o, yas);  // 1/areasvol plane (k_rcp_planes)
  if (k + 1 >= nln) asv[1] = yas[1] = R(1);  // dry
  const double yv[2] = {Ratio<R>::scale(a.dt, asv[0], yas[0]), Ratio<R>::scale(a.dt, asv[1], yas[1])};
  __syncwarp();
#pragma unroll
  for (int t = 0; t < G; t++) {
    // the layers above and below (lib/oce_adv_tra_fct.F90:183-229)
    const R mxu = __shfl_up_sync(kFull, mx[2 * t + 1], 1), mxd = __shfl_down_sync(kFull, mx[2 * t], 1);
    const R mnu = __shfl_up_sync(kFull, mn[2 * t + 1], 1), mnd = __shfl_down_sync(kFull, mn[2 * t], 1);
    R bx[2], bn[2], out[4];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = 2 * t + q, kk = k + q;
      const bool edge_lev = kk == 0 || kk == nln - 1;
      const R ux = q == 0 ? fmax3(mxu, mx[2 * t], mx[2 * t + 1]) : fmax3(mx[2 * t], mx[2 * t + 1], mxd);
      const R un = q == 0 ? fmin3(mnu, mn[2 * t], mn[2 * t + 1]) : fmin3(mn[2 * t], mn[2 * t + 1], mnd);
      bx[q] = (edge_lev ? mx[i] : ux) - lo[i];
      bn[q] = (edge_lev ? mn[i] : un) - lo[i];
    }
    // R+ = min(1, bmax / (P+ dt / V + eps)), R- likewise; flux_eps is a
    // default-real literal.  In FP32 the denominators, where cancellation with it
    // matters, and the quotients are formed in FP64 too.  A quotient of a positive
    // denominator not above bmax is at least 1: a lane where that holds of all its
    // quotients (limiting is local) does not divide in the FP32 kernels, which round
    // to FP32 (FP64: the test costs more than it saves, 0.277 against 0.258 ms at 400x400x64).
    const double eps = (double)1e-16f;
    PairBad bad(k + 1 < nln);
    bool need = false;
    double up[2], um[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = 2 * t + q;
      up[q] = Ratio<R>::den(fp[i], a.dt, asv[q], yv[q], eps, bad[q]);
      um[q] = Ratio<R>::den(fm[i], a.dt, asv[q], yv[q], -eps, bad[q]);
      out[2 * q] = out[2 * q + 1] = R(1);
      need |= k + q < nln && (!(up[q] > 0.0 && (double)bx[q] >= up[q]) || !(um[q] < 0.0 && (double)bn[q] <= um[q]));
    }
    if (sizeof(R) == 8 || need) {
#pragma unroll
      for (int q = 0; q < 2; q++) {
        out[2 * q] = Ratio<R>::ratio(bx[q], up[q], bad[q]);
        out[2 * q + 1] = Ratio<R>::ratio(bn[q], um[q], bad[q]);
      }
    }
    if (k + 1 >= nln) out[2] = out[3] = R(0);  // dry: read by k_col3 against a zero flux
    if (l.stores()) {
      stv4(a.rpm[t0 + t] + 2 * (size_t)o, out);
      if (bad.any) {
        for (int q = 0; q < 2; q++) {
          const int i = 2 * t + q;
          const double u = (double)fp[i] * (double)a.dt / (double)asv[q], v = (double)fm[i] * (double)a.dt / (double)asv[q];
          out[2 * q] = (R)fmin2(1.0, (double)bx[q] / (u + eps));
          out[2 * q + 1] = (R)fmin2(1.0, (double)bn[q] / (v - eps));
        }
        if (k + 1 >= nln) out[2] = out[3] = R(0);
        stv4(a.rpm[t0 + t] + 2 * (size_t)o, out);
      }
    }
  }
}

template <typename R, typename TS, int NT>
__device__ __forceinline__ void col2_block(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int blk, int per) {
  constexpr int G = LaneTracers<R, NT>::col2;
  col_warps(m, blk, per, [&](const PairLane &l) {
#pragma unroll
    for (int t0 = 0; t0 < NT; t0 += G) col2_pair<R, TS, NT, G>(m, a, t0, l);
  });
}
template <typename R, typename TS, int NT>
__global__ void __launch_bounds__(kColThreads, StepBlocks<R, NT>::col2)
    k_col2(const __grid_constant__ DMeshT<R> m, const __grid_constant__ FusedArgs<R, TS> a, int per) {
  pdl_launch();
  col2_block<R, TS, NT>(m, a, blockIdx.x, per);
}

// ---------------------------------------------------------------------------
// k_col3: limiting + flux2dtracer + update
// ---------------------------------------------------------------------------
// Reciprocals of the static cell geometry, 1/areasvol and 1/hnode_new, for
// the Markstein divisions of k_col1's LO solution, k_col2's ratio
// denominators and k_col3's update.
template <typename R>
__global__ void k_rcp_planes(DMeshT<R> m, R *rcp) {
  const size_t plane = (size_t)m.S * m.N;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < plane; q += (size_t)gridDim.x * blockDim.x) {
    const int n = (int)(q / m.S), k = (int)(q - (size_t)n * m.S);
    if (k >= m.nlev_node[n] - 1) continue;  // dry cells stay zero
    rcp[q] = R(1) / m.areasvol[q];
    rcp[plane + q] = R(1) / m.hnode_new[q];
  }
}

// limited vertical flux (lib/oce_adv_tra_fct.F90:396-427): ra = (R+, R-) of
// the layer above the interface, rh of the layer below it
template <typename R>
__device__ __forceinline__ R limit_v(R f, const R *ra, const R *rh, bool top) {
  const R p = top ? rh[0] : fmin2(ra[1], rh[0]);
  const R q = top ? rh[1] : fmin2(ra[0], rh[1]);
  return (f >= R(0) ? p : q) * f;
}

template <typename R, typename TS, int NT>
__device__ __forceinline__ void col3_store(const FusedArgs<R, TS> &a, int t, cix o, int wet, const R *v) {
  TS s[2];
#pragma unroll
  for (int q = 0; q < 2; q++)
    s[q] = stT<R, TS>(v[q], a.off[t], a.sround != 0, a.sround ? mix32(a.seed[t] ^ mix32((uint32_t)(o + q))) : 0u);
  if constexpr (std::is_same<R, TS>::value) {
    if (wet == 2) stv2(a.T_out[t] + o, v);
    else a.T_out[t][o] = s[0];
  } else {
    a.T_out[t][o] = s[0];
    if (wet == 2) a.T_out[t][o + 1] = s[1];
  }
  if (a.nonfinite) {
    const int c = !isfinite(v[0]) + (wet == 2 && !isfinite(v[1]));
    if (c) atomicAdd(a.nonfinite, (unsigned long long)c);
  }
}

// A pair's update with the divisions `div` (the fast ones, or plain ones again
// for the lanes whose operands lie outside their range).
template <typename R, typename TS, int NT, int G, int LIM, typename D>
__device__ __forceinline__ void col3_update(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t0, int n, int k, const NodeRec &rec,
                                            D div, R (*out)[2]) {
  const int S = m.S;
  const cix o = (cix)n * S + k, oh = (cix)n * m.hS + k;
  const int nln = rec.nlev() - 1;
  R asv[2], yas[2], hn[2], yhn[2], h[2], av[2 * G], lo[2 * G], dh[G][2], rs[G][4];
  ldv2(m.areasvol + o, asv);
  ldv2(m.rcp + o, yas);
  ldv2(m.hnT + oh, hn);
  ldv2(m.yhnT + oh, yhn);
  ld_pair_il<NT, G>(a.adf_v, t0, o, av);
  if (LIM == LIM_FCT) {
    ldv2(m.hT + oh, h);
    ld_pair_il<NT, G>(a.lo, t0, o, lo);
#pragma unroll
    for (int t = 0; t < G; t++) ldv4(a.rpm[t0 + t] + 2 * (size_t)o, rs[t]);
  }
#pragma unroll
  for (int t = 0; t < G; t++) dh[t][0] = dh[t][1] = R(0);
  for_edges(m, n, k, rec, [&](cix oe, cix oo, bool second, int lev) {
    const bool w0 = k < lev;
    R f[2 * G], ro[G][4];
    ld_pair_il_if<NT, G>(a.adf_h, t0, oe, w0, f);
    if (LIM == LIM_FCT)
#pragma unroll
      for (int t = 0; t < G; t++) ldv4_if(a.rpm[t0 + t] + 2 * (size_t)oo, w0, ro[t]);
#pragma unroll
    for (int t = 0; t < G; t++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        // flux into this node (zero where the edge is dry): positive ones are
        // limited by its R+ and the other node's R-, negative ones by the converse
        R g = second ? -f[2 * t + q] : f[2 * t + q];
        if (LIM == LIM_FCT) {
          const R p = fmin2(rs[t][2 * q], ro[t][2 * q + 1]), r = fmin2(rs[t][2 * q + 1], ro[t][2 * q]);
          g = (g >= R(0) ? p : r) * g;
        }
        dh[t][q] = dh[t][q] + div(g * a.dt, asv[q], yas[q]);
      }
  });
#pragma unroll
  for (int t = 0; t < G; t++) {
    R tt[2];
    ld_pair_T(a.T[t0 + t], o, a.off[t0 + t], tt);
    R fv[3];
    const R a2 = k + 2 < nln ? il<NT>(a.adf_v, t0 + t, o + 2) : R(0);
    if (LIM == LIM_FCT) {
      R ru[2] = {R(1), R(1)}, rd[2] = {R(1), R(1)};
      if (k > 0) ld_pair(a.rpm[t0 + t] + 2 * (size_t)(o - 1), ru[0], ru[1]);
      if (k + 2 < nln) ld_pair(a.rpm[t0 + t] + 2 * (size_t)(o + 2), rd[0], rd[1]);
      fv[0] = limit_v(av[2 * t], ru, rs[t], k == 0);
      fv[1] = limit_v(av[2 * t + 1], rs[t], rs[t] + 2, false);
      fv[2] = limit_v(a2, rs[t] + 2, rd, false);
    } else {
      fv[0] = av[2 * t];
      fv[1] = av[2 * t + 1];
      fv[2] = a2;
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      R dv = R(0);
      if (LIM == LIM_FCT) dv = dv - tt[q] * h[q] + lo[2 * t + q] * hn[q];
      dv = dv + div((fv[q] - fv[q + 1]) * a.dt, asv[q], yas[q]);
      R del = R(0) + dh[t][q] + dv;
      if (q == 1 && k + 1 >= nln) del = R(0);  // dry: its fluxes are zero, its cells hold anything
      out[t][q] = tt[q] + div(del, hn[q], yhn[q]);
    }
  }
}

template <typename R, typename TS, int NT, int G, int LIM>
__device__ __noinline__ void col3_pair_slow(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t0, int n, int k) {
  const NodeRec rec = node_rec(m, n);
  R out[G][2];
  col3_update<R, TS, NT, G, LIM>(m, a, t0, n, k, rec, [](R x, R y, R) { return x / y; }, out);
  for (int t = 0; t < G; t++) col3_store<R, TS, NT>(a, t0 + t, (cix)n * m.S + k, min(rec.nlev() - 1 - k, 2), out[t]);
}

template <typename R, typename TS, int NT, int G, int LIM>
__device__ __forceinline__ void col3_pair(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int t0, const PairLane &l) {
  if (!l.stores()) return;
  const int n = l.item, k = l.k();
  const NodeRec rec = node_rec(m, n);
  const int wet = min(rec.nlev() - 1 - k, 2);
  bool bad = false;
  R out[G][2];
  col3_update<R, TS, NT, G, LIM>(m, a, t0, n, k, rec, [&](R x, R y, R z) { return div_fast(x, y, z, bad); }, out);
  if (bad) {
    col3_pair_slow<R, TS, NT, G, LIM>(m, a, t0, n, k);
    return;
  }
#pragma unroll
  for (int t = 0; t < G; t++) col3_store<R, TS, NT>(a, t0 + t, (cix)n * m.S + k, wet, out[t]);
}

template <typename R, typename TS, int NT, int LIM>
__device__ __forceinline__ void col3_block(const DMeshT<R> &m, const FusedArgs<R, TS> &a, int blk, int per) {
  constexpr int G = LaneTracers<R, NT>::col3;
  col_warps(m, blk, per, [&](const PairLane &l) {
#pragma unroll
    for (int t0 = 0; t0 < NT; t0 += G) col3_pair<R, TS, NT, G, LIM>(m, a, t0, l);
  });
}
template <typename R, typename TS, int NT, int LIM>
__global__ void __launch_bounds__(kColThreads, StepBlocks<R, NT>::col3)
    k_col3(const __grid_constant__ DMeshT<R> m, const __grid_constant__ FusedArgs<R, TS> a, int per) {
  pdl_launch();
  col3_block<R, TS, NT, LIM>(m, a, blockIdx.x, per);
}

// dynamic shared memory of the cell-map kernels (the learned flux's training)
constexpr size_t smem_edge() { return sizeof(int) * (kMaxItemsPerBlock + 1 + kMaxCellsPerBlock + 1); }

FESOM_VARIANT_END
}  // namespace fesom
