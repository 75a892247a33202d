// Level pairs: the unit of work of the step kernels.  A lane handles two
// consecutive levels (k even, k and k + 1) of one column or edge, so that
// every field access is one vector load of both levels and the per-column or
// per-edge data are fetched once for the two.  Columns are padded to a level
// stride that is a multiple of 4, so a pair never leaves its column; the
// second level of a pair may be dry (its results are discarded or predicated).
#pragma once
#include <type_traits>

#include "advect_ops.cuh"

namespace fesom {
FESOM_VARIANT_BEGIN

// ---- vector accesses of 2, 4 or 8 consecutive values ------------------------
// Four doubles are one 32-byte access on sm_100 (PTX ld/st .v4.f64), eight
// floats two of 16 bytes (the same bytes a cycle from L1; CUDA 12.9's ptxas fails on
// some kernels with .v8.f32).  The address is a multiple of the access size.
// The asm forms are volatile,
// so they stay between the barriers they are written between, and carry no
// memory clobber, so that plain loads move across them.
__device__ __forceinline__ void ldv2(const double *p, double *v) {
  const double2 a = *reinterpret_cast<const double2 *>(p);
  v[0] = a.x; v[1] = a.y;
}
__device__ __forceinline__ void ldv2(const float *p, float *v) {
  const float2 a = *reinterpret_cast<const float2 *>(p);
  v[0] = a.x; v[1] = a.y;
}
__device__ __forceinline__ void stv2(double *p, const double *v) { *reinterpret_cast<double2 *>(p) = make_double2(v[0], v[1]); }
__device__ __forceinline__ void stv2(float *p, const float *v) { *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]); }
__device__ __forceinline__ void ldv4(const double *p, double *v) {
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
               : "l"(p));
}
__device__ __forceinline__ void ldv4(const float *p, float *v) {
  const float4 a = *reinterpret_cast<const float4 *>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void stv4(double *p, const double *v) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]));
}
__device__ __forceinline__ void stv4(float *p, const float *v) {
  *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
template <typename R>
__device__ __forceinline__ void ldv8(const R *p, R *v) {
  ldv4(p, v);
  ldv4(p + 4, v + 4);
}
template <typename R>
__device__ __forceinline__ void stv8(R *p, const R *v) {
  stv4(p, v);
  stv4(p + 4, v + 4);
}

// Work arrays of a batch of NT tracers (adf_h, adf_v, lo): level pairs of all
// tracers side by side, the value of tracer t at cell o (o even for the first
// level of a pair) at [(o - o % 2) NT + 2 t + o % 2].  A lane's pairs of G
// consecutive tracers from t are 2 G consecutive values, v[2 i + level].
template <int NT>
__device__ __forceinline__ size_t il_at(int t, cix o) {
  return (size_t)(o & ~1u) * NT + 2 * t + (o & 1u);
}
template <int NT, typename R>
__device__ __forceinline__ R &il(R *x0, int t, cix o) {
  return x0[il_at<NT>(t, o)];
}
template <int NT, int G, typename R>
__device__ __forceinline__ void ld_pair_il(const R *x0, int t, cix o, R *v) {
  const R *p = x0 + (size_t)o * NT + 2 * t;
  if constexpr (G == 1) ldv2(p, v);
  else if constexpr (G == 2) ldv4(p, v);
  else ldv8(p, v);
}
template <int NT, int G, typename R>
__device__ __forceinline__ void st_pair_il(R *x0, int t, cix o, const R *v) {
  R *p = x0 + (size_t)o * NT + 2 * t;
  if constexpr (G == 1) stv2(p, v);
  else if constexpr (G == 2) stv4(p, v);
  else stv8(p, v);
}

// Pair of a tracer's storage column, as R.
template <typename R, typename TS>
__device__ __forceinline__ void ld_pair_T(const TS *p, cix o, R off, R *v) {
  if constexpr (std::is_same<R, TS>::value) {
    (void)off;
    ldv2(p + o, v);
  } else if constexpr (std::is_same<TS, f64u>::value) {
    (void)off;
    v[0] = p[o].v;
    v[1] = p[o + 1].v;
  } else if constexpr (std::is_same<TS, __nv_bfloat16>::value) {
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162 *>(p + o);
    v[0] = R(__low2bfloat16(a)) + off;
    v[1] = R(__high2bfloat16(a)) + off;
  } else {
    const __half2 a = *reinterpret_cast<const __half2 *>(p + o);
    v[0] = R(__low2half(a)) + off;
    v[1] = R(__high2half(a)) + off;
  }
}
// The same, zero without an access where `on` is false (predicated, no branch).
__device__ __forceinline__ void ldv2_if(const double *p, bool on, double *v) {
  asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %3, 0;\nmov.f64 %0, 0d0000000000000000;\nmov.f64 %1, 0d0000000000000000;\n"
               "@q ld.global.v2.f64 {%0, %1}, [%2];\n}"
               : "=&d"(v[0]), "=&d"(v[1])
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ldv2_if(const float *p, bool on, float *v) {
  asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %3, 0;\nmov.f32 %0, 0f00000000;\nmov.f32 %1, 0f00000000;\n"
               "@q ld.global.v2.f32 {%0, %1}, [%2];\n}"
               : "=&f"(v[0]), "=&f"(v[1])
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ldv4_if(const double *p, bool on, double *v) {
  asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %5, 0;\nmov.f64 %0, 0d0000000000000000;\nmov.f64 %1, 0d0000000000000000;\n"
               "mov.f64 %2, 0d0000000000000000;\nmov.f64 %3, 0d0000000000000000;\n"
               "@q ld.global.v4.f64 {%0, %1, %2, %3}, [%4];\n}"
               : "=&d"(v[0]), "=&d"(v[1]), "=&d"(v[2]), "=&d"(v[3])
               : "l"(p), "r"((int)on));
}
__device__ __forceinline__ void ldv4_if(const float *p, bool on, float *v) {
  asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %5, 0;\nmov.f32 %0, 0f00000000;\nmov.f32 %1, 0f00000000;\n"
               "mov.f32 %2, 0f00000000;\nmov.f32 %3, 0f00000000;\n@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
               : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3])
               : "l"(p), "r"((int)on));
}
template <int NT, int G, typename R>
__device__ __forceinline__ void ld_pair_il_if(const R *x0, int t, cix o, bool on, R *v) {
  const R *p = x0 + (size_t)o * NT + 2 * t;
  if constexpr (G == 1) ldv2_if(p, on, v);
  else ldv4_if(p, on, v);
  if constexpr (G == 4) ldv4_if(p + 4, on, v + 4);
}
template <typename R, typename TS>
__device__ __forceinline__ void ld_pair_T_if(const TS *p, cix o, R off, bool on, R *v) {
  if constexpr (std::is_same<R, TS>::value) {
    (void)off;
    ldv2_if(p + o, on, v);
  } else if constexpr (std::is_same<TS, f64u>::value) {
    (void)off;
    v[0] = on ? p[o].v : 0.0;
    v[1] = on ? p[o + 1].v : 0.0;
  } else {
    unsigned b;
    asm volatile("{\n.reg .pred q;\nsetp.ne.b32 q, %2, 0;\nmov.b32 %0, 0;\n@q ld.global.b32 %0, [%1];\n}"
                 : "=&r"(b)
                 : "l"(p + o), "r"((int)on));
    if constexpr (std::is_same<TS, __nv_bfloat16>::value) {
      v[0] = __uint_as_float(b << 16) + off;
      v[1] = __uint_as_float(b & 0xffff0000u) + off;
    } else {
      const __half2 h = *reinterpret_cast<const __half2 *>(&b);
      v[0] = __low2float(h) + off;
      v[1] = __high2float(h) + off;
    }
  }
}

// A lane's entry of a pair schedule (DPairs in dmesh.hpp).  Lanes without a
// pair hold some item and level 0.
struct PairLane {
  int item;
  unsigned code;
  __device__ __forceinline__ bool on() const { return code != kPairNone; }
  __device__ __forceinline__ bool stores() const { return code < kPairHalo; }
  __device__ __forceinline__ bool ring() const { return (code & kPairRing) != 0; }
  __device__ __forceinline__ int k() const { return on() ? (int)(code & kPairLevel) : 0; }
};
__device__ __forceinline__ PairLane pair_lane(const DPairs &s, int warp) {
  const int i = warp * 32 + (int)(threadIdx.x & 31);
  return PairLane{s.item[i], s.lev[i]};
}

FESOM_VARIANT_END
}  // namespace fesom
