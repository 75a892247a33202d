// Device self-tests of arithmetic primitives of the step kernels:
//  * the reciprocal-based correctly rounded division of the fused patch kernel:
//    div_rcp(a, b, 1/b) must return the bits of the IEEE quotient a / b for
//    every operand pair (Markstein's correction; see advect_fused.cuh);
//  * the straight-line divisions of the five step kernels (div_fast, div_any,
//    rcp_exact, div_3k): every result that is not flagged `bad` has the bits of the
//    IEEE quotient, the sign of a zero aside;
//  * the stochastic rounding of 16-bit tracer stores (advect_ops.cuh): every
//    result is one of the two storage neighbours of the input, and the
//    fraction rounded up matches (remainder / spacing) without bias.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/fesom_tracer.h"
#include "advect_fused.cuh"

namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t x) {  // splitmix64 finaliser
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// double with a random 52-bit mantissa, random sign and exponent in [lo, hi]
__device__ __forceinline__ double rand_double(uint64_t r, int lo, int hi) {
  const uint64_t mant = r & ((1ull << 52) - 1);
  const int e = lo + (int)((r >> 52) % (uint64_t)(hi - lo + 1));
  const uint64_t sign = (r >> 63) << 63;
  const uint64_t bits = sign | ((uint64_t)(e + 1023) << 52) | mant;
  return __longlong_as_double((long long)bits);
}

__global__ void k_div_check(long long n, uint64_t seed, unsigned long long *bad, double *first) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    const uint64_t r1 = mix64(seed ^ (uint64_t)(2 * i)), r2 = mix64(seed ^ (uint64_t)(2 * i + 1));
    double a, b;
    switch (i & 3) {
      case 0: a = rand_double(r1, -80, 80); b = rand_double(r2, -60, 60); break;       // general
      case 1: a = rand_double(r1, -40, 40); b = 6.0; break;                           // MUSCL /6
      case 2: a = rand_double(r1, -30, 50); b = fabs(rand_double(r2, 10, 30)); break;  // areas
      default: a = rand_double(r1, -30, 30); b = fabs(rand_double(r2, -4, 12)); break; // thicknesses
    }
    const double y = 1.0 / b;
    const double q = fesom::div_rcp(a, b, y), ref = a / b;
    if (__double_as_longlong(q) != __double_as_longlong(ref)) {
      unsigned long long k = atomicAdd(bad, 1ull);
      if (k == 0) { first[0] = a; first[1] = b; first[2] = q; first[3] = ref; }
    }
  }
}

// Operands of the straight-line divisions.  mode 0: ordinary (the flag must stay
// down); 1: exponents up to 4 beside the edges of the ranges that set the flag, and
// beyond the largest and smallest ones; 2: significands of all ones, or but a few of
// them, and powers of two; 3: subnormals of a few bits, zeros, infinities, NaN.
template <typename R> struct Bits;
template <> struct Bits<double> {
  using U = uint64_t;
  static constexpr int mant = 52, bias = 1023, emax = 2047;
  __device__ static double make(U u) { return __longlong_as_double((long long)u); }
  __device__ static U get(double x) { return (U)__double_as_longlong(x); }
};
template <> struct Bits<float> {
  using U = uint32_t;
  static constexpr int mant = 23, bias = 127, emax = 255;
  __device__ static float make(U u) { return __uint_as_float(u); }
  __device__ static U get(float x) { return __float_as_uint(x); }
};
template <typename R>
__device__ R special(uint64_t r, int mode, int lo, int hi, int edge) {
  using B = Bits<R>;
  using U = typename B::U;
  U m = (U)r & (((U)1 << B::mant) - 1);
  int e = lo + (int)((r >> 52) % (uint64_t)(hi - lo + 1));
  const uint64_t h = mix64(r);
  if (mode == 1) e = ((h >> 1) & 1 ? edge : -edge) + (int)((h >> 2) % 9) - 4;
  if (mode == 2) {
    const int few = (int)((h >> 8) % 4);
    m = few == 0 ? ((U)1 << B::mant) - 1 : (few == 1 ? ((U)1 << B::mant) - 1 - ((U)(h >> 16) & 7) : (few == 2 ? (U)(h >> 16) & 7 : (U)0));
  }
  int eb = e + B::bias;
  if (mode == 3) {
    const int kind = (int)(h % 8);
    eb = kind == 6 ? B::emax : 0;
    if (kind == 7) m = 0;
    else if (kind == 6) m = (h >> 32) & 1 ? m : 0;
    else m >>= (h >> 32) % B::mant;
  }
  eb = max(0, min(B::emax, eb));
  return B::make(((U)(r >> 63) << (B::mant + (sizeof(R) == 8 ? 11 : 8))) | ((U)eb << B::mant) | m);
}
template <typename R>
__device__ bool same_quotient(R q, R ref) {
  return Bits<R>::get(q) == Bits<R>::get(ref) || (q == R(0) && ref == R(0)) || (q != q && ref != ref);
}

enum { Q_DIV_FAST = 0, Q_DIV_ANY, Q_RCP, Q_DIV3, Q_DIV6, Q_RATIO, Q_COURANT, Q_SCALE, Q_COUNT };
// out: results that are neither flagged nor the quotient's bits; flagged results of
// ordinary operands
template <typename R>
__global__ void k_quotients(int kind, long long n, uint64_t seed, unsigned long long *out, double *first) {
  // edges of the flagged ranges (advect_fused.cuh): numerators of div_fast and
  // div_3k, divisors (and numerators of div_any)
  constexpr int ea = sizeof(R) == 8 ? 900 : 100, eb = sizeof(R) == 8 ? 500 : 60;
  constexpr int ord = sizeof(R) == 8 ? 80 : 40;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint64_t r1 = mix64(seed ^ (uint64_t)(2 * i)), r2 = mix64(seed ^ (uint64_t)(2 * i + 1));
    const int ma = (int)(i & 3), mb = (int)((i >> 2) & 3);
    bool bad = false, plain = ma == 0 && mb == 0;
    R a = special<R>(r1, ma, -ord, ord, kind == Q_DIV_ANY ? eb : ea), b, q, ref;
    switch (kind) {
      case Q_DIV_FAST:
        // divisors that leave the quotient of an unflagged numerator normal
        b = special<R>(r2, mb & 2, -20, 20, 0);
        plain = ma == 0;
        q = fesom::div_fast(a, b, R(1) / b, bad);
        ref = a / b;
        break;
      case Q_DIV_ANY:
        b = special<R>(r2, mb, -ord, ord, eb);
        q = fesom::div_any(a, b, bad);
        ref = a / b;
        break;
      case Q_RCP:
        b = special<R>(r2, mb, -ord, ord, eb);
        a = R(1);
        plain = mb == 0;
        q = fesom::rcp_exact(b, bad);
        ref = R(1) / b;
        break;
      case Q_DIV3:
        b = R(3);
        plain = ma == 0;
        q = fesom::div3(a, bad);
        ref = a / b;
        break;
      case Q_DIV6:
        b = R(6);
        plain = ma == 0;
        q = fesom::div6(a, bad);
        ref = a / b;
        break;
      case Q_RATIO: {
        // min(1, a / (P dt / V + eps)) of values in the model's range: P and V of
        // any significand, bounds from 2^-40 to 2 times the denominator
        const double eps = (double)1e-16f;
        const R dt = (R)(100.0 + (double)(r1 % 1000));
        const R P = fabs(special<R>(r1, ma == 3 ? 3 : 0, -60, 30, 0)), V = fabs(special<R>(r2, mb & 2, 10, 40, 0));
        const double den = (double)P * (double)dt / (double)V + eps;
        a = (R)(den * ldexp(1.0 + (double)(mix64(r1) >> 12) * 0x1p-52, -(int)(mix64(r2) % 41)));
        b = V;
        const double y = fesom::Ratio<R>::scale(dt, V, R(1) / V);
        if (ma == 2 && mb == 3) a = R(mix64(r2) & 1 ? -INFINITY : INFINITY);
        q = fesom::Ratio<R>::ratio(a, fesom::Ratio<R>::den(P, dt, V, y, eps, bad), bad);
        ref = (R)fesom::fmin2(1.0, (double)a / den);
        break;
      }
      default:
        // the learned flux's Courant number and reciprocal variation (FP32 only)
        if constexpr (sizeof(R) == 4) {
          if (kind == Q_COURANT) {
            b = fabsf(special<float>(r2, mb & 2, 10, 50, 0));
            a = special<float>(r1, 0, -30, 30, 0);
            q = fesom::edge_courant(a, 600.0f, b, fesom::FeatFast{bad});
            ref = fminf(fabsf(a) * 600.0f / b, 4.0f);
          } else {
            b = fabsf(special<float>(r2, mb, -66, 30, 100));
            a = 1.0f;
            q = fesom::FeatFast{bad}.rcp(b);
            ref = 1.0f / b;
          }
          plain = mb == 0;
        } else {
          a = b = q = ref = R(0);
        }
        break;
    }
    if (bad && plain) atomicAdd(&out[1], 1ull);
    if (!bad && !same_quotient(q, ref) && atomicAdd(&out[0], 1ull) == 0) {
      first[0] = a; first[1] = b; first[2] = q; first[3] = ref;
    }
  }
}

// storage neighbours of x toward zero (lo) and away from zero (hi)
__device__ __forceinline__ void nbrs_bf16(float x, float &lo, float &hi) {
  const uint32_t u = __float_as_uint(x) & 0xffff0000u;
  lo = __uint_as_float(u);
  hi = __uint_as_float(u + 0x10000u);
}
__device__ __forceinline__ void nbrs_f16(float x, float &lo, float &hi) {
  const __half l = __float2half_rz(x);
  lo = __half2float(l);
  hi = __half2float(__ushort_as_half((unsigned short)(__half_as_ushort(l) + 1)));
}

// fmt 0: BF16, 1: FP16.  Per input: `draws` roundings with the kernels'
// stream (per-step seed word, per-cell index); counts results outside
// {lo, hi} and accumulates (ups - draws p) and draws p (1 - p).
__global__ void k_sround_check(int fmt, long long n, int draws, uint32_t seed, unsigned long long *bad,
                               double *acc) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  double dev = 0.0, var = 0.0;
  for (; i < n; i += stride) {
    const uint64_t r = mix64((uint64_t)seed * 0x100000001ull ^ (uint64_t)i);
    // magnitudes 2^-6 .. 2^10 with random sign; one input in 16 exactly
    // representable in the format
    float x = ldexpf(1.0f + (float)(r & 0xffffff) * 0x1p-24f, (int)((r >> 24) % 16) - 6);
    if ((r >> 40) & 1) x = -x;
    float lo, hi;
    if (fmt == 0) nbrs_bf16(x, lo, hi);
    else nbrs_f16(x, lo, hi);
    if (((r >> 44) & 15) == 0) x = lo;
    const float gap = fabsf(hi - lo), rem = fabsf(x - lo);
    const double p = (double)rem / (double)gap;
    int ups = 0;
    for (int d = 0; d < draws; d++) {
      const uint32_t step_seed = fesom::mix32(seed + 0x9e3779b9u * (uint32_t)d);
      const uint32_t word = fesom::mix32(step_seed ^ fesom::mix32((uint32_t)i));
      const float y = fmt == 0 ? __bfloat162float(fesom::bf16_sround(x, word))
                               : __half2float(fesom::f16_sround(x, word));
      if (y == hi && rem > 0.0f) ups++;
      else if (y != lo) atomicAdd(bad, 1ull);
    }
    dev += (double)ups - draws * p;
    var += draws * p * (1.0 - p);
  }
  atomicAdd(&acc[0], dev);
  atomicAdd(&acc[1], var);
}

}  // namespace

extern "C" int tracer_selftest_sround(int fmt, long long n, int draws, uint32_t seed, long long *outside,
                                      double *z) {
  if (fmt < 0 || fmt > 1 || n < 1 || draws < 1) return -1;
  unsigned long long *d_bad = nullptr;
  double *d_acc = nullptr;
  if (cudaMalloc(&d_bad, sizeof(unsigned long long)) != cudaSuccess) return -1;
  if (cudaMalloc(&d_acc, 2 * sizeof(double)) != cudaSuccess) { cudaFree(d_bad); return -1; }
  cudaMemset(d_bad, 0, sizeof(unsigned long long));
  cudaMemset(d_acc, 0, 2 * sizeof(double));
  k_sround_check<<<148 * 4, 256>>>(fmt, n, draws, seed, d_bad, d_acc);
  cudaError_t e = cudaDeviceSynchronize();
  unsigned long long bad = 0;
  double acc[2] = {0, 0};
  if (e == cudaSuccess) {
    cudaMemcpy(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost);
    cudaMemcpy(acc, d_acc, sizeof(acc), cudaMemcpyDeviceToHost);
  }
  cudaFree(d_bad);
  cudaFree(d_acc);
  if (e != cudaSuccess) return -1;
  if (outside) *outside = (long long)bad;
  if (z) *z = acc[1] > 0.0 ? acc[0] / sqrt(acc[1]) : 0.0;
  return 0;
}

extern "C" int tracer_selftest_quotients(int kind, int fp32, long long n, uint64_t seed, long long *wrong, long long *flagged,
                                         double *example4) {
  if (kind < 0 || kind >= Q_COUNT || n < 1) return -1;
  unsigned long long *d = nullptr, h[2] = {0, 0};
  double *d_first = nullptr, first[4] = {0, 0, 0, 0};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return -1;
  if (cudaMalloc(&d_first, sizeof(first)) != cudaSuccess) { cudaFree(d); return -1; }
  cudaMemset(d, 0, sizeof(h));
  cudaMemset(d_first, 0, sizeof(first));
  if (fp32) k_quotients<float><<<148 * 8, 256>>>(kind, n, seed, d, d_first);
  else k_quotients<double><<<148 * 8, 256>>>(kind, n, seed, d, d_first);
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(first, d_first, sizeof(first), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(d_first);
  if (e != cudaSuccess) return -1;
  if (wrong) *wrong = (long long)h[0];
  if (flagged) *flagged = (long long)h[1];
  if (example4)
    for (int k = 0; k < 4; k++) example4[k] = first[k];
  return 0;
}

extern "C" int tracer_selftest_division(long long n, uint64_t seed, long long *mismatches, double *example4) {
  unsigned long long *d_bad = nullptr;
  double *d_first = nullptr;
  if (cudaMalloc(&d_bad, sizeof(unsigned long long)) != cudaSuccess) return -1;
  if (cudaMalloc(&d_first, 4 * sizeof(double)) != cudaSuccess) { cudaFree(d_bad); return -1; }
  cudaMemset(d_bad, 0, sizeof(unsigned long long));
  cudaMemset(d_first, 0, 4 * sizeof(double));
  k_div_check<<<148 * 8, 256>>>(n, seed, d_bad, d_first);
  cudaError_t e = cudaDeviceSynchronize();
  unsigned long long bad = 0;
  double first[4] = {0, 0, 0, 0};
  if (e == cudaSuccess) {
    cudaMemcpy(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost);
    cudaMemcpy(first, d_first, sizeof(first), cudaMemcpyDeviceToHost);
  }
  cudaFree(d_bad);
  cudaFree(d_first);
  if (e != cudaSuccess) return -1;
  if (mismatches) *mismatches = (long long)bad;
  if (example4)
    for (int k = 0; k < 4; k++) example4[k] = first[k];
  return 0;
}
