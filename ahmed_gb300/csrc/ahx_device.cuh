// Device-side primitives shared by the assembly and product kernels.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ahx {

constexpr double kFourPi = 4.0 * 3.14159265358979323846;

// Collocation points in permuted (cluster) order, structure of arrays.
struct PointsSoA {
  const double* x;
  const double* y;
  const double* z;
};

// FP32 image of a double times 2^-shift, truncated, by integer operations (the
// conversion instruction shares the FP64 pipe); 0 below FP32's range
__device__ __forceinline__ float to_f32(double x, int shift) {
  const int hi = __double2hiint(x);
  const int f = (hi >> 20) & 0x7ff, e = f - shift - 896;
  if (f == 0 || e <= 0) return 0.f;
  const uint32_t m = __funnelshift_l((uint32_t)__double2loint(x), (uint32_t)hi & 0xfffffu, 3);
  return __int_as_float((hi & 0x80000000) | (e << 23) | (int)(m & 0x7fffffu));
}
// a normal FP32 number as a double
__device__ __forceinline__ double to_f64(float f) {
  const int b = __float_as_int(f);
  return __hiloint2double((b & 0x80000000) | (int)((((uint32_t)b & 0x7fffffffu) >> 3) + 0x38000000u), b << 29);
}
__device__ __forceinline__ float rsqrt_f32(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ bool f32_range(double x) {  // 2^-120 <= x < 2^120
  return (uint32_t)(__double2hiint(x) - ((1023 - 120) << 20)) < (uint32_t)(240 << 20);
}
// 1 / sqrt(x) for f32_range(x): an FP32 seed y (relative error e < 2^-20) and one step
// of Halley's series y (1 + e/2 + 3 e^2/8), remainder below 2^-61
__device__ __forceinline__ double rsqrt_seeded(double x) {
  const double y = to_f64(rsqrt_f32(to_f32(x, 0)));
  const double e = fma(-x, y * y, 1.0);  // y * y is exact (24-bit y)
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// r = sqrt(r2) and s = 1 / (4 pi r), every operation rounded to nearest, so that entries
// equal the host's bit for bit.  One reciprocal square root serves both, by the final steps
// r + (r2 - r^2) y / 2 and z + z (1 - t z) (Markstein).
//   root: before its last rounding within 2^-102.  Arguments X 2^q whose root lies closer to
//     the middle of two doubles have M^2 = X 2^q + c with M odd of 54 bits, |c| < 95: 37 in
//     all, which all round right.
//   reciprocal: z is off by up to 2.6 2^-53, the result before rounding by its square; that
//     rounds wrong for some t (T M = 2^106 - 2: T = 5276938686109394).  So the remainder 1 -
//     t s, which is exact, is looked at: below half a unit of s times t (by its high word, one
//     in 2^18 is not) s is the rounded one, otherwise the division decides.
// 22 FP64 instructions an entry; with the mirror images written by the same task, the dense
// leaves of 65,536 points take 2.7 ms instead of 5.1.  (The general case is a function of
// its own: predicated in line its FP64 instructions would occupy the pipe for every entry.)
static __device__ __noinline__ double2 rounded_r_s_any(double r2) {
  const double r = __dsqrt_rn(r2);
  return make_double2(r, __ddiv_rn(1.0, __dmul_rn(kFourPi, r)));
}
static __device__ __noinline__ double reciprocal_rounded(double t) { return __ddiv_rn(1.0, t); }
__device__ __forceinline__ void rounded_r_s(double r2, double& r, double& s) {
  if (f32_range(r2)) {
    const double y = rsqrt_seeded(r2), g = __dmul_rn(r2, y);
    r = fma(fma(-g, g, r2), 0.5 * y, g);
    const double t = __dmul_rn(kFourPi, r), z = __dmul_rn(1.0 / kFourPi, y);
    s = fma(z, fma(-t, z, 1.0), z);
    const int left = __double2hiint(fma(-t, s, 1.0)) & 0x7fffffff;
    const int half = __double2hiint(t) + (__double2hiint(s) & 0x7ff00000) - ((1023 + 53) << 20);  // t ulp(s) / 2
    if (left >= half) s = reciprocal_rounded(t);
  } else {
    const double2 v = rounded_r_s_any(r2);
    r = v.x;
    s = v.y;
  }
}
static __device__ __noinline__ double rsqrt_other(double x) { return rsqrt(x); }
__device__ __forceinline__ double rsqrt_any(double x) { return f32_range(x) ? rsqrt_seeded(x) : rsqrt_other(x); }
__device__ __forceinline__ double rounded_r2(double xi, double yi, double zi, double xj, double yj, double zj) {
  const double dx = __dsub_rn(xi, xj), dy = __dsub_rn(yi, yj), dz = __dsub_rn(zi, zj);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Laplace single-layer entry K(i,j) = 1/(4 pi |x_i - x_j|), diag = 1/(4 pi h).
__device__ __forceinline__ double lap_entry(const PointsSoA& P, uint32_t i, uint32_t j,
                                            double xi, double yi, double zi, double diag) {
  if (i == j) return diag;
  double r, s;
  rounded_r_s(rounded_r2(xi, yi, zi, P.x[j], P.y[j], P.z[j]), r, s);
  return s;
}

// a > b for non-negative doubles, on the integer pipe (IEEE order of the bit patterns)
__device__ __forceinline__ bool gt_nonneg(double a, double b) {
  return __double_as_longlong(a) > __double_as_longlong(b);
}

// ---------------------------------------------------------------------------
// Cooperative groups of G threads working on one block.  G == 32: one warp
// (several groups per CTA).  G > 32: the whole CTA.  All reductions are
// all-reduces whose result is bitwise identical on every thread (xor
// butterflies are symmetric; the cross-warp stage combines warp results in a
// fixed order), so control decisions taken on reduced values stay uniform.

struct ArgMax {
  double v;      // |value| (>= 0); 0 means "no candidate"
  uint32_t idx;  // smallest index among equal maxima
  double sv;     // signed value at idx
};

__device__ __forceinline__ void argmax_merge(ArgMax& a, const ArgMax& b) {
  const long long bv = __double_as_longlong(b.v), av = __double_as_longlong(a.v);
  if (bv > av || (bv == av && b.idx < a.idx)) a = b;
}

struct ArgMinI {
  int v;         // value (INT_MAX: none)
  uint32_t idx;  // smallest index among equal minima
};

__device__ __forceinline__ void argmin_merge(ArgMinI& a, const ArgMinI& b) {
  if (b.v < a.v || (b.v == a.v && b.idx < a.idx)) a = b;
}

template <int G>
struct Group;

template <>
struct Group<32> {
  uint32_t rank;  // 0..31
  __device__ explicit Group(uint32_t r) : rank(r) {}
  __device__ static void sync() { __syncwarp(); }
  __device__ static double sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  __device__ static void sum2(double& a, double& b) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
  }
  __device__ static void sum3(double& a, double& b, double& c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
    }
  }
  __device__ static ArgMax argmax(ArgMax a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax b;
      b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
      b.idx = __shfl_xor_sync(0xffffffffu, a.idx, o);
      b.sv = __shfl_xor_sync(0xffffffffu, a.sv, o);
      argmax_merge(a, b);
    }
    return a;
  }
  __device__ static ArgMinI argmin(ArgMinI a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMinI b;
      b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
      b.idx = __shfl_xor_sync(0xffffffffu, a.idx, o);
      argmin_merge(a, b);
    }
    return a;
  }
  __device__ static uint32_t umin(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = min(v, (uint32_t)__shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
  __device__ static int imax(int v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
};

// Whole-CTA group of G threads (G a multiple of 32, <= 1024).  Uses a small
// shared scratch area; every call begins and ends with a CTA barrier.
template <int G>
struct Group {
  static constexpr int W = G / 32;
  uint32_t rank;
  double* red;  // shared scratch of 3*W doubles + 2*W words (see ctor users)
  __device__ Group(uint32_t r, double* scratch) : rank(r), red(scratch) {}
  __device__ static void sync() { __syncthreads(); }
  __device__ double sum(double v) const {
    v = Group<32>::sum(v);
    __syncthreads();
    if ((rank & 31) == 0) red[rank >> 5] = v;
    __syncthreads();
    double s = red[0];
    for (int w = 1; w < W; ++w) s += red[w];
    return s;
  }
  __device__ void sum2(double& a, double& b) const {
    Group<32>::sum2(a, b);
    __syncthreads();
    if ((rank & 31) == 0) {
      red[rank >> 5] = a;
      red[W + (rank >> 5)] = b;
    }
    __syncthreads();
    a = red[0];
    b = red[W];
    for (int w = 1; w < W; ++w) {
      a += red[w];
      b += red[W + w];
    }
  }
  __device__ void sum3(double& a, double& b, double& c) const {
    Group<32>::sum3(a, b, c);
    __syncthreads();
    if ((rank & 31) == 0) {
      red[rank >> 5] = a;
      red[W + (rank >> 5)] = b;
      red[2 * W + (rank >> 5)] = c;
    }
    __syncthreads();
    a = red[0];
    b = red[W];
    c = red[2 * W];
    for (int w = 1; w < W; ++w) {
      a += red[w];
      b += red[W + w];
      c += red[2 * W + w];
    }
  }
  __device__ ArgMax argmax(ArgMax a) const {
    a = Group<32>::argmax(a);
    __syncthreads();
    uint32_t* ri = reinterpret_cast<uint32_t*>(red + 2 * W);
    if ((rank & 31) == 0) {
      red[rank >> 5] = a.v;
      red[W + (rank >> 5)] = a.sv;
      ri[rank >> 5] = a.idx;
    }
    __syncthreads();
    ArgMax r{red[0], ri[0], red[W]};
    for (int w = 1; w < W; ++w) argmax_merge(r, ArgMax{red[w], ri[w], red[W + w]});
    return r;
  }
  __device__ ArgMinI argmin(ArgMinI a) const {
    a = Group<32>::argmin(a);
    __syncthreads();
    int* rv = reinterpret_cast<int*>(red);
    uint32_t* ri = reinterpret_cast<uint32_t*>(red) + W;
    if ((rank & 31) == 0) {
      rv[rank >> 5] = a.v;
      ri[rank >> 5] = a.idx;
    }
    __syncthreads();
    ArgMinI r{rv[0], ri[0]};
    for (int w = 1; w < W; ++w) argmin_merge(r, ArgMinI{rv[w], ri[w]});
    return r;
  }
  __device__ uint32_t umin(uint32_t v) const {
    v = Group<32>::umin(v);
    __syncthreads();
    uint32_t* ri = reinterpret_cast<uint32_t*>(red);
    if ((rank & 31) == 0) ri[rank >> 5] = v;
    __syncthreads();
    uint32_t r = ri[0];
    for (int w = 1; w < W; ++w) r = min(r, ri[w]);
    return r;
  }
  __device__ int imax(int v) const {
    v = Group<32>::imax(v);
    __syncthreads();
    int* ri = reinterpret_cast<int*>(red);
    if ((rank & 31) == 0) ri[rank >> 5] = v;
    __syncthreads();
    int r = ri[0];
    for (int w = 1; w < W; ++w) r = max(r, ri[w]);
    return r;
  }
};

}  // namespace ahx
