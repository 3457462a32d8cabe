// Adaptive cross approximation of one block and its recompression to the truncated
// SVD, FP64 real and complex, by a team of W warps.
//
//   ACA row/column steps, driver   Include/ACA.h:29-350
//   ACAr (symmetric assembly)      Include/ACA.h:579-720
//   recompression addtrll          H/mblock_D.cpp:356-465, H/mblock_Z.cpp:200-300
//
// What bounds it: the FP64 pipe (2 multiply-adds per clock and SM; a warp
// instruction occupies its scheduler's share for 64 clocks, whichever lanes are
// live).  The design therefore counts FP64 warp instructions:
//   * reductions over a warp are made for 8 values at a time (9 additions instead
//     of 40): at the finest leaves, 32-64 rows, they outnumber the sums themselves;
//   * arg-max and arg-min run on the integer reduction unit;
//   * the Gram matrices that the stopping rule needs (U_l^H U_k, V_l^H V_k) are kept:
//     their Cholesky factors are the R factors of both QRs, and the truncated
//     factors U (R1^-1 W S), V (R2^-1 Z) need one pass over the rows instead of
//     Householder's five.  U = Q1 R1 holds to rounding whatever Q1's orthogonality,
//     so that the product U V^H keeps Householder's backward error as long as the
//     columns are not nearly dependent; kCholTau guards that, and other blocks (and
//     tolerances near rounding) take a Householder QR;
//   * the Jacobi rotations are found in FP32 (the angle need not be exact, only
//     c^2 + s^2 = 1 must: one more sweep at most), their right factor is not
//     accumulated (Z = M^H (W S) S^-2 afterwards), column norms are updated; M is
//     brought to triangular form first (lq: all of the assembly 31.6 -> 29.9 ms below,
//     19.9 -> 17.5 ms complex);
//   * matrix entries take a reciprocal square root seeded in FP32.
// All admissible leaves of 65,536 sphere points (60,012, ranks about 10 before and 7
// after the truncation): 95 ms with Householder QRs and one value per reduction, 20 ms
// so; Helmholtz, 12,289 points, k = 8: 96 ms, 15 ms.  FP64 pipe 85 % busy (68 % complex).
#pragma once
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "ahx_aca.cuh"

namespace ahx {

struct Cx {
  double re, im;
};

namespace lowrank {

// ---------------------------------------------------------------------------
// arithmetic shared by both element types

__device__ __forceinline__ double zero_of(double) { return 0.0; }
__device__ __forceinline__ Cx zero_of(Cx) { return Cx{0.0, 0.0}; }
__device__ __forceinline__ double conj_(double a) { return a; }
__device__ __forceinline__ Cx conj_(Cx a) { return Cx{a.re, -a.im}; }
__device__ __forceinline__ double re_(double a) { return a; }
__device__ __forceinline__ double re_(Cx a) { return a.re; }
__device__ __forceinline__ double from_re(double, double v) { return v; }
__device__ __forceinline__ Cx from_re(Cx, double v) { return Cx{v, 0.0}; }
__device__ __forceinline__ double abs2(double a) { return a * a; }
__device__ __forceinline__ double abs2(Cx a) { return fma(a.re, a.re, a.im * a.im); }
// the order of magnitudes: |a|, squared for complex elements (no square root)
__device__ __forceinline__ double mag(double a) { return fabs(a); }
__device__ __forceinline__ double mag(Cx a) { return abs2(a); }
__device__ __forceinline__ double mag_of(double, double x) { return x; }
__device__ __forceinline__ double mag_of(Cx, double x) { return x * x; }
__device__ __forceinline__ double abs_of_mag(double, double m) { return m; }
__device__ __forceinline__ double abs_of_mag(Cx, double m) { return sqrt(m); }
__device__ __forceinline__ double scale_(double a, double s) { return a * s; }
__device__ __forceinline__ Cx scale_(Cx a, double s) { return Cx{a.re * s, a.im * s}; }
__device__ __forceinline__ double mul_(double a, double b) { return a * b; }
__device__ __forceinline__ Cx mul_(Cx a, Cx b) {
  return Cx{fma(a.re, b.re, -(a.im * b.im)), fma(a.re, b.im, a.im * b.re)};
}
// acc + a b, acc + conj(a) b, acc - a b, acc - conj(a) b
__device__ __forceinline__ double madd(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ Cx madd(Cx acc, Cx a, Cx b) {
  return Cx{fma(-a.im, b.im, fma(a.re, b.re, acc.re)), fma(a.im, b.re, fma(a.re, b.im, acc.im))};
}
__device__ __forceinline__ double maddc(double acc, double a, double b) { return fma(a, b, acc); }
__device__ __forceinline__ Cx maddc(Cx acc, Cx a, Cx b) {
  return Cx{fma(a.im, b.im, fma(a.re, b.re, acc.re)), fma(-a.im, b.re, fma(a.re, b.im, acc.im))};
}
__device__ __forceinline__ double msub(double acc, double a, double b) { return fma(-a, b, acc); }
__device__ __forceinline__ Cx msub(Cx acc, Cx a, Cx b) { return madd(acc, Cx{-a.re, -a.im}, b); }
__device__ __forceinline__ double msubc(double acc, double a, double b) { return fma(-a, b, acc); }
__device__ __forceinline__ Cx msubc(Cx acc, Cx a, Cx b) { return madd(acc, Cx{-a.re, a.im}, b); }

__device__ __forceinline__ double shfl_(double a, int src, int w = 32) { return __shfl_sync(0xffffffffu, a, src, w); }
__device__ __forceinline__ Cx shfl_(Cx a, int src, int w = 32) {
  return Cx{__shfl_sync(0xffffffffu, a.re, src, w), __shfl_sync(0xffffffffu, a.im, src, w)};
}

__device__ __forceinline__ double sqrt_any(double x) { return x > 0.0 ? x * rsqrt_any(x) : sqrt(x); }
__device__ __forceinline__ float sqrt_f32(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------
// matrix entries

struct LapGen {  // 1 / (4 pi r)
  using T = double;
  PointsSoA P;
  double diag;
  struct Fix {
    double x, y, z;
    uint32_t i;
  };
  __device__ __forceinline__ Fix fix(uint32_t i) const { return Fix{P.x[i], P.y[i], P.z[i], i}; }
  __device__ __forceinline__ double entry(const Fix& f, uint32_t j) const {
    if (f.i == j) return diag;
    const double dx = f.x - P.x[j], dy = f.y - P.y[j], dz = f.z - P.z[j];
    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
    return (1.0 / kFourPi) * rsqrt_any(r2);
  }
};

struct HelmGen {  // exp(i k r) / (4 pi r)
  using T = Cx;
  PointsSoA P;
  double k, h;
  struct Fix {
    double x, y, z;
    uint32_t i;
  };
  __device__ __forceinline__ Fix fix(uint32_t i) const { return Fix{P.x[i], P.y[i], P.z[i], i}; }
  __device__ __forceinline__ Cx entry(const Fix& f, uint32_t j) const {
    double r, s;
    const double dx = f.x - P.x[j], dy = f.y - P.y[j], dz = f.z - P.z[j];
    const double r2 = fma(dz, dz, fma(dy, dy, dx * dx));
    if (f.i != j && f32_range(r2)) {
      const double y = rsqrt_seeded(r2);
      r = r2 * y;
      r = fma(0.5 * y, fma(-r, r, r2), r);
      s = (1.0 / kFourPi) * y;
    } else if (f.i == j) {
      r = h;
      s = reciprocal_rounded(kFourPi * h);
    } else {
      const double2 v = rounded_r_s_any(r2);
      r = v.x;
      s = v.y;
    }
    double sn, cs;
    sincos(k * r, &sn, &cs);
    return Cx{cs * s, sn * s};
  }
};

// ---------------------------------------------------------------------------
// a team of W warps; reductions leave the same bits on every thread

template <int W>
struct Team {
  static constexpr uint32_t G = 32 * W;
  uint32_t rank, lane, warp;
  double* red;  // W > 1: 64 doubles of shared memory, two halves used in turn
  uint32_t ph = 0;
  __device__ Team(uint32_t r, double* scratch) : rank(r), lane(r & 31), warp(r >> 5), red(scratch) {}
  __device__ static void sync() {
    if constexpr (W == 1) __syncwarp();
    else __syncthreads();
  }
  __device__ double* half() {
    double* b = red + ph * 32;
    ph ^= 1;
    return b;
  }
  __device__ bool owns(uint32_t i) const { return i % G == rank; }
  // the sums of 8 values over the team; the thread gets that of value (lane >> 2) & 7
  __device__ double sum8(double (&v)[8]) {
#pragma unroll
    for (int m = 4; m >= 1; m >>= 1) {
      const bool up = lane & (4 * m);
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const double send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * m);
      }
    }
    double r = v[0];
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    if constexpr (W > 1) {
      double* b = half();
      if ((lane & 3) == 0) b[warp * 8 + (lane >> 2)] = r;
      __syncthreads();
      r = b[lane >> 2];
      for (int w = 1; w < W; ++w) r += b[w * 8 + (lane >> 2)];
    }
    return r;
  }
  // the sums of 4 values, all of them on every thread
  __device__ void sum4(double (&v)[4]) {
#pragma unroll
    for (int m = 2; m >= 1; m >>= 1) {
      const bool up = lane & (8 * m);
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const double send = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8 * m);
      }
    }
    double r = v[0];
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    if constexpr (W > 1) {
      double* b = half();
      if ((lane & 7) == 0) b[warp * 4 + (lane >> 3)] = r;
      __syncthreads();
      r = b[lane >> 3];
      for (int w = 1; w < W; ++w) r += b[w * 4 + (lane >> 3)];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __shfl_sync(0xffffffffu, r, 8 * q);
  }
  // largest magnitude (ordered by its bits), the smallest index among equals, its value
  template <class T>
  __device__ void argmax(double& m, uint32_t& idx, T& val) {
    const uint32_t hi = (uint32_t)__double2hiint(m), lo = (uint32_t)__double2loint(m);
    const uint32_t mh = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const uint32_t c = hi == mh && lo == ml ? idx : 0xffffffffu;
    const uint32_t mi = __reduce_min_sync(0xffffffffu, c);
    const uint32_t who = __ballot_sync(0xffffffffu, c == mi);
    m = __hiloint2double((int)mh, (int)ml);
    idx = mi;
    val = shfl_(val, who ? __ffs((int)who) - 1 : 0);
    if constexpr (W > 1) {
      double* b = half();
      T* bv = reinterpret_cast<T*>(b + 2 * W);
      if (lane == 0) {
        b[warp] = m;
        b[W + warp] = __hiloint2double(0, (int)idx);
        bv[warp] = val;
      }
      __syncthreads();
      m = b[0];
      idx = (uint32_t)__double2loint(b[W]);
      int at = 0;
      for (int w = 1; w < W; ++w) {
        const double om = b[w];
        const uint32_t oi = (uint32_t)__double2loint(b[W + w]);
        if (gt_nonneg(om, m) || (__double_as_longlong(om) == __double_as_longlong(m) && oi < idx)) {
          m = om;
          idx = oi;
          at = w;
        }
      }
      val = bv[at];
    } else {
      __syncwarp();
    }
  }
  // smallest value, the smallest index among equals
  __device__ void argmin(int& v, uint32_t& idx) {
    const int mv = __reduce_min_sync(0xffffffffu, v);
    idx = __reduce_min_sync(0xffffffffu, v == mv ? idx : 0xffffffffu);
    v = mv;
    if constexpr (W > 1) {
      double* b = half();
      if (lane == 0) b[warp] = __hiloint2double(v, (int)idx);
      __syncthreads();
      v = __double2hiint(b[0]);
      idx = (uint32_t)__double2loint(b[0]);
      for (int w = 1; w < W; ++w) {
        const int ov = __double2hiint(b[w]);
        const uint32_t oi = (uint32_t)__double2loint(b[w]);
        if (ov < v || (ov == v && oi < idx)) {
          v = ov;
          idx = oi;
        }
      }
    }
  }
  __device__ uint32_t umin(uint32_t v) {
    int s = (int)(v ^ 0x80000000u);  // unsigned order as signed
    uint32_t i = 0;
    argmin(s, i);
    return (uint32_t)s ^ 0x80000000u;
  }
};

template <class Gen>
struct Blk {
  using T = typename Gen::T;
  Gen gen;
  uint32_t b1, n1, b2, n2;
  T* U;
  T* V;
  int* Z;
  int* S;
  // Gram matrices, column by column as crosses come: P(l, k) = U_l^H U_k for l <= k,
  // P(k, l) = V_l^H V_k for l < k (row-major, stride ld), d2[k] = |V_k|^2; null: not kept
  T* P;
  double* d2;
  uint32_t ld;
};

// next index >= j (cyclic) whose counter is not -1 (ACA.h:29-36)
template <int W>
__device__ uint32_t nexti(Team<W>& g, const int* Z, uint32_t n, uint32_t j) {
  uint32_t d = 0xffffffffu;
  for (uint32_t i = g.rank; i < n; i += Team<W>::G)
    if (Z[i] != -1) d = min(d, i >= j ? i - j : i + n - j);
  d = g.umin(d);
  return d == 0xffffffffu ? j : (j + d) % n;
}

// residual of the entry: e - sum_l conj(c_l) X(i, l) over the k crosses so far, with
// c_l the other factor's values in the fixed row or column (stride sc)
template <class T>
__device__ __forceinline__ T residual(T e, uint32_t k, const T* c, size_t sc, const T* x, size_t sx) {
#pragma unroll 4
  for (uint32_t l = 0; l < k; ++l) e = msubc(e, c[l * sc], x[l * sx]);
  return e;
}

// ACA_row_step (ACA.h:46-130) and, with SYM, ACAr_step (ACA.h:579-655: rows are skipped
// only for a small pivot, the pivot column is searched over all columns)
template <bool SYM, int W, class Gen>
__device__ bool row_step(Team<W>& g, const Blk<Gen>& B, uint32_t& klast, uint32_t& i0, uint32_t k, uint32_t& no,
                         double& nrmu2, double& nrmv2, double& v2, double scale) {
  using T = typename Gen::T;
  constexpr uint32_t G = Team<W>::G;
  const uint32_t n1 = B.n1, n2 = B.n2;
  T* const pu = B.U + (size_t)k * n1;
  T* const pv = B.V + (size_t)k * n2;
  double am;
  uint32_t j0;
  T piv;
  for (;;) {
    g.sync();
    klast = (uint32_t)B.Z[i0];
    const auto f = B.gen.fix(B.b1 + i0);
    am = 0.0;
    j0 = 0xffffffffu;
    piv = zero_of(T());
    for (uint32_t j = g.rank; j < n2; j += G) {
      const T v = residual(conj_(B.gen.entry(f, B.b2 + j)), k, B.U + i0, n1, B.V + j, n2);
      pv[j] = v;
      if (SYM || B.S[j] >= 0) {
        const double a = mag(v);
        if (gt_nonneg(a, am)) {
          am = a;
          j0 = j;
          piv = v;
        }
      }
    }
    g.argmax(am, j0, piv);
    if (j0 != 0xffffffffu && !(am < mag_of(T(), 1e-14 * scale))) break;
    if (g.owns(i0)) B.Z[i0] = -1;
    if (++no >= n1) return false;
    g.sync();
    i0 = nexti(g, B.Z, n1, i0);
  }
  // v *= sqrt|p| / p, u /= sqrt|p| (p: the pivot)
  const double ap = abs_of_mag(T(), am), rs = rsqrt_any(ap), sq = ap * rs;
  T sca;
  if constexpr (sizeof(T) == 8) sca = copysign(rs, piv);
  else sca = scale_(conj_(piv), rs * (rs * rs));
  const double thr = mag_of(T(), 1e-8 * scale * sq);
  nrmv2 = v2 = 0.0;
  for (uint32_t j = g.rank; j < n2; j += G) {
    T e = pv[j];
    if (SYM || B.S[j] >= 0) {
      e = mul_(e, sca);
      pv[j] = e;
      const double a2 = abs2(e);
      nrmv2 += a2;
      if (!SYM && gt_nonneg(sizeof(T) == 8 ? mag(e) : a2, thr)) ++B.S[j];
    } else {
      v2 += abs2(e);  // a used column: kept as it is, outside the norm
    }
  }
  const auto f = B.gen.fix(B.b2 + j0);
  if (g.owns(i0)) B.Z[i0] = -1;
  if (!SYM && g.owns(j0)) B.S[j0] = -1;
  ++no;
  nrmu2 = 0.0;
  double nm = 0.0;
  uint32_t ni = 0xffffffffu;
  for (uint32_t i = g.rank; i < n1; i += G) {
    const T e = scale_(residual(B.gen.entry(f, B.b1 + i), k, B.V + j0, n2, B.U + i, n1), rs);
    pu[i] = e;
    const double a2 = abs2(e), a = sizeof(T) == 8 ? mag(e) : a2;
    nrmu2 += a2;
    const int z = B.Z[i];
    if (z >= 0) {
      if (!SYM && gt_nonneg(a, thr)) B.Z[i] = z + 1;
      if (gt_nonneg(a, nm)) {
        nm = a;
        ni = i;
      }
    }
  }
  T dummy = zero_of(T());
  g.argmax(nm, ni, dummy);
  if (nm > 0.0) i0 = ni;
  double s[4] = {nrmu2, nrmv2, v2, 0.0};
  g.sum4(s);
  nrmu2 = s[0];
  nrmv2 = s[1];
  v2 = s[1] + s[2];
  return true;
}

// ACA_col_step (ACA.h:134-213)
template <int W, class Gen>
__device__ bool col_step(Team<W>& g, const Blk<Gen>& B, uint32_t& j0, uint32_t k, uint32_t& no, double& nrmu2,
                         double& u2, double& nrmv2, double scale) {
  using T = typename Gen::T;
  constexpr uint32_t G = Team<W>::G;
  const uint32_t n1 = B.n1, n2 = B.n2;
  T* const pu = B.U + (size_t)k * n1;
  T* const pv = B.V + (size_t)k * n2;
  double am;
  uint32_t i0;
  T piv;
  for (;;) {
    g.sync();
    const auto f = B.gen.fix(B.b2 + j0);
    am = 0.0;
    i0 = 0xffffffffu;
    piv = zero_of(T());
    for (uint32_t i = g.rank; i < n1; i += G) {
      const T u = residual(B.gen.entry(f, B.b1 + i), k, B.V + j0, n2, B.U + i, n1);
      pu[i] = u;
      if (B.Z[i] >= 0) {
        const double a = mag(u);
        if (gt_nonneg(a, am)) {
          am = a;
          i0 = i;
          piv = u;
        }
      }
    }
    g.argmax(am, i0, piv);
    if (i0 != 0xffffffffu && !(am < mag_of(T(), 1e-14 * scale))) break;
    if (g.owns(j0)) B.S[j0] = -1;
    if (++no >= n2) return false;
    g.sync();
    j0 = nexti(g, B.S, n2, j0);
  }
  const double ap = abs_of_mag(T(), am), rs = rsqrt_any(ap), sq = ap * rs;
  T sca;
  if constexpr (sizeof(T) == 8) sca = copysign(rs, piv);
  else sca = scale_(conj_(piv), rs * (rs * rs));
  const double thr = mag_of(T(), 1e-8 * scale * sq);
  nrmu2 = u2 = 0.0;
  for (uint32_t i = g.rank; i < n1; i += G) {
    T e = pu[i];
    if (B.Z[i] >= 0) {
      e = mul_(e, sca);
      pu[i] = e;
      const double a2 = abs2(e);
      nrmu2 += a2;
      if (gt_nonneg(sizeof(T) == 8 ? mag(e) : a2, thr)) ++B.Z[i];
    } else {
      u2 += abs2(e);
    }
  }
  const auto f = B.gen.fix(B.b1 + i0);
  if (g.owns(i0)) B.Z[i0] = -1;
  if (g.owns(j0)) B.S[j0] = -1;
  ++no;
  nrmv2 = 0.0;
  double nm = 0.0;
  uint32_t nj = 0xffffffffu;
  for (uint32_t j = g.rank; j < n2; j += G) {
    const T e = scale_(residual(conj_(B.gen.entry(f, B.b2 + j)), k, B.U + i0, n1, B.V + j, n2), rs);
    pv[j] = e;
    const double a2 = abs2(e), a = sizeof(T) == 8 ? mag(e) : a2;
    const int s = B.S[j];
    if (s >= 0 && gt_nonneg(a, thr)) B.S[j] = s + 1;
    nrmv2 += a2;
    if (gt_nonneg(a, nm)) {  // no S filter here, as in the reference
      nm = a;
      nj = j;
    }
  }
  T dummy = zero_of(T());
  g.argmax(nm, nj, dummy);
  if (nm > 0.0) j0 = nj;
  double s[4] = {nrmu2, u2, nrmv2, 0.0};
  g.sum4(s);
  nrmu2 = s[0];
  u2 = s[0] + s[1];
  nrmv2 = s[2];
  return true;
}

// Column k of both Gram matrices; returns Re sum_l (U_l^H U_k) (V_l^H V_k), l < k.
template <int W, class Gen>
__device__ double gram(Team<W>& g, const Blk<Gen>& B, uint32_t k, double u2, double v2) {
  using T = typename Gen::T;
  constexpr uint32_t G = Team<W>::G;
  constexpr int NC = sizeof(T) / 8, LC = 4 / NC;  // components, columns per pass
  const uint32_t n1 = B.n1, n2 = B.n2;
  const T* uk = B.U + (size_t)k * n1;
  const T* vk = B.V + (size_t)k * n2;
  const uint32_t at = g.lane >> 2, side = at >> 2, ll = (at & 3) / NC, comp = (at & 3) % NC;
  double acc = 0.0;
  for (uint32_t l0 = 0; l0 < k; l0 += LC) {
    T du[LC], dv[LC];
#pragma unroll
    for (int q = 0; q < LC; ++q) du[q] = dv[q] = zero_of(T());
    for (uint32_t i = g.rank; i < n1; i += G) {
      const T x = uk[i];
#pragma unroll
      for (int q = 0; q < LC; ++q)
        if (l0 + q < k) du[q] = maddc(du[q], B.U[(size_t)(l0 + q) * n1 + i], x);
    }
    for (uint32_t j = g.rank; j < n2; j += G) {
      const T x = vk[j];
#pragma unroll
      for (int q = 0; q < LC; ++q)
        if (l0 + q < k) dv[q] = maddc(dv[q], B.V[(size_t)(l0 + q) * n2 + j], x);
    }
    double v[8];
#pragma unroll
    for (int q = 0; q < LC; ++q) {
      if constexpr (NC == 1) {
        v[q] = du[q];
        v[4 + q] = dv[q];
      } else {
        v[2 * q] = du[q].re;
        v[2 * q + 1] = du[q].im;
        v[4 + 2 * q] = dv[q].re;
        v[4 + 2 * q + 1] = dv[q].im;
      }
    }
    const double t = g.sum8(v);
    const double o = __shfl_xor_sync(0xffffffffu, t, 16);
    acc = fma(comp ? -t : t, o, acc);
    const uint32_t l = l0 + ll;
    if (B.P && g.warp == 0 && (g.lane & 3) == 0 && l < k) {
      const size_t e = side ? (size_t)k * B.ld + l : (size_t)l * B.ld + k;
      reinterpret_cast<double*>(B.P)[e * NC + comp] = t;
    }
  }
  if (B.P && g.rank == 0) {
    B.P[(size_t)k * B.ld + k] = from_re(T(), u2);
    B.d2[k] = v2;
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 4);
  acc += __shfl_xor_sync(0xffffffffu, acc, 8);
  return acc;
}

// ACA driver (ACA.h:217-350).  Returns the status, the rank in kout.
template <int W, class Gen>
__device__ int aca(Team<W>& g, const Blk<Gen>& B, uint32_t i0, uint32_t kmax, uint32_t kcap, double eps,
                   uint32_t& kout) {
  using T = typename Gen::T;
  constexpr uint32_t G = Team<W>::G;
  const uint32_t n1 = B.n1, n2 = B.n2;
  for (uint32_t i = g.rank; i < n1; i += G) B.Z[i] = 0;
  for (uint32_t j = g.rank; j < n2; j += G) B.S[j] = 0;
  double scale = abs_of_mag(T(), mag(B.gen.entry(B.gen.fix(B.b1), B.b2)));
  const double inv_n = 1.0 / (double)(uint32_t)(n1 * n2);
  uint32_t k = 0, no = 0, klast = 0, inext = i0, j0 = 0;
  int kmin = -2, keps = -1;
  double nrmlsk2 = 0.0, nrms2 = 0.0, nu, nv, w2;
  int outcome = -1;  // 0 NSUCC, 1 SUCC, 2 overflow
  do {
    if (k >= kcap) { outcome = kAcaOverflow; break; }
    inext = i0;
    if (!row_step<false>(g, B, klast, inext, k, no, nu, nv, w2, scale)) {
      nrmlsk2 = 0.0;
      outcome = kAcaOk;
      break;
    }
    nrmlsk2 = nu * nv;
    nrms2 += 2.0 * gram(g, B, k, nu, w2) + nrmlsk2;
    const bool stpcrit = nrmlsk2 < eps * eps * nrms2;
    if (stpcrit && keps == -1) keps = (int)klast + 1;
    ++k;
    scale = sqrt_any(nrmlsk2 * inv_n);
    if (keps > 0) {
      int mv = INT_MAX;
      uint32_t mi = 0xffffffffu;
      for (uint32_t i = g.rank; i < n1; i += G)
        if (B.Z[i] >= 0 && B.Z[i] < mv) {
          mv = B.Z[i];
          mi = i;
        }
      g.argmin(mv, mi);
      if (mv == INT_MAX) {
        nrmlsk2 = 0.0;
        outcome = kAcaOk;
        break;
      }
      kmin = mv;
      i0 = mi;
      if ((uint32_t)kmin == k) i0 = inext;
    } else {
      i0 = inext;
    }
  } while (no < n1 && k < kmax && kmin < keps);

  if (outcome < 0) {
    if ((no == n1 || k == kmax) && kmin < keps) {
      outcome = kAcaFail;
    } else {
      do {
        int mv = INT_MAX;
        uint32_t mi = 0xffffffffu;
        for (uint32_t j = g.rank; j < n2; j += G)
          if (B.S[j] >= 0 && B.S[j] < mv) {
            mv = B.S[j];
            mi = j;
          }
        g.argmin(mv, mi);
        if (mv == INT_MAX) {
          nrmlsk2 = 0.0;
          outcome = kAcaOk;
          break;
        }
        kmin = mv;
        j0 = mi;
        if (kmin >= keps) { outcome = kAcaOk; break; }
        if (k >= kcap) { outcome = kAcaOverflow; break; }
        if (!col_step(g, B, j0, k, no, nu, w2, nv, scale)) {
          nrmlsk2 = 0.0;
          outcome = kAcaOk;
          break;
        }
        nrmlsk2 = nu * nv;
        if (B.P) gram(g, B, k, w2, nv);
        ++k;
      } while (no < n2 && k < kmax);
      if (outcome < 0) outcome = kAcaFail;
    }
  }
  if (outcome == kAcaOk) {
    const double epsa = sqrt(nrmlsk2 / nrms2);
    if (epsa >= eps) outcome = kAcaFail;  // NaN (0/0) stays a success, as in the reference
  }
  kout = k;
  g.sync();
  return outcome;
}

// ACAr driver (ACA.h:657-720): crosses until the last one is below eps of the
// approximation's norm, no more than n2 rows used, or kmax crosses.
template <int W, class Gen>
__device__ int acar(Team<W>& g, const Blk<Gen>& B, uint32_t i0, uint32_t kmax, uint32_t kcap, double eps,
                    uint32_t& kout) {
  using T = typename Gen::T;
  const uint32_t n1 = B.n1, n2 = B.n2;
  for (uint32_t i = g.rank; i < n1; i += Team<W>::G) B.Z[i] = 0;
  double scale = abs_of_mag(T(), mag(B.gen.entry(B.gen.fix(B.b1), B.b2)));
  const double inv_n = 1.0 / (double)(uint32_t)(n1 * n2);
  uint32_t k = 0, no = 0, klast = 0;
  double nrmlsk2 = 0.0, nrms2 = 0.0, nu, nv, w2;
  int outcome = -1;
  do {
    if (k >= kcap) {
      outcome = kAcaOverflow;
      break;
    }
    if (!row_step<true>(g, B, klast, i0, k, no, nu, nv, w2, scale)) {
      nrmlsk2 = 0.0;
      break;
    }
    nrmlsk2 = nu * nv;
    nrms2 += 2.0 * gram(g, B, k, nu, w2) + nrmlsk2;
    ++k;
    scale = sqrt_any(nrmlsk2 * inv_n);
  } while (no < n2 && k < kmax && nrmlsk2 >= eps * eps * nrms2);
  if (outcome < 0) {
    const double epsa = sqrt(nrmlsk2 / nrms2);
    outcome = epsa >= eps ? kAcaFail : kAcaOk;  // NaN (0/0) stays a success, as in the reference
  }
  kout = k;
  g.sync();
  return outcome;
}

// ---------------------------------------------------------------------------
// recompression

// A column whose part orthogonal to the earlier ones is below sqrt(kCholTau) of its
// norm sends the block to the Householder QR: with the guard the rounding error of
// U (R1^-1 x) is at most eps_mach / 1e-3 of x.  On admissible blocks of surface
// meshes the part is 1e-2 to 1e-1 (smallest seen: 1.3e-2).  Truncation tolerances
// below kCholEps, where that error would show, take Householder's as well.
constexpr double kCholTau = 1e-6;
constexpr double kCholEps = 1e-10;

constexpr uint32_t kSmSq = 1088;   // shared elements per team: 4 squares of 16 x 17, or one of 32 x 33
constexpr uint32_t kSmDbl = 180;   // shared doubles per team: dinv[64] nrm[32] inv[32] d2[32] perm[33 ints]
template <class T>
constexpr size_t team_smem() { return kSmSq * sizeof(T) + kSmDbl * sizeof(double); }

// Work arrays of a block: square (k x k) arrays row-major
template <class T>
struct Work {
  T *P, *M0, *M, *C2;
  double *d2, *dinv, *nrm, *inv;
  int* perm;
  uint32_t ld, ldm;  // stride of P, M0, C2; of M
};

// Cholesky factors of both Gram matrices in place, by one warp (for k <= 16 one matrix
// per half-warp): R1(r, c) = P(r, c), R2(r, c) = P(c, r) (r < c) and d2[c]; dinv: the
// reciprocal diagonals.  false: a column is nearly dependent (or not finite).
template <class T>
__device__ bool cholesky(const Work<T>& w, uint32_t k, uint32_t lane) {
  const uint32_t wd = k <= 16 ? 16 : 32, hl = lane & (wd - 1);
  for (uint32_t s0 = 0; s0 < 2; s0 += 32 / wd) {
    const uint32_t side = s0 + (wd == 16 ? lane >> 4 : 0);
    const size_t sr = side ? 1 : w.ld, sc = side ? w.ld : 1;  // R(r, c) at r sr + c sc
    T* const A = w.P;
    for (uint32_t c = 0; c < k; ++c) {
      double inv = 0.0;
      for (uint32_t j0 = c; j0 < k; j0 += wd) {
        const uint32_t j = j0 + hl;
        T s = zero_of(T());
        double g0 = 0.0;
        if (j < k) {
          s = j == c && side ? from_re(T(), w.d2[c]) : A[c * sr + j * sc];
          g0 = re_(s);
          for (uint32_t l = 0; l < c; ++l) s = msubc(s, A[l * sr + c * sc], A[l * sr + j * sc]);
        }
        if (j0 == c) {
          const double d = __shfl_sync(0xffffffffu, re_(s), 0, wd);
          g0 = __shfl_sync(0xffffffffu, g0, 0, wd);
          if (!__all_sync(0xffffffffu, d > kCholTau * g0 && d < 1e300 && d > 1e-290)) return false;
          inv = rsqrt_any(d);
          if (hl == 0) w.dinv[side * (k <= 32 ? 32 : k) + c] = inv;
        }
        if (j < k) {
          if (j == c) {
            if (side) w.d2[c] = re_(s) * inv;
            else A[c * sr + c * sc] = from_re(T(), re_(s) * inv);
          } else {
            A[c * sr + j * sc] = scale_(s, inv);
          }
        }
      }
      __syncwarp();
    }
  }
  return true;
}

// Householder QR of A (m x k, column-major), LAPACK's form: H_c = I - tau_c v_c v_c^H,
// v_c(c) = 1, a real diagonal; row i belongs to thread i % G
template <int W, class T>
__device__ void qr(Team<W>& g, uint32_t m, uint32_t k, T* A, T* tau) {
  constexpr uint32_t G = Team<W>::G;
  constexpr int NC = sizeof(T) / 8, QC = 8 / NC;
  const uint32_t kk = min(m, k);
  for (uint32_t c = 0; c < kk; ++c) {
    T* a = A + (size_t)c * m;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint32_t i = g.rank; i < m; i += G) {
      if (i > c) s[0] += abs2(a[i]);
      else if (i == c) {
        s[1] = re_(a[i]);
        if constexpr (NC == 2) s[2] = a[i].im;
      }
    }
    g.sum4(s);
    const double xn2 = s[0], ar = s[1], ai = s[2];
    if (xn2 == 0.0 && ai == 0.0) {
      if (g.rank == 0) tau[c] = zero_of(T());
      continue;
    }
    const double nrm = sqrt(ar * ar + ai * ai + xn2);
    const double beta = ar >= 0.0 ? -nrm : nrm;
    T t, sc;
    if constexpr (NC == 1) {
      t = (beta - ar) / beta;
      sc = 1.0 / (ar - beta);
    } else {
      t = Cx{(beta - ar) / beta, -ai / beta};
      const double d = 1.0 / ((ar - beta) * (ar - beta) + ai * ai);
      sc = Cx{(ar - beta) * d, -ai * d};
    }
    if (g.rank == 0) tau[c] = t;
    for (uint32_t i = g.rank; i < m; i += G) {
      if (i > c) a[i] = mul_(a[i], sc);
      else if (i == c) a[i] = from_re(T(), beta);
    }
    const T tc = conj_(t);
    for (uint32_t q0 = c + 1; q0 < k; q0 += QC) {
      T d[QC];
#pragma unroll
      for (int q = 0; q < QC; ++q) d[q] = zero_of(T());
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i < c) continue;
        const T x = i == c ? from_re(T(), 1.0) : a[i];
#pragma unroll
        for (int q = 0; q < QC; ++q)
          if (q0 + q < k) d[q] = maddc(d[q], x, A[(size_t)(q0 + q) * m + i]);
      }
      double v[8];
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        if constexpr (NC == 1) v[q] = d[q];
        else {
          v[2 * q] = d[q].re;
          v[2 * q + 1] = d[q].im;
        }
      }
      const double tot = g.sum8(v);
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        T sq;
        if constexpr (NC == 1) sq = __shfl_sync(0xffffffffu, tot, 4 * q);
        else sq = Cx{__shfl_sync(0xffffffffu, tot, 8 * q), __shfl_sync(0xffffffffu, tot, 8 * q + 4)};
        d[q] = mul_(tc, sq);
      }
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i < c) continue;
        const T x = i == c ? from_re(T(), 1.0) : a[i];
#pragma unroll
        for (int q = 0; q < QC; ++q)
          if (q0 + q < k) A[(size_t)(q0 + q) * m + i] = msub(A[(size_t)(q0 + q) * m + i], d[q], x);
      }
    }
  }
}

// C (m x nc, column-major) := H_0 ... H_{kr-1} C
template <int W, class T>
__device__ void apply_q(Team<W>& g, uint32_t m, uint32_t kr, const T* A, const T* tau, uint32_t nc, T* C) {
  constexpr uint32_t G = Team<W>::G;
  constexpr int NC = sizeof(T) / 8, QC = 8 / NC;
  for (int c = (int)kr - 1; c >= 0; --c) {
    const T t = tau[c];
    if (abs2(t) == 0.0) continue;
    const T* a = A + (size_t)c * m;
    for (uint32_t q0 = 0; q0 < nc; q0 += QC) {
      T d[QC];
#pragma unroll
      for (int q = 0; q < QC; ++q) d[q] = zero_of(T());
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i < (uint32_t)c) continue;
        const T x = i == (uint32_t)c ? from_re(T(), 1.0) : a[i];
#pragma unroll
        for (int q = 0; q < QC; ++q)
          if (q0 + q < nc) d[q] = maddc(d[q], x, C[(size_t)(q0 + q) * m + i]);
      }
      double v[8];
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        if constexpr (NC == 1) v[q] = d[q];
        else {
          v[2 * q] = d[q].re;
          v[2 * q + 1] = d[q].im;
        }
      }
      const double tot = g.sum8(v);
#pragma unroll
      for (int q = 0; q < QC; ++q) {
        T sq;
        if constexpr (NC == 1) sq = __shfl_sync(0xffffffffu, tot, 4 * q);
        else sq = Cx{__shfl_sync(0xffffffffu, tot, 8 * q), __shfl_sync(0xffffffffu, tot, 8 * q + 4)};
        d[q] = mul_(t, sq);
      }
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i < (uint32_t)c) continue;
        const T x = i == (uint32_t)c ? from_re(T(), 1.0) : a[i];
#pragma unroll
        for (int q = 0; q < QC; ++q)
          if (q0 + q < nc) C[(size_t)(q0 + q) * m + i] = msub(C[(size_t)(q0 + q) * m + i], d[q], x);
      }
    }
  }
}

// M := L with M = L Q^H, Q's columns orthonormal (modified Gram-Schmidt on M's rows,
// whose triangular factor is as accurate as Householder's, Bjorck 1967): same left
// singular vectors and singular values, L lower triangular.  The rows are R1's, in the
// order of falling pivots, so that L's columns are nearly orthogonal already and Jacobi
// needs about 3 sweeps less (7 -> 4-5; this costs 0.6 of one); rows that the threshold
// has emptied leave no column: returns the number of columns to work on.
// G: scratch (m x n, row-major, stride ldg), nrm: n.
template <int NW, class T>
__device__ uint32_t lq(Team<NW>& g, uint32_t m, uint32_t n, T* M, uint32_t ld, T* G, uint32_t ldg, double* nrm) {
  const uint32_t q = min(m, n);
  for (uint32_t j = 0; j < q; ++j) {
    const uint32_t rows = m - j;
    const uint32_t L = rows <= 4 * NW ? 8 : rows <= 8 * NW ? 4 : rows <= 16 * NW ? 2 : 1;
    const uint32_t sub = g.lane & (L - 1), grp = g.rank / L, groups = 32 * NW / L;
    const T* const rj = M + j * ld;
    for (uint32_t i0 = j; i0 < m; i0 += groups) {
      const uint32_t i = i0 + grp;
      T s = zero_of(T());
      if (i < m)
        for (uint32_t l = sub; l < n; l += L) s = maddc(s, rj[l], M[i * ld + l]);
      for (uint32_t o = 1; o < L; o <<= 1) {
        if constexpr (sizeof(T) == 16) {
          s.re += __shfl_xor_sync(0xffffffffu, s.re, o);
          s.im += __shfl_xor_sync(0xffffffffu, s.im, o);
        } else {
          s += __shfl_xor_sync(0xffffffffu, s, o);
        }
      }
      if (i < m && sub == 0) G[i * ldg + j] = s;
    }
    g.sync();
    const double d = re_(G[j * ldg + j]);
    // an empty row: no column (a NaN, which the FP64 unit makes with its sign set, is no empty
    // row: the leaf is to show it)
    const double rs = (__double2hiint(d) & 0x7fffffff) >= 0x00100000 ? rsqrt_any(d) : 0.0;
    if (g.rank == 0) nrm[j] = rs;
    const double r2 = rs * rs;
    for (uint32_t i = j + 1 + grp; i < m; i += groups) {
      const T f = scale_(G[i * ldg + j], r2);
      for (uint32_t l = sub; l < n; l += L) M[i * ld + l] = msub(M[i * ld + l], f, rj[l]);
    }
    g.sync();
  }
  uint32_t cols = 0;
  for (uint32_t j0 = 0; j0 < q; j0 += 32) {
    const uint32_t b =
        __ballot_sync(0xffffffffu, j0 + g.lane < q && __double_as_longlong(nrm[min(j0 + g.lane, q - 1)]) != 0);
    if (b) cols = j0 + 32 - __clz(b);
  }
  for (uint32_t e = g.rank; e < m * n; e += 32 * NW) {
    const uint32_t i = e / n, j = e - i * n;
    M[i * ld + j] = j < cols && j <= i ? scale_(G[i * ldg + j], nrm[j]) : zero_of(T());
  }
  g.sync();
  return cols;
}

// One-sided Jacobi (Hestenes) on the columns of M (m x n, row-major) in tournament
// order (Brent-Luk round robin) by NW warps: 8, 4 or 2 lanes per column pair.  A pair
// rotates unless |x^H y| <= 1e-15 |x| |y|.  The tangent is found in FP32, c and s from
// it in FP64; the squared norms are computed once a sweep and updated between.  A sweep
// whose cosines and angles (against the columns' lengths) all stayed below kJacLast is
// the last: a rotation leaves 1e-7 of its own cosine (FP32 angle) and changes the others
// by products of two such numbers, so that all are below the threshold after it.
constexpr float kJacLast = 3e-9f;
template <int NW, class T>
__device__ void jacobi(Team<NW>& g, uint32_t m, uint32_t n, T* M, uint32_t ld, double* nrm) {
  constexpr bool CX = sizeof(T) == 16;
  __shared__ int again;  // NW > 1 only
  const uint32_t ne = n + (n & 1), np = ne / 2;
  const uint32_t L = np <= 4 ? 8 : np <= 8 ? 4 : 2, sub = g.lane & (L - 1);
  const uint32_t grp = g.rank / L, groups = 32 * NW / L;
  for (int sweep = 0; sweep < 40; ++sweep) {
    g.sync();
    if (NW > 1 && g.rank == 0) again = 0;
    for (uint32_t j = g.rank; j < n; j += 32 * NW) {
      double s = 0.0;
      for (uint32_t i = 0; i < m; ++i) {
        if constexpr (CX) s = fma(M[i * ld + j].im, M[i * ld + j].im, fma(M[i * ld + j].re, M[i * ld + j].re, s));
        else s = fma(M[i * ld + j], M[i * ld + j], s);
      }
      nrm[j] = s;
    }
    g.sync();
    bool large = false;
    for (uint32_t r = 0; r + 1 < ne; ++r) {
      for (uint32_t p0 = 0; p0 < np; p0 += groups) {
        const uint32_t p = p0 + grp;
        uint32_t a = 0, b = 0;
        bool live = p < np;
        if (live) {
          const uint32_t pa = p, pb = ne - 1 - p;
          uint32_t x = pa - 1 + r, y = pb - 1 + r;  // both below 2 (ne - 1)
          x = x >= ne - 1 ? x - (ne - 1) : x;
          y = y >= ne - 1 ? y - (ne - 1) : y;
          a = pa == 0 ? 0 : 1 + x;
          b = 1 + y;
          if (a > b) {
            const uint32_t t = a;
            a = b;
            b = t;
          }
          live = b < n;
        }
        T ga = zero_of(T());
        if (live)
          for (uint32_t i = sub; i < m; i += L) ga = maddc(ga, M[i * ld + a], M[i * ld + b]);
        for (uint32_t o = 1; o < L; o <<= 1) {
          if constexpr (CX) {
            ga.re += __shfl_xor_sync(0xffffffffu, ga.re, o);
            ga.im += __shfl_xor_sync(0xffffffffu, ga.im, o);
          } else {
            ga += __shfl_xor_sync(0xffffffffu, ga, o);
          }
        }
        if (live) {
          const double al = nrm[a], be = nrm[b];
          double gm;       // signed (real) or absolute (complex) inner product
          T e = zero_of(T());  // complex: conj(ga) / |ga|
          if constexpr (CX) {
            const double g2 = abs2(ga);
            const double gi = rsqrt_any(g2);
            gm = g2 > 0.0 ? g2 * gi : 0.0;
            e = Cx{ga.re * gi, -ga.im * gi};
          } else {
            gm = ga;
          }
          // updated norms of small columns may have cancelled to below |gm|: it is scaled for too
          const int sh =
              (max(max(__double2hiint(al), __double2hiint(be)), __double2hiint(gm) & 0x7fffffff) >> 20) - 1023;
          const float fg = to_f32(gm, sh);
          const float fal = to_f32(al, sh), fbe = to_f32(be, sh);
          const float fd = to_f32(be - al, sh);
          const float g2 = 2.f * fg;
          const float t = __fdividef(g2, fd + copysignf(sqrt_f32(fmaf(fd, fd, g2 * g2)), fd));
          const float sa = sqrt_f32(fal), sb = sqrt_f32(fbe);
          if (fabsf(fg) > 1e-15f * sa * sb && fabsf(t) > 1e-37f) {
            large |= fabsf(fg) > kJacLast * sa * sb || fabsf(t) * fmaxf(sa, sb) > kJacLast * fminf(sa, sb);
            const double td = to_f64(t);
            const double c = rsqrt_seeded(fma(td, td, 1.0)), s = c * td;
            if constexpr (CX) {
              const Cx se{s * e.re, s * e.im}, ce{c * e.re, c * e.im};
              for (uint32_t i = sub; i < m; i += L) {
                const Cx x = M[i * ld + a], y = M[i * ld + b];
                M[i * ld + a] = msub(scale_(x, c), se, y);
                M[i * ld + b] = madd(scale_(x, s), ce, y);
              }
            } else {
              for (uint32_t i = sub; i < m; i += L) {
                const double x = M[i * ld + a], y = M[i * ld + b];
                M[i * ld + a] = fma(c, x, -(s * y));
                M[i * ld + b] = fma(s, x, c * y);
              }
            }
            if (sub == 0) {
              const double na = fma(-td, gm, al), nb = fma(td, gm, be);
              nrm[a] = __double2hiint(na) < 0 ? 0.0 : na;
              nrm[b] = __double2hiint(nb) < 0 ? 0.0 : nb;
            }
          }
        }
      }
      g.sync();
    }
    if constexpr (NW > 1) {
      if (large) again = 1;
      __syncthreads();
      if (!again) break;
    } else {
      if (!__any_sync(0xffffffffu, large)) break;
    }
  }
  g.sync();
}

// Un (n x kt) = X C with the rows of X (n x k) owned by thread i % G
template <int W, class T>
__device__ void times(Team<W>& g, uint32_t n, uint32_t k, const T* X, const T* C, uint32_t ldc, const int* perm,
                      uint32_t kt, T* Out) {
  constexpr int QC = 8 * 8 / sizeof(T);
  for (uint32_t q0 = 0; q0 < kt; q0 += QC) {
    uint32_t col[QC];
#pragma unroll
    for (int q = 0; q < QC; ++q) {
      const uint32_t j = min(q0 + q, kt - 1);
      col[q] = perm ? (uint32_t)perm[j] : j;
    }
    for (uint32_t i = g.rank; i < n; i += Team<W>::G) {
      T s[QC];
#pragma unroll
      for (int q = 0; q < QC; ++q) s[q] = zero_of(T());
      for (uint32_t l = 0; l < k; ++l) {
        const T x = X[(size_t)l * n + i];
#pragma unroll
        for (int q = 0; q < QC; ++q)
          if (q0 + q < kt) s[q] = madd(s[q], x, C[l * ldc + col[q]]);
      }
#pragma unroll
      for (int q = 0; q < QC; ++q)
        if (q0 + q < kt) Out[(size_t)(q0 + q) * n + i] = s[q];
    }
  }
}

// addtrll (H/mblock_D.cpp:356-465) for a fresh block U V^H of rank k (Grams in w):
// truncated to kt columns (relative threshold delta, absolute 1e-64), written through
// alloc(kt, Un, Vn).  tau: 2 k elements.  Returns false if alloc refuses.
template <int W, class T, class Alloc>
__device__ bool compress(Team<W>& g, uint32_t n1, uint32_t n2, uint32_t k, T* U, T* V, Work<T> w, T* tau, double delta,
                         T* smem, Alloc alloc, uint32_t& kt) {
  double* const smd = reinterpret_cast<double*>(smem + kSmSq);
  const uint32_t lane = g.lane;
  const bool first = W == 1 || g.warp == 0;  // the warp that works on the k x k arrays
  if (k <= 32) {
    w.dinv = smd;
    w.nrm = smd + 64;
    w.inv = smd + 96;
    w.perm = reinterpret_cast<int*>(smd + 160);
    w.M = smem;
    w.ldm = 33;
  }
  if (k <= 16) {
    // everything in shared memory
    if (first)
      for (uint32_t e = lane; e < k * k; e += 32) {
        const uint32_t i = e / k, j = e - i * k;
        smem[272 + i * 17 + j] = w.P[(size_t)i * w.ld + j];
        if (j == 0) smd[128 + i] = w.d2[i];
      }
    w.P = smem + 272;
    w.M0 = smem + 2 * 272;
    w.C2 = smem + 3 * 272;
    w.d2 = smd + 128;
    w.ld = w.ldm = 17;
  }
  const uint32_t mm = min(n1, k), nn = min(n2, k);
  __syncwarp();
  bool chol = k <= min(n1, n2) && delta >= kCholEps;
  if (first && chol) chol = cholesky(w, k, lane);
  if constexpr (W > 1) chol = __syncthreads_and(!first || chol);
  if (!chol) {
    qr(g, n1, k, U, tau);
    qr(g, n2, k, V, tau + k);
    g.sync();
    if (first)
      for (uint32_t e = lane; e < k * k; e += 32) {
        const uint32_t i = e / k, j = e - i * k;
        if (i <= j && i < mm) w.P[i * w.ld + j] = U[(size_t)j * n1 + i];
        if (i < j && i < nn) w.P[j * w.ld + i] = V[(size_t)j * n2 + i];
        if (i == j && i < nn) w.d2[i] = re_(V[(size_t)i * n2 + i]);
      }
    __syncwarp();
  }
  if (first) {
    // M = R1 R2^H (Include/blas.h:2767-2781), entries below the threshold dropped
    double f[4] = {0.0, 0.0, 0.0, 0.0};
    for (uint32_t e = lane; e < mm * nn; e += 32) {
      const uint32_t i = e / nn, j = e - i * nn;
      T s = zero_of(T());
      for (uint32_t l = max(i, j); l < k; ++l) {
        const T r1 = w.P[i * w.ld + l], r2 = l == j ? from_re(T(), w.d2[j]) : w.P[l * w.ld + j];
        s = madd(s, r1, conj_(r2));
      }
      w.M[i * w.ldm + j] = s;
      f[0] += abs2(s);
    }
    Team<1> g1(lane, nullptr);
    g1.sum4(f);
    const double thresh = mag_of(T(), delta * sqrt(f[0]) / (double)sqrtf((float)mm * (float)nn));
    for (uint32_t e = lane; e < mm * nn; e += 32) {
      const uint32_t i = e / nn, j = e - i * nn;
      T s = w.M[i * w.ldm + j];
      if (mag(s) < thresh) w.M[i * w.ldm + j] = s = zero_of(T());
      w.M0[i * w.ld + j] = s;
    }
    __syncwarp();
    if (W == 1 || k <= 32) {
      const uint32_t cols = lq<1>(g1, mm, nn, w.M, w.ldm, w.C2, w.ld, w.nrm);
      jacobi<1>(g1, mm, cols, w.M, w.ldm, w.nrm);
    }
  }
  if constexpr (W > 1) {
    __syncthreads();
    if (k > 32) {
      const uint32_t cols = lq<W>(g, mm, nn, w.M, w.ldm, w.C2, w.ld, w.nrm);
      jacobi<W>(g, mm, cols, w.M, w.ldm, w.nrm);
    }
  }
  if (first) {
    // singular values in descending order (the first among equals first), the rank
    for (uint32_t j = lane; j < nn; j += 32) {
      double s = 0.0;
      for (uint32_t i = 0; i < mm; ++i) s += abs2(w.M[i * w.ldm + j]);
      w.nrm[j] = s;
      w.inv[j] = sqrt(s);
    }
    __syncwarp();
    for (uint32_t j = lane; j < nn; j += 32) {
      uint32_t at = 0;
      const double s = w.inv[j];
      for (uint32_t q = 0; q < nn; ++q) {
        const double o = w.inv[q];
        at += gt_nonneg(o, s) || (__double_as_longlong(o) == __double_as_longlong(s) && q < j);
      }
      w.perm[at] = (int)j;
    }
    __syncwarp();
    const double s0 = nn ? w.inv[w.perm[0]] : 0.0;
    uint32_t kept = 0;
    for (uint32_t j = lane; j < nn; j += 32) {
      const double s = w.inv[j];
      kept += !(s <= delta * s0 || s < 1e-64);
    }
    kept = min(__reduce_add_sync(0xffffffffu, kept), mm);
    __syncwarp();
    for (uint32_t j = lane; j < nn; j += 32) w.inv[j] = 1.0 / w.nrm[j];
    if (lane == 0) w.perm[nn] = (int)kept;
    __syncwarp();
    // Z(:, j) = M0^H (W S)(:, j) / s_j^2
    for (uint32_t e = lane; e < nn * kept; e += 32) {
      const uint32_t i = e / kept, j = e - i * kept, c = (uint32_t)w.perm[j];
      T s = zero_of(T());
      for (uint32_t r = 0; r < mm; ++r) s = maddc(s, w.M0[r * w.ld + i], w.M[r * w.ldm + c]);
      w.C2[i * w.ld + j] = scale_(s, w.inv[c]);
    }
    __syncwarp();
    if (chol) {
      // R1^-1 (W S) in place of M's columns, R2^-1 Z in place of C2's
      for (uint32_t q = lane; q < 2 * kept; q += 32) {
        const uint32_t side = q >= kept, j = side ? q - kept : q;
        T* x = side ? w.C2 + j : w.M + w.perm[j];
        const size_t sx = side ? w.ld : w.ldm;
        const size_t sr = side ? 1 : w.ld, sc = side ? w.ld : 1;
        const double* di = w.dinv + side * (k <= 32 ? 32 : k);
        for (int c = (int)k - 1; c >= 0; --c) {
          T s = x[c * sx];
          for (uint32_t l = c + 1; l < k; ++l) s = msub(s, w.P[c * sr + l * sc], x[l * sx]);
          x[c * sx] = scale_(s, di[c]);
        }
      }
    }
  }
  g.sync();
  kt = (uint32_t)w.perm[nn];
  T *Un, *Vn;
  if (!alloc(kt, Un, Vn)) return false;
  if (kt == 0) return true;
  if (chol) {
    times(g, n1, k, U, w.M, w.ldm, w.perm, kt, Un);
    times(g, n2, k, V, w.C2, w.ld, nullptr, kt, Vn);
  } else {
    for (uint32_t j = 0; j < kt; ++j) {
      const uint32_t c = (uint32_t)w.perm[j];
      for (uint32_t i = g.rank; i < n1; i += Team<W>::G)
        Un[(size_t)j * n1 + i] = i < mm ? w.M[i * w.ldm + c] : zero_of(T());
      for (uint32_t i = g.rank; i < n2; i += Team<W>::G)
        Vn[(size_t)j * n2 + i] = i < nn ? w.C2[i * w.ld + j] : zero_of(T());
    }
    apply_q(g, n1, mm, U, tau, kt, Un);
    apply_q(g, n2, nn, V, tau + k, kt, Vn);
  }
  return true;
}

// One admissible leaf in the workspace at ws (aca_ws_bytes): ACA, recompression,
// factors through alloc(kt, Un, Vn).
template <int W, class Gen, class Alloc>
__device__ void leaf(Team<W>& g, const Gen& gen, const AcaTask& t, double eps, int variant, void* ws,
                     typename Gen::T* smem, Alloc alloc, int& st, uint32_t& k, uint32_t& kt) {
  using T = typename Gen::T;
  const uint32_t kc = t.kcap, kw = aca_work_k(t.n1, t.n2, kc);
  Blk<Gen> B;
  B.gen = gen;
  B.b1 = t.b1;
  B.n1 = t.n1;
  B.b2 = t.b2;
  B.n2 = t.n2;
  B.U = static_cast<T*>(ws);
  B.V = B.U + (size_t)t.n1 * kc;
  T* const sq = B.V + (size_t)t.n2 * kc;
  const size_t k2 = (size_t)kw * kw;
  T* const tau = sq + 4 * k2;
  double* const dbl = reinterpret_cast<double*>(tau + 2 * (size_t)kw);
  B.Z = reinterpret_cast<int*>(dbl + 5 * (size_t)kw);
  B.S = B.Z + t.n1;
  B.P = sq;
  B.d2 = dbl;
  B.ld = kw;
  g.sync();
  k = kt = 0;
  st = variant == kAcaVariantSym ? acar(g, B, t.i0, t.kmax, kc, eps, k) : aca(g, B, t.i0, t.kmax, kc, eps, k);
  if (st != kAcaOk || k == 0) return;
  Work<T> w;
  w.P = sq;
  w.M0 = sq + k2;
  w.M = sq + 2 * k2;
  w.C2 = sq + 3 * k2;
  w.d2 = dbl;
  w.dinv = dbl + kw;
  w.nrm = dbl + 3 * (size_t)kw;
  w.inv = dbl + 4 * (size_t)kw;
  w.perm = B.Z;  // k + 1 <= n1 + n2 ints
  w.ld = w.ldm = kw;
  if (!compress(g, t.n1, t.n2, k, B.U, B.V, w, tau, eps, smem, alloc, kt)) st = kAcaNoSpace;
}

// ---------------------------------------------------------------------------
// All leaves of an assembly in one launch of resident CTAs of four warps.  Phase 1: a
// CTA per leaf for the nlarge first tasks; phase 2: a warp per leaf.  Tasks are in
// descending order of workspace, so that the slot of the first task a team takes holds
// every later one; after the first, tasks are drawn from a counter.  Workspace is that
// of the resident teams, not of all leaves.
template <class Gen>
__global__ void __launch_bounds__(kAcaThreads) aca_kernel(Gen gen, AcaParams p) {
  using T = typename Gen::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long box;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (blockIdx.x < p.nslot_l) {
    // reductions use the second warp's share of the shared memory, the k x k work the first's
    Team<kAcaThreads / 32> g(threadIdx.x, reinterpret_cast<double*>(smem_raw + team_smem<T>()));
    T* const sm = reinterpret_cast<T*>(smem_raw);
    uint32_t t = blockIdx.x;
    while (t < p.nlarge) {
      const AcaTask task = p.tasks[t];
      uint64_t off = 0;
      int st;
      uint32_t k, kt;
      leaf(g, gen, task, p.eps, p.variant, p.ws + p.slots[blockIdx.x], sm,
           [&](uint32_t r, T*& Un, T*& Vn) {
             const uint64_t need = (uint64_t)r * ((uint64_t)task.n1 + task.n2);
             __syncthreads();
             if (threadIdx.x == 0) box = atomicAdd(p.used, (unsigned long long)need);
             __syncthreads();
             off = box;
             Un = static_cast<T*>(p.arena) + off;
             Vn = Un + (uint64_t)r * task.n1;
             return off + need <= p.cap;
           },
           st, k, kt);
      if (threadIdx.x == 0) p.res[t] = AcaResult{st, k, kt, 0u, off};
      __syncthreads();
      if (threadIdx.x == 0) box = p.nslot_l + atomicAdd(p.ctr, 1u);
      __syncthreads();
      t = (uint32_t)box;
    }
  }
  __syncthreads();
  const uint32_t slot = blockIdx.x * (kAcaThreads / 32) + warp;
  if (slot >= p.nslot_s) return;
  Team<1> g(lane, nullptr);
  T* const sm = reinterpret_cast<T*>(smem_raw + warp * team_smem<T>());
  const AcaTask* const tasks = p.tasks + p.nlarge;
  AcaResult* const res = p.res + p.nlarge;
  uint32_t t = slot;
  while (t < p.nsmall) {
    const AcaTask task = tasks[t];
    uint64_t off = 0;
    int st;
    uint32_t k, kt;
    leaf(g, gen, task, p.eps, p.variant, p.ws + p.slots[p.nslot_l + slot], sm,
         [&](uint32_t r, T*& Un, T*& Vn) {
           const uint64_t need = (uint64_t)r * ((uint64_t)task.n1 + task.n2);
           unsigned long long o = 0;
           if (lane == 0) o = atomicAdd(p.used, (unsigned long long)need);
           off = __shfl_sync(0xffffffffu, o, 0);
           Un = static_cast<T*>(p.arena) + off;
           Vn = Un + (uint64_t)r * task.n1;
           return off + need <= p.cap;
         },
         st, k, kt);
    if (lane == 0) res[t] = AcaResult{st, k, kt, 0u, off};
    if (lane == 0) t = p.nslot_s + atomicAdd(p.ctr + 1, 1u);
    t = __shfl_sync(0xffffffffu, t, 0);
  }
}

template <class Gen>
cudaError_t launch_aca_kernel(const Gen& gen, const AcaParams& p, uint32_t grid, cudaStream_t s) {
  constexpr size_t smem = team_smem<typename Gen::T>() * (kAcaThreads / 32);
  cudaError_t e = cudaFuncSetAttribute(aca_kernel<Gen>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  aca_kernel<Gen><<<grid, kAcaThreads, smem, s>>>(gen, p);
  return cudaGetLastError();
}

// CTAs of aca_kernel that fit the device at once
template <class Gen>
cudaError_t resident_aca_kernel(int device, uint32_t& n) {
  constexpr size_t smem = team_smem<typename Gen::T>() * (kAcaThreads / 32);
  cudaError_t e = cudaFuncSetAttribute(aca_kernel<Gen>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per = 0, sms = 0;
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, aca_kernel<Gen>, kAcaThreads, smem);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  n = (uint32_t)(per > 0 ? per : 1) * (uint32_t)(sms > 0 ? sms : 1);
  return e;
}

}  // namespace lowrank
}  // namespace ahx
