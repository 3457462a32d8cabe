// Complex H-matrix product Y += d op(A) X with op = A (mltaGeHVec / mltaGeHGeM),
// A^H (mltaGeHhVec / mltaGeHhGeM) or A^T (mltaGeHtVec / mltaGeHtGeM) for the
// complex leaves of H/mltaGeHVec.cpp:16-150 and H/mblock.cpp:126-215: a low-rank
// leaf U V^H applies as U (V^H x), V (U^H x) or conj(V) (U^T x); a dense leaf D
// as D x, D^H x or D^T x (Include/mblock.h:99-130).
//
// One CTA per leaf, leaves in descending cost order.  Right-hand sides in
// groups of PG; the input rows of a leaf are staged in shared memory; the
// low-rank inner products T = Q^H X (Q the input-side factor) split every
// output over several threads and sum the parts in a fixed order; the output
// side has one row per thread (coalesced factor reads).  Complex128 leaves
// accumulate in FP64, complex64 leaves in FP32; contributions reach Y through
// FP64 atomics (leaves share rows).
//
// Complex64 leaves with more than four right-hand sides: FP64 instructions bound the
// kernel (one warp instruction occupies the SM's FP64 pipe for 16 clocks, 64 FP32 issue
// slots, also when it is predicated off; rounding X per leaf, widening the sums and
// multiplying by d kept that pipe 73 % busy).  With PRE, X is rounded to complex64 once
// (zc_x_kernel), sums are widened by integer operations, and d = 1 is not multiplied.
// 16,384 points: 16 right-hand sides 665 -> 462 us, 8: 366 -> 269 us (then bound by the
// L1: broadcast loads, atomic additions).  Up to four right-hand sides it gains nothing
// (p = 3: 170 -> 171 us), below 3 10^7 (elements x right-hand sides) the extra launch
// outweighs it (1,025 points, p = 8: 54 -> 56 us).
#include <algorithm>
#include <type_traits>

#include "ahx_matvec.cuh"

namespace ahx {
namespace {

constexpr int kThreads = 128;
constexpr int kCh = 64;  // input rows per staged chunk
constexpr int kXW = 16;  // right-hand sides of the rounded copy

template <typename R>
struct C2 {
  R re, im;
};

// acc += a x
template <typename R>
__device__ __forceinline__ void cfma(C2<R>& acc, const C2<R>& a, const C2<R>& x) {
  acc.re = fma(a.re, x.re, acc.re);
  acc.re = fma(-a.im, x.im, acc.re);
  acc.im = fma(a.re, x.im, acc.im);
  acc.im = fma(a.im, x.re, acc.im);
}

__device__ __forceinline__ C2<double> ldz(const double2* p, bool cj) {
  const double2 v = __ldg(p);
  return C2<double>{v.x, cj ? -v.y : v.y};
}
__device__ __forceinline__ C2<float> ldz(const float2* p, bool cj) {
  const float2 v = __ldg(p);
  return C2<float>{v.x, cj ? -v.y : v.y};
}

// a float as a double by integer operations.  Zeros, denormals, infinities and NaN are
// converted in a function of its own: predicated in line, the conversion would occupy
// the FP64 pipe for every value.
__device__ __noinline__ double widen_other(float f) { return (double)f; }
__device__ __forceinline__ double widen(float f) {
  const uint32_t b = __float_as_uint(f), e = (b >> 23) & 0xffu;
  if (e == 0u || e == 255u) return widen_other(f);
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
__device__ __noinline__ void scale_pair(double dre, double dim, double& ar, double& ai) {
  const double t = dre * ar - dim * ai;
  ai = dre * ai + dim * ar;
  ar = t;
}

// Xs[j][r] = X[row0 + j, r0 + r] for j < jn (zero for r >= pg); PRE: from the rounded
// copy, rows of kXW
struct Rounded {
  const float2* xf;
  bool d_one;  // d = 1
};
template <typename R, int PG, bool PRE>
__device__ __forceinline__ void stage(C2<R> (*Xs)[PG], const ZArgs& a, const Rounded& w, uint32_t r0, uint32_t pg,
                                      uint32_t row0, uint32_t jn) {
  if constexpr (PRE) {
    for (uint32_t e = threadIdx.x; e < jn * PG; e += kThreads) {
      const uint32_t j = e / PG, r = e % PG;
      const float2 x = __ldg(w.xf + (uint64_t)(row0 + j) * kXW + r0 + r);
      Xs[j][r] = C2<R>{x.x, x.y};
    }
  } else {
    for (uint32_t e = threadIdx.x; e < jn * PG; e += kThreads) {
      const uint32_t j = e % jn, r = e / jn;
      C2<R> v{(R)0, (R)0};
      if (r < pg) {
        const double2 x = a.X[(uint64_t)(r0 + r) * a.ldX + row0 + j];
        v = C2<R>{(R)x.x, (R)x.y};
      }
      Xs[j][r] = v;
    }
  }
}

// Y[row, r0 + r] += d acc[r]
template <typename R, int PG, bool PRE>
__device__ __forceinline__ void emit(const ZArgs& a, const Rounded& w, uint32_t r0, uint32_t pg, uint64_t row,
                                     const C2<R>* acc) {
#pragma unroll
  for (int r = 0; r < PG; ++r) {
    if ((uint32_t)r < pg) {
      double ar, ai;
      if constexpr (PRE) {
        ar = widen(acc[r].re);
        ai = widen(acc[r].im);
        if (!w.d_one) scale_pair(a.dre, a.dim, ar, ai);
      } else {
        const double xr = (double)acc[r].re, xi = (double)acc[r].im;
        ar = a.dre * xr - a.dim * xi;
        ai = a.dre * xi + a.dim * xr;
      }
      double* y = &a.Y[(uint64_t)(r0 + r) * a.ldY + row].x;
      atomicAdd(y, ar);
      atomicAdd(y + 1, ai);
    }
  }
}

template <typename S, typename R, int PG, int OP, bool GUARD, bool PRE>
__device__ __forceinline__ void zmv_leaf(const ZArgs& a, const Guard& gd, const Rounded& w, uint32_t leaf,
                                         C2<R> (*Xs)[PG], C2<R>* Ts, C2<R>* red) {
  const MvLeaf L = a.leaves[a.order[leaf]];
  const S* base = reinterpret_cast<const S*>(a.arena) + L.off;
  const uint32_t tid = threadIdx.x;
  constexpr bool kFwd = OP == kZOpN;
  // output rows (ro, nr) and input rows (co, nc) of op(A)
  const uint32_t ro = kFwd ? L.b1 : L.b2, nr = kFwd ? L.n1 : L.n2;
  const uint32_t co = kFwd ? L.b2 : L.b1, nc = kFwd ? L.n2 : L.n1;
  for (uint32_t r0 = 0; r0 < a.p; r0 += PG) {
    if (GUARD && !gd.flags[r0 / gd.cols * gd.step]) continue;
    const uint32_t pg = min((uint32_t)PG, a.p - r0);
    if (L.rank < 0) {
      // dense: thread per output row; the forward product reads D by rows
      // (coalesced across threads), the adjoint ones read column ro + i of D
      for (uint32_t ib = 0; ib < nr; ib += kThreads) {
        const uint32_t i = ib + tid;
        C2<R> acc[PG];
#pragma unroll
        for (int r = 0; r < PG; ++r) acc[r] = C2<R>{(R)0, (R)0};
        for (uint32_t jb = 0; jb < nc; jb += kCh) {
          const uint32_t jn = min((uint32_t)kCh, nc - jb);
          __syncthreads();
          stage<R, PG, PRE>(Xs, a, w, r0, pg, co + jb, jn);
          __syncthreads();
          if (i < nr) {
            for (uint32_t j = 0; j < jn; ++j) {
              const C2<R> av = kFwd ? ldz(base + i + (uint64_t)(jb + j) * L.n1, false)
                                    : ldz(base + (jb + j) + (uint64_t)i * L.n1, OP == kZOpH);
#pragma unroll
              for (int r = 0; r < PG; ++r) cfma(acc[r], av, Xs[j][r]);
            }
          }
        }
        if (i < nr) emit<R, PG, PRE>(a, w, r0, pg, ro + i, acc);
      }
    } else if (L.rank > 0) {
      const uint32_t k = (uint32_t)L.rank;
      // P: output-side factor (nr rows), Q: input-side factor (nc rows)
      const S* P = kFwd ? base : base + (uint64_t)L.n1 * k;
      const S* Q = kFwd ? base + (uint64_t)L.n1 * k : base;
      constexpr bool kConjP = OP == kZOpT, kConjQ = OP != kZOpT;
      constexpr uint32_t kKt = kThreads / PG;
      for (uint32_t lb = 0; lb < k; lb += kKt) {
        const uint32_t kn = min(kKt, k - lb);
        // thread = (column l, row slice sub): each factor entry is loaded once and
        // multiplied with all PG right-hand sides; the slices are summed in order
        const uint32_t ns = kThreads / kn;
        const uint32_t l = tid % kn, sub = tid / kn;
        C2<R> t[PG];
#pragma unroll
        for (int r = 0; r < PG; ++r) t[r] = C2<R>{(R)0, (R)0};
        for (uint32_t jb = 0; jb < nc; jb += kCh) {
          const uint32_t jn = min((uint32_t)kCh, nc - jb);
          __syncthreads();
          stage<R, PG, PRE>(Xs, a, w, r0, pg, co + jb, jn);
          __syncthreads();
          if (sub < ns) {
            const S* qc = Q + (uint64_t)(lb + l) * nc + jb;
            for (uint32_t j = sub; j < jn; j += ns) {
              const C2<R> q = ldz(qc + j, kConjQ);
#pragma unroll
              for (int r = 0; r < PG; ++r) cfma(t[r], q, Xs[j][r]);
            }
          }
        }
        if (sub < ns) {
#pragma unroll
          for (int r = 0; r < PG; ++r) red[(sub * kn + l) * PG + r] = t[r];
        }
        __syncthreads();
        if (tid < kn * PG) {
          const uint32_t l2 = tid / PG, r2 = tid % PG;
          C2<R> s = red[l2 * PG + r2];
          for (uint32_t q = 1; q < ns; ++q) {
            s.re += red[(q * kn + l2) * PG + r2].re;
            s.im += red[(q * kn + l2) * PG + r2].im;
          }
          Ts[tid] = s;  // Ts[l * PG + r]
        }
        __syncthreads();
        for (uint32_t ib = 0; ib < nr; ib += kThreads) {
          const uint32_t i = ib + tid;
          if (i < nr) {
            C2<R> acc[PG];
#pragma unroll
            for (int rr = 0; rr < PG; ++rr) acc[rr] = C2<R>{(R)0, (R)0};
            const S* pc = P + (uint64_t)lb * nr + i;
            for (uint32_t ll = 0; ll < kn; ++ll) {
              const C2<R> pv = ldz(pc + (uint64_t)ll * nr, kConjP);
#pragma unroll
              for (int rr = 0; rr < PG; ++rr) cfma(acc[rr], pv, Ts[ll * PG + rr]);
            }
            emit<R, PG, PRE>(a, w, r0, pg, ro + i, acc);
          }
        }
        __syncthreads();
      }
    }
  }
}

// CTAs an SM that the compiler is to leave registers for (0: its own choice).  Of its own it
// takes 32 registers in the complex128 A^H with one right-hand side, which costs loads in
// flight (9,000 points on a cube 332 us, with 48 registers 255; 40,000 on a sphere the same),
// and 44 in the complex64 A with two (48 with the bound: sphere of 9,000 points 72 -> 70 us,
// 16,384 142 -> 138, cube of 9,000 68 -> 67, ellipsoid of 5,497 78 both).
template <typename S, int PG, int OP>
constexpr int kMinCtas = (sizeof(S) == 16 && PG == 1) || (sizeof(S) == 8 && PG == 2 && OP == kZOpN) ? 10 : 0;
// What a kernel is passed.  The complex64 A with one right-hand side reads no more of ZRun than
// of ZArgs, but the compiler schedules it better with the longer parameter block (31 registers
// against 32: sphere of 9,000 points 52 -> 50 us, 16,384 101 -> 97, cube of 9,000 83 -> 81);
// A^T with one right-hand side is the other way round (cube of 9,000 points 112 us with ZRun, 88).
template <typename S, int PG, int OP>
using PlainArgs = std::conditional_t<sizeof(S) == 8 && PG == 1 && OP == kZOpN, ZRun, ZArgs>;
template <typename S, typename R, int PG, int OP>
__global__ void __launch_bounds__(kThreads, kMinCtas<S, PG, OP>) zmv_kernel(PlainArgs<S, PG, OP> a) {
  __shared__ C2<R> Xs[kCh][PG];
  __shared__ C2<R> Ts[kThreads];       // kThreads / PG columns x PG right-hand sides
  __shared__ C2<R> red[kThreads * PG];  // per-slice partial inner products
  zmv_leaf<S, R, PG, OP, false, false>(a, Guard{}, Rounded{}, blockIdx.x, Xs, Ts, red);
}

// the right-hand sides of the passes whose flag is set
template <typename S, typename R, int PG, int OP>
__global__ void __launch_bounds__(kThreads) zmv_guard_kernel(ZArgs a, Guard gd) {
  __shared__ C2<R> Xs[kCh][PG];
  __shared__ C2<R> Ts[kThreads];
  __shared__ C2<R> red[kThreads * PG];
  bool any = false;
  for (uint32_t q = threadIdx.x; q * gd.cols < a.p; q += kThreads) any = any || gd.flags[q * gd.step];
  if (!__syncthreads_or(any)) return;
  for (uint32_t l = blockIdx.x; l < a.nleaves; l += gridDim.x)
    zmv_leaf<S, R, PG, OP, true, false>(a, gd, Rounded{}, l, Xs, Ts, red);
}

// X rounded beforehand
template <int PG, int OP>
__global__ void __launch_bounds__(kThreads) zmv_rounded_kernel(ZArgs a, Rounded w) {
  __shared__ C2<float> Xs[kCh][PG];
  __shared__ C2<float> Ts[kThreads];
  __shared__ C2<float> red[kThreads * PG];
  zmv_leaf<float2, float, PG, OP, false, true>(a, Guard{}, w, blockIdx.x, Xs, Ts, red);
}

template <typename S, typename R, int OP>
void launch_op(const ZRun& a, cudaStream_t s) {
  if (a.guard.flags) {
    // (complex64: only after right-hand sides of 2^40 or infinity, so that a short launch counts more)
    constexpr uint32_t kCtas = sizeof(R) == 4 ? 152 * 4 : kGuardCtas;
    const uint32_t grid = std::min(a.nleaves, kCtas);
    if (a.p == 1) zmv_guard_kernel<S, R, 1, OP><<<grid, kThreads, 0, s>>>(a, a.guard);
    else if (a.p == 2) zmv_guard_kernel<S, R, 2, OP><<<grid, kThreads, 0, s>>>(a, a.guard);
    else if (a.p <= 4) zmv_guard_kernel<S, R, 4, OP><<<grid, kThreads, 0, s>>>(a, a.guard);
    else zmv_guard_kernel<S, R, 8, OP><<<grid, kThreads, 0, s>>>(a, a.guard);
    return;
  }
  const uint32_t grid = a.nleaves;
  if (a.p == 1) zmv_kernel<S, R, 1, OP><<<grid, kThreads, 0, s>>>(a);
  else if (a.p == 2) zmv_kernel<S, R, 2, OP><<<grid, kThreads, 0, s>>>(a);
  else if (a.p <= 4) zmv_kernel<S, R, 4, OP><<<grid, kThreads, 0, s>>>(a);
  // wider groups (16) measured slower: fewer columns per pass, lower occupancy
  else zmv_kernel<S, R, 8, OP><<<grid, kThreads, 0, s>>>(a);
}

template <typename S, typename R>
void launch_typed(const ZRun& a, cudaStream_t s) {
  if (a.op == kZOpH) launch_op<S, R, kZOpH>(a, s);
  else if (a.op == kZOpT) launch_op<S, R, kZOpT>(a, s);
  else launch_op<S, R, kZOpN>(a, s);
}

// xf[row * kXW + r] = (complex64) X[row, r], zero for r >= p; rows fastest in its reads, r in
// its writes
__global__ void zc_x_kernel(const double2* __restrict__ X, uint64_t ldX, uint32_t n, uint32_t p,
                            float2* __restrict__ xf) {
  __shared__ float2 t[32][kXW + 1];
  const uint32_t row0 = blockIdx.x * 32;
  for (uint32_t e = threadIdx.x; e < 32 * kXW; e += blockDim.x) {
    const uint32_t i = e & 31, r = e >> 5;
    float2 v = make_float2(0.f, 0.f);
    if (r < p && row0 + i < n) {
      const double2 x = X[(uint64_t)r * ldX + row0 + i];
      v = make_float2((float)x.x, (float)x.y);
    }
    t[i][r] = v;
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < 32 * kXW; e += blockDim.x) {
    const uint32_t i = e / kXW, r = e % kXW;
    if (row0 + i < n) xf[(uint64_t)(row0 + i) * kXW + r] = t[i][r];
  }
}

__global__ void z_to_c64_kernel(const double2* __restrict__ src, uint64_t n, float2* __restrict__ dst) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const double2 v = src[i];
    dst[i] = make_float2((float)v.x, (float)v.y);
  }
}

}  // namespace

cudaError_t launch_matvec_z(const ZRun& a, cudaStream_t s) {
  if (a.op < kZOpN || a.op > kZOpT) return cudaErrorInvalidValue;
  if (a.nleaves == 0 || a.p == 0) return cudaSuccess;
  if (!a.single) {
    launch_typed<double2, double>(a, s);
    count_product_launches(1);
    return cudaGetLastError();
  }
  if (a.guard.flags || a.p <= 4 || a.elems * a.p < 30000000ull || !a.xf) {
    launch_typed<float2, float>(a, s);
    count_product_launches(1);
    return cudaGetLastError();
  }
  for (uint32_t r0 = 0; r0 < a.p; r0 += kXW) {
    ZArgs b = a;
    b.p = std::min<uint32_t>(kXW, a.p - r0);
    b.X = a.X + (uint64_t)r0 * a.ldX;
    b.Y = a.Y + (uint64_t)r0 * a.ldY;
    const Rounded w{a.xf, a.dre == 1.0 && a.dim == 0.0};
    zc_x_kernel<<<(a.n + 31) / 32, 128, 0, s>>>(b.X, b.ldX, a.n, b.p, a.xf);
    if (a.op == kZOpH) zmv_rounded_kernel<8, kZOpH><<<a.nleaves, kThreads, 0, s>>>(b, w);
    else if (a.op == kZOpT) zmv_rounded_kernel<8, kZOpT><<<a.nleaves, kThreads, 0, s>>>(b, w);
    else zmv_rounded_kernel<8, kZOpN><<<a.nleaves, kThreads, 0, s>>>(b, w);
    count_product_launches(2);
  }
  return cudaGetLastError();
}

size_t matvec_z_xf_bytes(uint64_t n) { return n * kXW * sizeof(float2); }

cudaError_t launch_z_to_c64(const double2* src, uint64_t n, float2* dst, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, 152ull * 16);
  z_to_c64_kernel<<<grid, 256, 0, s>>>(src, n, dst);
  return cudaGetLastError();
}

}  // namespace ahx
