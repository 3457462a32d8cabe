// FP64 product with one right-hand side over the layout of the digit-sliced product
// (ahx_dg.cuh): Y += d op(A) X, op = A, A^T (mltaGeHVec / mltaGeHtVec,
// H/mltaGeHVec.cpp:16-150), with plain FP64 multiply-adds.
//
// Two sweeps, a CTA of 192 threads per piece (<= 48 rows over a range of K):
//   V sweep     T = Q^T X: a lane quad per factor column reads 32 consecutive bytes of it,
//               eight columns a warp load, two of them per lane
//   rows sweep  Y += P T + D X: a thread per row and K slice, neighbouring rows of a column
//               in neighbouring lanes; the values that meet them are gathered into shared
//               memory first
// What bounds it: one multiply-add per value on the FP64 pipe, 412 us for the 2.09 GB of
// 65,536 points at two lanes a clock and SM, above their memory time (307 us); the rows
// sweep keeps the pipe 94 % busy, the V sweep 88 %.  The plain kernel (ahx_matvec.cu: a
// CTA per leaf) reads its factors in a chain of dependent steps and half fills its
// warps.  A x, 65,536 points: 628 -> 524 us; 10,007: 128 -> 92; 4,096: 65 -> 39 us.
#include <algorithm>
#include <cstdlib>

#include "ahx_dg.cuh"
#include "ahx_hmat.hpp"

namespace ahx {
namespace {

constexpr uint32_t kThreads = 192;

struct KArgs {
  const DgPiece* pieces;
  const uint64_t* rowptr;
  const DgPos* pos;
  const double* arena;
  const double* X;
  double* T;
  double* Y;
  double d;
  uint32_t n;
};

__global__ void __launch_bounds__(kThreads, 5) f1_v_kernel(const KArgs a) {
  constexpr int B = 4;  // loads in flight per row
  __shared__ double xs[kDgK];
  __shared__ double part[kDgRows];
  const DgPiece pc = a.pieces[blockIdx.x];
  // three warps of 16 rows, twice: the second ones take every other 16 positions
  const uint32_t tid = threadIdx.x, h = tid >= kThreads / 2, warp = (tid >> 5) - 3 * h, lane = tid & 31, g = lane >> 2,
                 c = lane & 3;
  const bool active = warp * 16 < pc.nrows;
  const uint32_t ra = min(warp * 16 + g, pc.nrows - 1), rb = min(warp * 16 + g + 8, pc.nrows - 1);
  const double* pa = a.arena + (a.rowptr[pc.row0 + ra] & ~kDgConj) + pc.k0;
  const double* pb = a.arena + (a.rowptr[pc.row0 + rb] & ~kDgConj) + pc.k0;
  for (uint32_t k = tid; k < pc.kn; k += kThreads) xs[k] = a.X[pc.in0 + pc.k0 + k];
  double sa = 0.0, sb = 0.0, va[B], vb[B];
  const uint32_t full = pc.kn > 4 * (B - 1) ? pc.kn - 4 * (B - 1) : 0u;  // k < full: B steps of 4 fit
  uint32_t k = c + 4 * B * h;
  auto load = [&](uint32_t e) {
#pragma unroll
    for (int u = 0; u < B; ++u) {
      va[u] = __ldg(pa + e + 4 * u);
      vb[u] = __ldg(pb + e + 4 * u);
    }
  };
  if (active && k < full) load(k);
  __syncthreads();
  if (active) {
    for (; k < full; k += 8 * B) {
      double wa[B], wb[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        wa[u] = va[u];
        wb[u] = vb[u];
      }
      if (k + 8 * B < full) load(k + 8 * B);
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const double x = xs[k + 4 * u];
        sa = fma(wa[u], x, sa);
        sb = fma(wb[u], x, sb);
      }
    }
    // what is left of the last 16 positions
    const uint32_t end = min(pc.kn, (k & ~(4u * B - 1)) + 4 * B);
#pragma unroll 4
    for (; k < end; k += 4) {
      const double x = xs[k];
      sa = fma(__ldg(pa + k), x, sa);
      sb = fma(__ldg(pb + k), x, sb);
    }
    // lanes c = 0, 1 end with the sums of rows ra, rb
    const bool up = c & 1;
    const double send = up ? sa : sb, keep = up ? sb : sa;
    sa = keep + __shfl_xor_sync(0xffffffffu, send, 1);
    sa += __shfl_xor_sync(0xffffffffu, sa, 2);
  }
  const uint32_t row = warp * 16 + g + 8 * c;
  const bool mine = active && c < 2 && row < pc.nrows;
  if (h && mine) part[row] = sa;
  __syncthreads();
  if (!h && mine) {
    sa += part[row];
    if (pc.add) atomicAdd(a.T + pc.row0 + row, sa);
    else a.T[pc.row0 + row] = sa;
  }
}

// RS1: every position's rows are consecutive in the arena
template <bool RS1>
__global__ void __launch_bounds__(kThreads) f1_rows_kernel(const KArgs a) {
  constexpr int B = 8;  // loads in flight
  __shared__ uint64_t off[kDgK];
  __shared__ double zv[kDgK];
  __shared__ uint32_t rs[RS1 ? 1 : kDgK];
  __shared__ double part[kThreads];
  const DgPiece pc = a.pieces[blockIdx.x];
  // thread = (slice of K, row): as many slices as fit, since lanes without a row would take
  // the FP64 pipe's time all the same
  const uint32_t tid = threadIdx.x, S = min(kThreads / pc.nrows, 16u), s = tid / pc.nrows, row = tid - s * pc.nrows;
#pragma unroll 4
  for (uint32_t k = tid; k < pc.kn; k += kThreads) {
    const DgPos P = a.pos[pc.k0 + k];
    off[k] = P.off;
    zv[k] = P.z < a.n ? a.X[P.z] : a.T[P.z - a.n];
    if (!RS1) rs[k] = P.rsf & 0x7fffffffu;
  }
  __syncthreads();
  double acc = 0.0;
  if (s < S) {
    const double* const A = a.arena + (RS1 ? row : 0u);
    auto value = [&](uint32_t k) { return __ldg(A + off[k] + (RS1 ? 0ull : (uint64_t)row * rs[RS1 ? 0 : k])); };
    // four consecutive positions a turn: where rows are not consecutive, those are a sector
    const uint32_t step = 4 * S;
    uint32_t k = 4 * s;
    double v[B];
    const uint32_t full = pc.kn > step + 3 ? pc.kn - step - 3 : 0u;  // k < full: two turns fit
    auto load = [&](uint32_t e) {
#pragma unroll
      for (int u = 0; u < B; ++u) v[u] = value(e + (u >> 2) * step + (u & 3));
    };
    if (k < full) load(k);
    for (; k < full; k += 2 * step) {
      double w[B];
#pragma unroll
      for (int u = 0; u < B; ++u) w[u] = v[u];
      if (k + 2 * step < full) load(k + 2 * step);
#pragma unroll
      for (int u = 0; u < B; ++u) acc = fma(w[u], zv[k + (u >> 2) * step + (u & 3)], acc);
    }
    for (; k < pc.kn; k += step)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u < pc.kn) acc = fma(value(k + u), zv[k + u], acc);
  }
  part[tid] = acc;
  __syncthreads();
  if (s == 0) {
    for (uint32_t q = 1; q < S; ++q) acc += part[q * pc.nrows + row];
    atomicAdd(a.Y + pc.row0 + row, a.d * acc);
  }
}

}  // namespace

cudaError_t launch_matvec_f1(const DgPlan& pl, double d, const double* X, double* Y, cudaStream_t s) {
  KArgs k{};
  k.rowptr = pl.rowptr;
  k.pos = pl.pos;
  k.arena = static_cast<const double*>(pl.arena);
  k.X = X;
  k.T = reinterpret_cast<double*>(pl.work);
  k.Y = Y;
  k.d = d;
  k.n = pl.n;
  cudaError_t e;
  if (pl.nv) {
    if (pl.t_split && (e = cudaMemsetAsync(k.T, 0, (size_t)pl.t_split * 8, s)) != cudaSuccess) return e;
    k.pieces = pl.vpieces;
    f1_v_kernel<<<pl.nv, kThreads, 0, s>>>(k);
    count_product_launches(1);
  }
  k.pieces = pl.rpieces;
  if (pl.rs1) f1_rows_kernel<true><<<pl.nr, kThreads, 0, s>>>(k);
  else f1_rows_kernel<false><<<pl.nr, kThreads, 0, s>>>(k);
  count_product_launches(1);
  return cudaGetLastError();
}

// A from 10^6 elements on (1,025 points: 53 us with a CTA per leaf, 23 so), A^T from 2 10^7
// (6,000 points, 1.4 10^7 elements: 50 us with a CTA per leaf, 60 so; 10,007 points: 152, 99:
// the dense leaves' rows are far apart here).  AHX_F1_MIN overrides both (and lays out at
// the first product).
bool f1_wanted(uint64_t elems, bool transposed) {
  const char* e = std::getenv("AHX_F1_MIN");
  if (e && *e) return elems >= std::strtoull(e, nullptr, 10);
  return elems >= (transposed ? 20000000ull : 1000000ull);
}

}  // namespace ahx
