// Complex64 H-matrix product on the warp-level tensor cores (TF32), over the layout of
// the digit-sliced product (ahx_dg.cuh): Y += d op(A) X, op = A, A^H, A^T, for the
// complex64 copies of Helmholtz leaves (scomp instantiations H/mltaGeHVec.cpp:908-940).
//
// Two sweeps, each a GEMM D[m][n] = sum_k A[m][k] B[k][n] with a CTA of three warps per
// piece (a tile of <= 48 rows, a warp per 16, over a range of K):
//   V sweep     T = Q^H X: m = factor columns of one column cluster, k = its rows
//   rows sweep  Y += P T + D X: m = rows of a finest row block, k = every rank column
//               and dense column of the leaves over it
// A complex element is two real K positions, re(a) with the row (x.re | x.im) and im(a)
// with (-x.im | x.re); columns 2r and 2r + 1 belong to right-hand side r.  A lane's
// element (re, im) is both its K positions c and c + 4 of an m16n8k8 step, one 8-byte
// load, full sectors in either sweep.
//
// Accuracy: a = ah + al with ah its 11 bits to nearest, and al bh + ah bl + ah bh is
// summed over one step (8 positions) by the tensor core, steps by FP32 additions, chunks of
// eight by FP32 additions whose rounding goes on into the next chunk: what is left out (al
// bl, the last bits of al and bl) is 2^-24 of a term, and no long sum is rounded at every
// term.  Against the complex128 product on the same leaves (8 right-hand sides, 1,024 to
// 16,384 points on sphere, cube and ellipsoid, k 1 to 12; norms per right-hand side):
//   random vectors   1.2e-7 to 1.9e-7   the plain kernel 1.9e-7 to 3.0e-7
//   plane waves      6e-8 to 1.0e-7                      5e-8 to 3.5e-7
//   constants        7e-8 to 1.0e-7                      3e-8 to 3.1e-7
// 5e-8 of it is that the tensor core cuts its sums off (a second MMA that finds half a unit
// of each sum to add halves plane waves' and takes 13 % longer); truncated splits
// gave 4.8e-7, one FP32 sum per piece 2.3e-7.
//
// What bounds it: latency (DRAM 22 %, tensor 30 % busy; 27 warps a multiprocessor).  The
// plain kernel (ahx_matvec_z.cu) reads X and adds to Y once per leaf; its atomic
// additions and shared-memory broadcasts take 72 % of the L1's bandwidth.  Here a row of
// Y meets a few dozen additions, and leaf values go from memory into fragments.
// 16,384 points (445 MB): 16 right-hand sides 433 -> 296 us, 8: 253 -> 199 us (cold
// caches; the whole call 321 us).  The carried rounding and the checks of the range came
// later: the whole call 329 us.
#include <algorithm>

#include "ahx_dg.cuh"
#include "ahx_hmat.hpp"

namespace ahx {
namespace {

constexpr int kThreads = 2 * kDgRows;
constexpr uint32_t kCE = 32;     // elements per staged chunk
constexpr uint32_t kBlock = kZtPassCols;  // right-hand sides per pass

// Range.  The low part of a split operand must not fall below FP32's normal numbers, no sum
// may reach infinity, and an infinite or NaN operand has no split (inf - inf; the GPU's NaN
// 0x7fffffff rounds to -0).  So: elements of the leaves up to 2^kExp and a largest entry of
// 2^-kExp at least in every column (zt_fits), right-hand sides whose largest entries lie in
// [2^-kExp, 2^kExp] or are zero (zt_x_kernel), V^H X below 2^kTExp a piece (the V sweep).  A pass of
// other right-hand sides raises its flag before anything is added to Y, and the plain kernel
// runs instead.
constexpr int kExp = 40, kTExp = 50;
constexpr uint32_t kXLeast = (uint32_t)(127 - kExp) << 23, kXMost = (uint32_t)(127 + kExp) << 23;

// floats of a staged Z row: four rows apart in the banks, 16-byte multiples
template <int NT>
constexpr int kZS = NT == 1 ? 8 : NT == 2 ? 24 : 40;

struct KArgs {
  const DgPiece* pieces;
  const uint64_t* rowptr;
  const DgPos* pos;
  const float2* arena;
  int* flag;    // of the pass (zt_x_kernel writes it)
  float* z;     // Z rows of 8 NT floats: X rows, then T rows (at zt)
  float* zt;
  double2* Y;   // first column of the pass
  uint64_t ldY;
  double dre, dim;
  bool d_one;
  uint32_t p;   // right-hand sides of the pass
};

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// v = hi + lo: hi its 11 bits to nearest; lo (12 bits, signed) to nearest when the tensor
// core drops the low 13 bits of the word
__device__ __forceinline__ void split(float v, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(v - __uint_as_float(hi)) + 0x1000u;
}

// RS1: every position's rows are consecutive in the arena (rows sweep of A)
template <int NT, bool ROWS, bool RS1>
__global__ void __launch_bounds__(kThreads, 9) zt_sweep_kernel(const KArgs a) {
  constexpr int ZS = kZS<NT>;
  __shared__ __align__(16) float z[2][kCE * ZS];
  __shared__ __align__(16) DgPos pos[3][kCE];
  __shared__ float sum[NT * 4][kThreads];  // of the chunks before (registers would be spilled)
  const DgPiece pc = a.pieces[blockIdx.x];
  const int out_of_range = *a.flag;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const uint32_t nch = (pc.kn + kCE - 1) / kCE;
  // this lane's rows of the fragment (rows past the tile repeat its last one)
  const bool active = warp * 16 < pc.nrows;
  const uint32_t ra = min(warp * 16 + g, pc.nrows - 1), rb = min(warp * 16 + g + 8, pc.nrows - 1);
  const float2 *pa = a.arena, *pb = a.arena;
  uint32_t cja = 0, cjb = 0;
  if (!ROWS) {
    const uint64_t qa = a.rowptr[pc.row0 + ra], qb = a.rowptr[pc.row0 + rb];
    cja = (uint32_t)(qa >> 63) << 31;
    cjb = (uint32_t)(qb >> 63) << 31;
    pa += (qa & ~kDgConj) + pc.k0;
    pb += (qb & ~kDgConj) + pc.k0;
  } else if (RS1) {
    pa += ra;
    pb += rb;
  }
  auto copy_pos = [&](uint32_t ch) {
    // (past the piece: its last position again; zero Z rows meet it)
    if (ROWS && tid < kCE) cp16(su32(&pos[ch % 3][tid]), a.pos + pc.k0 + min(ch * kCE + tid, pc.kn - 1));
  };
  auto copy_z = [&](uint32_t ch) {
    for (uint32_t q = tid; q < kCE * 2 * NT; q += kThreads) {
      const uint32_t r = q / (2 * NT), w = q % (2 * NT), k = ch * kCE + r;
      float* const dst = &z[ch & 1][r * ZS + w * 4];
      if (k < pc.kn) {
        const uint64_t zr = ROWS ? pos[ch % 3][r].z : pc.in0 + pc.k0 + k;
        cp16(su32(dst), a.z + zr * (8 * NT) + w * 4);
      } else {
        *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  };
  // elements 16 h + 4 s + c of chunk ch, rows ra and rb
  auto load_a = [&](float2 (&v)[4][2], uint32_t ch, uint32_t h) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t e = 16 * h + 4 * s + c;
      uint32_t sa = cja, sb = cjb;
      if (ROWS) {
        const DgPos& P = pos[ch % 3][e];
        sa = sb = P.rsf & 0x80000000u;
        if (RS1) {
          v[s][0] = __ldg(pa + P.off);
          v[s][1] = __ldg(pb + P.off);
        } else {
          const uint64_t rs = P.rsf & 0x7fffffffu;
          v[s][0] = __ldg(pa + P.off + ra * rs);
          v[s][1] = __ldg(pa + P.off + rb * rs);
        }
      } else {
        const uint32_t k = min(ch * kCE + e, pc.kn - 1);
        v[s][0] = __ldg(pa + k);
        v[s][1] = __ldg(pb + k);
      }
      v[s][0].y = __uint_as_float(__float_as_uint(v[s][0].y) ^ sa);
      v[s][1].y = __uint_as_float(__float_as_uint(v[s][1].y) ^ sb);
    }
  };
  float acc[NT][4];  // of the present chunk
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[t][j] = sum[4 * t + j][tid] = 0.f;
  auto multiply = [&](const float2 (&v)[4][2], uint32_t ch, uint32_t h) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      uint32_t ah[4], al[4];
      split(v[s][0].x, ah[0], al[0]);
      split(v[s][1].x, ah[1], al[1]);
      split(v[s][0].y, ah[2], al[2]);
      split(v[s][1].y, ah[3], al[3]);
      const float* zr = &z[ch & 1][(16 * h + 4 * s + c) * ZS + (g & ~1u)];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const float2 x = *reinterpret_cast<const float2*>(zr + 8 * t);
        uint32_t bh[2], bl[2];
        split(g & 1 ? x.y : x.x, bh[0], bl[0]);
        split(g & 1 ? x.x : -x.y, bh[1], bl[1]);
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma(d, al, bh);
        mma(d, ah, bl);
        mma(d, ah, bh);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[t][j] += d[j];
      }
    }
  };
  float2 a0[4][2], a1[4][2];
  copy_pos(0);
  copy_pos(1);
  cp_commit();
  cp_wait_all();
  if (__syncthreads_or(out_of_range)) return;  // (the V sweep may raise it meanwhile)
  copy_z(0);
  cp_commit();
  if (active) {
    load_a(a0, 0, 0);
    load_a(a1, 0, 1);
  }
  for (uint32_t ch = 0; ch < nch; ++ch) {
    cp_wait_all();
    __syncthreads();
    if (ch + 1 < nch) copy_z(ch + 1);
    if (ch + 2 < nch) copy_pos(ch + 2);
    cp_commit();
    if (!active) continue;
    multiply(a0, ch, 0);
    if (ch + 1 < nch) load_a(a0, ch + 1, 0);
    multiply(a1, ch, 1);
    if (ch + 1 < nch) load_a(a1, ch + 1, 1);
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float old = sum[4 * t + j][tid], s = old + acc[t][j];
        acc[t][j] -= s - old;  // (what the addition rounded off goes on with the next chunk)
        sum[4 * t + j][tid] = s;
      }
  }
  if (!active) return;
  // lane: rows g, g + 8, right-hand side 4 t + c
#pragma unroll
  for (int t = 0; t < NT; ++t) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t row = warp * 16 + g + 8 * h;
      if (row >= pc.nrows) continue;
      const float2 v = make_float2(sum[4 * t + 2 * h][tid] + acc[t][2 * h], sum[4 * t + 2 * h + 1][tid] + acc[t][2 * h + 1]);
      if (!ROWS) {
        if (!(fmaxf(fabsf(v.x), fabsf(v.y)) < (float)(1ull << kTExp))) atomicOr(a.flag, 1);
        float2* T = reinterpret_cast<float2*>(a.zt + (uint64_t)(pc.row0 + row) * (8 * NT) + 8 * t + 2 * c);
        if (pc.add) atomicAdd(T, v);
        else *T = v;
      } else if (4 * t + c < a.p) {
        double re = v.x, im = v.y;
        if (!a.d_one) {
          const double x = a.dre * re - a.dim * im;
          im = a.dre * im + a.dim * re;
          re = x;
        }
        double* y = &a.Y[(uint64_t)(4 * t + c) * a.ldY + pc.row0 + row].x;
        atomicAdd(y, re);
        atomicAdd(y + 1, im);
      }
    }
  }
}

// Z rows of X: z[row][r] = (complex64) X[row, r], zero for p <= r < W.  most[r]: the largest
// part of column r (as bits: NaN above infinity); the last CTA looks whether they are in range.
// (128 threads: a warp has 32 rows of one column at a time)
__global__ void __launch_bounds__(128) zt_x_kernel(const double2* __restrict__ X, uint64_t ldX, uint32_t n, uint32_t p,
                                                   uint32_t W, float2* __restrict__ z, uint32_t* __restrict__ most,
                                                   uint32_t* __restrict__ ticket, int* __restrict__ flag) {
  __shared__ float2 t[32][kBlock + 1];
  __shared__ uint32_t part[kBlock];
  const uint32_t row0 = blockIdx.x * 32;
  for (uint32_t e = threadIdx.x; e < 32 * W; e += blockDim.x) {
    const uint32_t i = e & 31, r = e >> 5;
    float2 v = make_float2(0.f, 0.f);
    if (r < p && row0 + i < n) {
      const double2 x = X[(uint64_t)r * ldX + row0 + i];
      v = make_float2((float)x.x, (float)x.y);
    }
    t[i][r] = v;
    const uint32_t m = __reduce_max_sync(
        0xffffffffu, max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu));
    if (i == 0) part[r] = m;
  }
  __syncthreads();
  if (threadIdx.x < p && part[threadIdx.x]) atomicMax(most + threadIdx.x, part[threadIdx.x]);
  for (uint32_t e = threadIdx.x; e < 32 * W; e += blockDim.x) {
    const uint32_t i = e / W, r = e - i * W;
    if (row0 + i < n) z[(uint64_t)(row0 + i) * W + r] = t[i][r];
  }
  if (threadIdx.x >= 32) return;
  __threadfence();
  __syncwarp();
  uint32_t last = threadIdx.x == 0 ? (atomicAdd(ticket, 1u) == gridDim.x - 1 ? 1u : 0u) : 0u;
  if (!__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
  bool bad = false;
  if (threadIdx.x < p) {
    const uint32_t m = __ldcg(most + threadIdx.x);
    bad = m != 0u && (m < kXLeast || m > kXMost);
    most[threadIdx.x] = 0u;  // (for the next product)
  }
  bad = __any_sync(0xffffffffu, bad);
  if (threadIdx.x == 0) {
    *ticket = 0u;
    *flag = bad;
  }
}

// Control words of a pass: column maxima and ticket (zero between products), flag
constexpr uint32_t kPassWords = kZtPassWords;
static_assert(kZtFlagAt == kBlock + 1 && kPassWords == kBlock + 2, "maxima, ticket, flag");

int nt_of(uint32_t p) { return p <= 4 ? 1 : p <= 8 ? 2 : 4; }

template <int NT>
cudaError_t pass(const DgPlan& pl, KArgs k, uint32_t* most, const double2* X, uint64_t ldX, cudaStream_t s) {
  zt_x_kernel<<<(pl.n + 31) / 32, 128, 0, s>>>(X, ldX, pl.n, k.p, 4 * NT, reinterpret_cast<float2*>(k.z), most,
                                               most + kBlock, k.flag);
  k.zt = k.z + (uint64_t)pl.n * (8 * NT);
  cudaError_t e;
  if (pl.nv) {
    if (pl.t_split && (e = cudaMemsetAsync(k.zt, 0, (size_t)pl.t_split * NT * 32, s)) != cudaSuccess) return e;
    k.pieces = pl.vpieces;
    zt_sweep_kernel<NT, false, false><<<pl.nv, kThreads, 0, s>>>(k);
    count_product_launches(1);
  }
  k.pieces = pl.rpieces;
  if (pl.rs1) zt_sweep_kernel<NT, true, true><<<pl.nr, kThreads, 0, s>>>(k);
  else zt_sweep_kernel<NT, true, false><<<pl.nr, kThreads, 0, s>>>(k);
  count_product_launches(2);
  return cudaGetLastError();
}

}  // namespace

size_t zt_work_bytes(uint32_t n, uint32_t t_rows, uint32_t p) { return ((size_t)n + t_rows) * nt_of(p) * 32; }
size_t zt_control_bytes(uint32_t p) { return ((size_t)p + kBlock - 1) / kBlock * kPassWords * sizeof(int); }

bool zt_fits(const DgRange& r) { return r.emax <= kExp && r.wmax - r.drop >= -kExp; }

cudaError_t launch_matvec_zt(const DgPlan& pl, const DgArgs& a, int* control, cudaStream_t s) {
  const double2* X = static_cast<const double2*>(a.X);
  double2* Y = static_cast<double2*>(a.Y);
  KArgs k{};
  k.rowptr = pl.rowptr;
  k.pos = pl.pos;
  k.arena = static_cast<const float2*>(pl.arena);
  k.z = reinterpret_cast<float*>(pl.work);
  cudaError_t e;
  k.ldY = a.ldY;
  k.dre = a.dre;
  k.dim = a.dim;
  k.d_one = a.dre == 1.0 && a.dim == 0.0;
  for (uint32_t r0 = 0; r0 < a.p; r0 += kBlock) {
    k.p = std::min(kBlock, a.p - r0);
    k.Y = Y + (uint64_t)r0 * a.ldY;
    const double2* x = X + (uint64_t)r0 * a.ldX;
    uint32_t* const most = reinterpret_cast<uint32_t*>(control) + r0 / kBlock * kPassWords;
    k.flag = control + r0 / kBlock * kPassWords + kZtFlagAt;
    const int nt = nt_of(k.p);
    e = nt == 1 ? pass<1>(pl, k, most, x, a.ldX, s)
        : nt == 2 ? pass<2>(pl, k, most, x, a.ldX, s)
                  : pass<4>(pl, k, most, x, a.ldX, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Five right-hand sides and 9 10^7 (complex elements x right-hand sides) on.  Where the line
// is best depends on the leaves (cold caches; this against the plain kernel): sphere of 4,096
// points (10^7 elements), p = 8: 70 us against 58, 16: 94 against 91; of 6,007, 8: 105
// against 86, 16: 146 against 135; of 9,000, 5: 123 against 127, 16: 171 against 218; cube
// surface of 6,007 points, 5: 111 against 122, 16: 153 against 204; of 9,000, 5: 140 against
// 196.  AHX_ZT_MIN overrides both (and lays out at the first product).
bool zt_wanted(uint64_t elems, uint32_t p) {
  const char* e = std::getenv("AHX_ZT_MIN");
  if (e && *e) return elems * p >= std::strtoull(e, nullptr, 10);
  return p >= 5 && elems * p >= 90000000ull;
}

}  // namespace ahx
