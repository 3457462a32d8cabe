// Digit-sliced H-matrix product on mma.sync (see ahx_dg.cuh): Y += d op(A) X
// for FP64 and complex128 leaves and two or more right-hand sides (mltaGeHGeM /
// mltaGeHhGeM / mltaGeHtGeM, H/mltaGeHVec.cpp:16-150, 770-805).
//
// Two sweeps, each a GEMM D[m][n] = sum_k A[m][k] B[k][n] with the leaf data
// on M x K and the right-hand sides on N:
//   V sweep     T = Q^T X: m = factor columns of all leaves of one column
//               cluster (48 per tile), k = the cluster's rows
//   rows sweep  Y += P T + D X: m = the rows of one finest row block (<= 48),
//               k = every rank column and dense column of the leaves over it
// One CTA of three warps per piece (tile x K range), a warp per 16 rows: the
// finest clusters of the default leaf size hold 33 to 64 points, 45 on average,
// so that a fourth warp would mostly idle (128 threads: 1.47 ms instead of 1.42,
// 65,536 points, 16 right-hand sides).  A lane loads its eight elements of a
// 16 x 16 fragment straight from the arena (full 32-byte sectors in both
// orientations: the K positions of a fragment are permuted so that a lane quad
// reads four consecutive ones) one step ahead, cuts them into digits in registers
// and multiplies with the Z rows' digits, which the CTA stages in shared memory
// by cp.async.
//
// A complex leaf is the real matrix of its interleaved (re, im) storage: its K
// is twice as long (position 2k: re, 2k + 1: im) and a complex Z row becomes
// the two real rows (x.re | x.im) and (-x.im | x.re), columns 2r and 2r + 1;
// conjugated factors flip the sign of their im elements.
//
// Accuracy.  Digit products are integers of at most 2^16; the sums of the
// weights 2^0, 2^-9, 2^-18, 2^-27 over one step (16 positions, at most four
// digit pairs: <= 2^22) leave the MMA exactly, as offsets from 1.5 * 2^23, and
// are added up in 32-bit integers; those of 2^-36 gather in FP32 for one chunk
// and are then moved to the integers too; those of 2^-45 and 2^-54 stay in FP32.
// Pairs below are left out (2^-63).  So the error is that of the digits: 2^-58 of
// the row's largest term so far per entry, over all columns of the pass; that it stays
// below what the FP64 kernel rounds away in the sums of each column is seen to by
// dg_xprep_kernel.  Against long double on the same leaves (2,000 to 4,096 points,
// 2 to 20 right-hand sides): 0.9e-16 to 2.7e-16 per right-hand side, the FP64
// kernel 1.5e-16 to 5.0e-16.
//
// What bounds it: the ALU work of cutting (about 30 integer operations per
// element; ALU pipe 53%, issue 48%, tensor pipe 22% to 31% busy at 32,768 points).
// 65,536 points (2.09 GB): 8.35 -> 1.36 ms with 16 right-hand sides, 4.21 -> 0.99
// ms with 8 (2.1 TB/s); 8,300 us of it were the FP64 pipe.
#include <algorithm>
#include <cstdlib>
#include <new>

#include <cuda_fp16.h>

#include "ahx_dg.cuh"
#include "ahx_hmat.hpp"

namespace ahx {
namespace {

constexpr int kThreads = 2 * kDgRows;  // a warp per 16 rows
constexpr int kChunk = 64;          // real K positions staged at a time
constexpr int S = 6;                // digits of a value
constexpr int kMagic = 0x4B400000;  // 1.5 * 2^23

// Exponents.  Leaf elements other than zero lie in [2^-500, 2^500] and the
// exponents of the Z rows in [-200, 200] (anything else is left to the plain
// kernel: dg_weigh_kernel, the flag), zero Z rows have kZeroZ.  So exponent + Z
// exponent is at least 323 for a term that counts, at most 200 for a zero element
// and at most 123 for a zero Z row: neither moves a row's exponent, and both are
// more than 63 bits below it.
constexpr int kLeafMin = 523, kLeafMax = 1523;  // double exponent fields
constexpr int kZMin = -200, kZMax = 200;
constexpr int kZeroZ = -1400;
// a row's scale before its first element: above every zero, below every term
constexpr int kFloor = 260 * (1 << 20) + 0xfffff;

// fixed-point words: the digits' fields, 1.0 of the row's scale at 2^58
struct Dig {  // 64-bit: d5 [3,12], d4 [13,22], d3 [23,31] | d2 [0,8], d1 [9,17], d0 [18,28]
  uint32_t lo, hi;
};

// offsets that make the balanced digits non-negative fields, and half a unit of the last one
constexpr unsigned long long kBias = ((((256ull << 18) + (256ull << 9) + 256ull) << 32) |
                                       ((256ull << 23) + (512ull << 13) + (512ull << 3))) + 4ull;

// fixed-point word of a double (hi, lo words) sh = E - its exponent >= 0 bits below the scale
__device__ __forceinline__ Dig fix_f64(uint32_t hi, uint32_t lo, uint32_t sh) {
  const uint32_t mh = (__funnelshift_l(lo, hi, 5) & 0x1ffffffu) | 0x2000000u;
  const unsigned long long m = ((unsigned long long)mh << 32) | (lo << 5);
  unsigned long long v;
  asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(sh));  // (past 63: zero)
  // one's complement for negative values: an eighth of the last digit's unit off
  const uint32_t sg = (uint32_t)((int)hi >> 31);
  v = (v ^ (((unsigned long long)sg << 32) | sg)) + kBias;
  return {(uint32_t)v, (uint32_t)(v >> 32)};
}
__device__ __forceinline__ uint32_t h2sub(uint32_t v, float off) {
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&v), __float2half2_rn(off));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t h2fma(uint32_t v, float a, float b) {
  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&v), __float2half2_rn(a), __float2half2_rn(b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// digit pairs (x low half, y high half) as FP16: a field f < 1024 becomes 1024 + f
// by its bits alone, then the offset comes off; d4 / 2 and d5 / 4 bring both to
// multiples of the weights 2^-36 and 2^-45
__device__ __forceinline__ void digits(const Dig& x, const Dig& y, uint32_t (&d)[S]) {
  constexpr uint32_t k = 0x64006400u;
  d[0] = h2sub(((x.hi >> 18) & 0x3ffu) | ((y.hi >> 2) & 0x03ff0000u) | k, 1280.f);
  d[1] = h2sub(((x.hi >> 9) & 0x1ffu) | ((y.hi << 7) & 0x01ff0000u) | k, 1280.f);
  d[2] = h2sub((x.hi & 0x1ffu) | ((y.hi << 16) & 0x01ff0000u) | k, 1280.f);
  d[3] = h2sub((x.lo >> 23) | ((y.lo >> 7) & 0x01ff0000u) | k, 1280.f);
  d[4] = h2fma(((x.lo >> 13) & 0x3ffu) | ((y.lo << 3) & 0x03ff0000u) | k, 0.5f, -768.f);
  d[5] = h2fma(((x.lo >> 3) & 0x3ffu) | ((y.lo << 13) & 0x03ff0000u) | k, 0.25f, -384.f);
}
__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// d = a b + c
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2],
                                    const float (&c)[4]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c[0]), "f"(c[1]), "f"(c[2]),
        "f"(c[3]));
}

struct KArgs {
  const DgPiece* pieces;
  const uint64_t* rowptr;
  const DgPos* pos;
  const void* arena;
  const unsigned char* z;  // Z rows: S digits x NP FP16 values, then the exponent << 20
  const int* xexp;         // rows sweep: exponent of every column of X
  const int* flag;
  double* T;               // V sweep: T rows, NP doubles each
  double* Y;               // rows sweep (complex: interleaved), first column of the pass
  uint64_t ldY;            // in elements (complex: double2)
  double dre, dim;
  uint32_t pc;             // columns in use (real; <= NP)
};

// Partial sums of one accumulator element: integers (exact) and FP32, in units
// of a product of leading digits; wide(): the integers as one, units of 2^-kU.
constexpr int kU = 36;
struct Acc {
  int i0, i1, i2, i3;
  float f4, f;  // units of 2^-36, 2^-45
  __device__ __forceinline__ void clear() {
    i0 = i1 = i2 = i3 = 0;
    f4 = f = 0.f;
  }
  // the whole units of f4, which keeps the rest: FP32 never holds a long sum
  __device__ __forceinline__ int drain() {
    const float r = rintf(f4);
    f4 -= r;
    return __float2int_rn(r);
  }
  __device__ __forceinline__ long long wide() {
    return ((long long)i0 << 36) + ((long long)i1 << 27) + ((long long)i2 << 18) + ((long long)i3 << 9) +
           (long long)drain();
  }
  __device__ __forceinline__ float rest() const { return fmaf(f4, 512.f, f); }
};
__device__ __forceinline__ void mma_step(const uint32_t (&A)[S][4], const uint32_t (&B)[S][2], Acc (&acc)[4]) {
  const float mg = __int_as_float(kMagic);
  const float C[4] = {mg, mg, mg, mg}, zero[4] = {0.f, 0.f, 0.f, 0.f};
  float t0[4], t1[4], t2[4], t3[4], t4[4], f5[4], f6[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    t4[j] = acc[j].f4;
    f5[j] = acc[j].f;
  }
  mma(t0, A[0], B[0], C);
  mma(t1, A[0], B[1], C);
  mma(t2, A[0], B[2], C);
  mma(t3, A[0], B[3], C);
  mma(t4, A[0], B[4], t4);
  mma(f5, A[0], B[5], f5);
  mma(f6, A[1], B[5], zero);
  mma(t1, A[1], B[0], t1);
  mma(t2, A[1], B[1], t2);
  mma(t3, A[1], B[2], t3);
  mma(t4, A[1], B[3], t4);
  mma(f5, A[1], B[4], f5);
  mma(f6, A[2], B[4], f6);
  mma(t2, A[2], B[0], t2);
  mma(t3, A[2], B[1], t3);
  mma(t4, A[2], B[2], t4);
  mma(f5, A[2], B[3], f5);
  mma(f6, A[3], B[3], f6);
  mma(t3, A[3], B[0], t3);
  mma(t4, A[3], B[1], t4);
  mma(f5, A[3], B[2], f5);
  mma(f6, A[4], B[2], f6);
  mma(t4, A[4], B[0], t4);
  mma(f5, A[4], B[1], f5);
  mma(f6, A[5], B[1], f6);
  mma(f5, A[5], B[0], f5);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[j].i0 += __float_as_int(t0[j]) - kMagic;
    acc[j].i1 += __float_as_int(t1[j]) - kMagic;
    acc[j].i2 += __float_as_int(t2[j]) - kMagic;
    acc[j].i3 += __float_as_int(t3[j]) - kMagic;
    acc[j].f4 = t4[j];
    acc[j].f = fmaf(f6[j], 0x1p-9f, f5[j]);
  }
}
// 16-byte pieces of a Z row (digits, exponent): an odd number, so that ldmatrix
// reads 8 rows x 16 bytes without bank conflicts
template <int NT>
constexpr int kPR = S * NT + 1;
static_assert(S % 2 == 0, "odd row pitch");

template <int NT, int CW>
struct Smem {
  alignas(16) unsigned char z[2][kChunk * kPR<NT> * 16];
  alignas(16) DgPos pos[3][kChunk / CW];
  // sums at a row's earlier exponents, brought to its present one: units of
  // 2^-kU and 2^-(kU + 9)
  long long bi[NT * 4][kThreads];
  float bf[NT * 4][kThreads];
};

// v 2^e without the FP64 pipe where the result is a normal number
__device__ __forceinline__ double scale2(double v, int e) {
  const int hi = __double2hiint(v);
  const int x = ((hi >> 20) & 0x7ff) + e;
  if (v == 0.0) return v;
  if (x < 1 || x > 2046 || e < -2000 || e > 2000) return scalbn(v, e);
  return __hiloint2double(hi + (e << 20), __double2loint(v));
}

// RS1: every position's rows are
// consecutive in the arena (rows sweep of A; not the dense leaves of A^T).
template <int NT, int CW, bool ROWS, bool RS1>
__global__ void __launch_bounds__(kThreads, NT == 1 ? 5 : 4) dg_sweep_kernel(const KArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<Smem<NT, CW>*>(smem_raw);
  constexpr int NP = 8 * NT;
  constexpr uint32_t kCE = kChunk / CW;  // elements (complex: pairs) per chunk
  constexpr uint32_t kRow = kPR<NT> * 16;
  if (*a.flag) return;                   // X not fit for digits: the plain kernel runs instead
  const DgPiece pc = a.pieces[blockIdx.x];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
  const uint32_t nch = (pc.kn + kCE - 1) / kCE;

  // this lane's rows of the fragment (rows past the tile repeat its last one)
  const bool active = warp * 16 < pc.nrows;
  const uint32_t ra = min(warp * 16 + g, pc.nrows - 1), rb = min(warp * 16 + g + 8, pc.nrows - 1);
  uint64_t pa = 0, pb = 0;
  uint32_t cja = 0, cjb = 0;
  if (!ROWS) {
    pa = a.rowptr[pc.row0 + ra];
    pb = a.rowptr[pc.row0 + rb];
    cja = (uint32_t)(pa >> 63) << 31;
    cjb = (uint32_t)(pb >> 63) << 31;
    pa = (pa & ~kDgConj) + pc.k0;
    pb = (pb & ~kDgConj) + pc.k0;
  } else if (RS1) {
    pa = ra;
    pb = rb;
  }
  const uint2* const Aa = reinterpret_cast<const uint2*>(a.arena) + pa * CW + (CW == 2 ? (c & 1) : 0);
  const uint2* const Ab = reinterpret_cast<const uint2*>(a.arena) + pb * CW + (CW == 2 ? (c & 1) : 0);

  auto copy_pos = [&](uint32_t ch) {
    // (past the piece: its last position again; zero Z rows meet it)
    if (ROWS && tid < kCE)
      cp16(su32(&sm.pos[ch % 3][tid]), a.pos + pc.k0 + min(ch * kCE + tid, pc.kn - 1));
  };
  // kLR lanes to a row, a lane per piece
  auto copy_z = [&](uint32_t ch) {
    constexpr uint32_t kLR = kPR<NT> <= 8 ? 8 : kPR<NT> <= 16 ? 16 : 32;
    const uint32_t w = lane % kLR, zb = su32(sm.z[ch & 1]);
    const DgPos* ps = sm.pos[ch % 3];
    if (w < kPR<NT>) {
#pragma unroll 4
      for (uint32_t q = warp * (32 / kLR) + lane / kLR; q < (uint32_t)kChunk; q += kThreads / 32 * (32 / kLR)) {
        const uint32_t k = ch * kCE + q / CW;
        if (k < pc.kn) {
          const uint32_t zr = CW * (ROWS ? ps[q / CW].z : pc.in0 + pc.k0 + k) + q % CW;
          cp16(zb + q * kRow + w * 16, a.z + (uint64_t)zr * kRow + w * 16);
        } else {
          // past the piece: zero A digits meet these rows, which must be numbers
          *reinterpret_cast<uint4*>(sm.z[ch & 1] + q * kRow + w * 16) =
              make_uint4(w == S * NT ? (uint32_t)(kZeroZ * (1 << 20)) : 0u, 0u, 0u, 0u);
        }
      }
    }
  };
  // the eight elements of step s of chunk ch: row ra / rb, positions c + 4 i
  uint32_t raw[8][2];
  auto load_a = [&](uint32_t ch, uint32_t s) {
    const DgPos* ps = sm.pos[ch % 3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t q = s * 16 + c + 4 * i;
      uint2 va, vb;
      uint32_t sa = cja, sb = cjb;
      if (ROWS) {
        const DgPos& P = ps[q / CW];
        if (CW == 2) sa = sb = P.rsf & 0x80000000u;
        if (RS1) {
          va = __ldg(Aa + P.off * CW);
          vb = __ldg(Ab + P.off * CW);
        } else {
          const uint64_t rs = P.rsf & 0x7fffffffu;
          va = __ldg(Aa + (P.off + ra * rs) * CW);
          vb = __ldg(Aa + (P.off + rb * rs) * CW);
        }
      } else {
        const uint64_t k = min(ch * kCE + q / CW, pc.kn - 1);
        va = __ldg(Aa + k * CW);
        vb = __ldg(Ab + k * CW);
      }
      raw[2 * i][0] = va.y;
      raw[2 * i][1] = va.x;
      raw[2 * i + 1][0] = vb.y;
      raw[2 * i + 1][1] = vb.x;
      if (CW == 2 && (c & 1)) {
        raw[2 * i][0] ^= sa;
        raw[2 * i + 1][0] ^= sb;
      }
    }
  };

  Acc acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[t][j].clear();
      sm.bi[t * 4 + j][tid] = 0;
      sm.bf[t * 4 + j][tid] = 0.f;
    }
  // row scale 2^E as its limit (E << 20) + 0xfffff: the largest key that fits
  int La = kFloor, Lb = kFloor;

  copy_pos(0);
  copy_pos(1);
  cp_commit();
  cp_wait_all();
  __syncthreads();
  copy_z(0);
  cp_commit();
  if (active) load_a(0, 0);

  for (uint32_t ch = 0; ch < nch; ++ch) {
    cp_wait_all();
    __syncthreads();
    if (ch + 1 < nch) copy_z(ch + 1);
    if (ch + 2 < nch) copy_pos(ch + 2);
    cp_commit();
    if (!active) continue;
    const uint32_t left = (pc.kn - ch * kCE) * CW;  // real positions from this chunk on
    const uint32_t steps = min((left + 15) / 16, (uint32_t)kChunk / 16);
#pragma unroll 1
    for (uint32_t s = 0; s < steps; ++s) {
      // ---- exponents: keys = (exponent << 20) + leading mantissa bits
      int ka[4], kb[4];
      const unsigned char* zq = sm.z[ch & 1] + (s * 16 + c) * kRow + S * NT * 16;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int zx = *reinterpret_cast<const int*>(zq + 4 * i * kRow);
        const uint32_t ha = raw[2 * i][0] & 0x7fffffffu, hb = raw[2 * i + 1][0] & 0x7fffffffu;
        ka[i] = (int)ha + zx;
        kb[i] = (int)hb + zx;
      }
      int ma = max(max(ka[0], ka[1]), max(ka[2], ka[3])), mb = max(max(kb[0], kb[1]), max(kb[2], kb[3]));
      if (__any_sync(0xffffffffu, ma > La || mb > Lb)) {
        // a row meets a larger exponent: its sums so far are banked at the new scale
        ma = max(ma, __shfl_xor_sync(0xffffffffu, ma, 1));
        ma = max(ma, __shfl_xor_sync(0xffffffffu, ma, 2));
        mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 1));
        mb = max(mb, __shfl_xor_sync(0xffffffffu, mb, 2));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int& L = h ? Lb : La;
          const int m = h ? mb : ma;
          if (m > L) {
            const int N = m | 0xfffff;
            {
              const uint32_t sh = (uint32_t)(N - L) >> 20;
#pragma unroll
              for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int j = 2 * h; j < 2 * h + 2; ++j) {
                  const long long v = sh < 64 ? sm.bi[t * 4 + j][tid] + acc[t][j].wide() : 0;
                  const float f = sm.bf[t * 4 + j][tid] + acc[t][j].rest();
                  // the bits shifted out, as a fraction of the new unit (sh >= 1)
                  const unsigned long long lost = (unsigned long long)v << ((64u - sh) & 63u);
                  sm.bi[t * 4 + j][tid] = v >> min(sh, 63u);
                  sm.bf[t * 4 + j][tid] = f * __int_as_float((127 - (int)min(sh, 126u)) << 23) +
                                          __uint2float_rn((uint32_t)(lost >> 32)) * 0x1p-23f;
                  acc[t][j].clear();
                }
            }
            L = N;
          }
        }
      }
      // ---- digits of the fragment: a0 (row ra, first half of K), a1 (rb), a2 (ra, second half), a3 (rb)
      uint32_t A[S][4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Dig x[2], y[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = 2 * h + e;
          const uint32_t sa = (uint32_t)(La - ka[i]) >> 20, sb = (uint32_t)(Lb - kb[i]) >> 20;
          x[e] = fix_f64(raw[2 * i][0], raw[2 * i][1], sa);
          y[e] = fix_f64(raw[2 * i + 1][0], raw[2 * i + 1][1], sb);
        }
        uint32_t da[S], db[S];
        digits(x[0], x[1], da);
        digits(y[0], y[1], db);
#pragma unroll
        for (int d = 0; d < S; ++d) {
          A[d][2 * h] = da[d];
          A[d][2 * h + 1] = db[d];
        }
      }
      // ---- the next step's elements
      if (s + 1 < steps) load_a(ch, s + 1);
      else if (ch + 1 < nch) load_a(ch + 1, 0);
      // ---- multiply.  Matrix rows of ldmatrix in the lanes' K order: i -> (i >> 1) + 4 (i & 1)
      const uint32_t li = lane & 7, krow = (li >> 1) + 4 * (li & 1) + 8 * ((lane >> 3) & 1);
      const uint32_t zrow = su32(sm.z[ch & 1]) + (s * 16 + krow) * kRow;
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        uint32_t B[S][2];
#pragma unroll
        for (int d = 0; d + 1 < S; d += 2) {
          uint32_t r[4];
          ldsm4t(zrow + ((d + (lane >> 4)) * NT + t) * 16, r);
          B[d][0] = r[0];
          B[d][1] = r[1];
          B[d + 1][0] = r[2];
          B[d + 1][1] = r[3];
        }
        mma_step(A, B, acc[t]);
      }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < 4; ++j) sm.bi[t * 4 + j][tid] += acc[t][j].drain();
  }
  if (!active) return;
  // ---- output: lane holds rows g, g + 8, columns 8 t + 2 c, + 1
#pragma unroll
  for (int t = 0; t < NT; ++t) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t row = warp * 16 + g + 8 * h;
      if (row >= pc.nrows) continue;
      const int L = h ? Lb : La;
      const int ex = (L >> 20) - 1022 - 16;  // a product of leading digits: 2^-16
      const uint32_t col = 8 * t + 2 * c;
      double v[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int e = t * 4 + 2 * h + j;
        const long long i = sm.bi[e][tid] + acc[t][2 * h + j].wide();
        v[j] = fma((double)i, 512.0, (double)(sm.bf[e][tid] + acc[t][2 * h + j].rest()));  // units of 2^-(U + 9)
      }
      if (!ROWS) {
        double* T = a.T + (uint64_t)(pc.row0 + row) * NP + col;
        const double t0 = scale2(v[0], ex - kU - 9), t1 = scale2(v[1], ex - kU - 9);
        if (pc.add) {
          atomicAdd(T, t0);
          atomicAdd(T + 1, t1);
        } else {
          *reinterpret_cast<double2*>(T) = make_double2(t0, t1);
        }
      } else if (CW == 2) {
        if (col < a.pc) {
          const int x = a.xexp[col] + ex - kU - 9;
          const double re = scale2(v[0], x), im = scale2(v[1], x);
          double* y = a.Y + 2 * ((uint64_t)(col / 2) * a.ldY + pc.row0 + row);
          atomicAdd(y, a.dre * re - a.dim * im);
          atomicAdd(y + 1, a.dre * im + a.dim * re);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (col + j < a.pc)
            atomicAdd(a.Y + (uint64_t)(col + j) * a.ldY + pc.row0 + row,
                      a.dre * scale2(v[j], a.xexp[col + j] + ex - kU - 9));
      }
    }
  }
}

// ---- Z rows --------------------------------------------------------------

// exponent field of the largest |X_r| per column r = r0 + blockIdx.y (complex: of both
// parts), and the flag of its pass for a value that is not finite
template <int CW>
__global__ void dg_xmax_kernel(const double* __restrict__ X, uint64_t ldX, uint32_t n, uint32_t r0,
                               int* __restrict__ xmax, int* __restrict__ flags) {
  const uint32_t col = r0 + blockIdx.y;
  const double* x = X + (uint64_t)col * ldX * CW;
  uint32_t m = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (uint64_t)n * CW;
       i += (uint64_t)gridDim.x * blockDim.x)
    m = max(m, ((uint32_t)__double2hiint(x[i]) >> 20) & 0x7ffu);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(xmax + col, (int)m);
    if (m == 0x7ffu) atomicOr(flags + col / dg_pass_cols(CW == 2), 1);
  }
}

__device__ __forceinline__ bool subnormal(double v) {
  const uint32_t hi = (uint32_t)__double2hiint(v);
  return (hi & 0x7ff00000u) == 0u && ((hi << 1) | (uint32_t)__double2loint(v)) != 0u;
}

// Sums over the rows of a pass, of squared entries rounded down to powers of two, times the
// rows' squared weights (relative to the largest weight and column): of each column, and of
// the largest column of each row.
struct PassSums {
  float col[16], all;
  uint32_t ticket, pad[2];
};

// sums over the warp of R values a lane: value u ends in the lanes whose top log2(R) bits are u
template <int R>
__device__ __forceinline__ float warp_sums(float (&v)[R], uint32_t lane) {
  int o = 16;
#pragma unroll
  for (int r = R / 2; r > 0; r >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int u = 0; u < r; ++u) {
      const float keep = up ? v[u + r] : v[u], give = up ? v[u] : v[u + r];
      v[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// X rows, a thread each; real row CW i + e of a complex row: e = 0 (re | im), e = 1 (-im | re):
// the digits of the 8 NT columns and the row's exponent.
//
// One exponent serves a row's columns, and one scale the terms that meet a row of A.  So what a
// column's result loses is relative to the largest terms of all columns of the pass: its norm
// is at most 2^-58 W, W^2 = sum_k c_k^2 z_k^2 with c_k the largest |A_ik| and z_k the row's
// largest entry, each column scaled to 1.  A column r whose own terms are small beside the
// others' (S_r^2 = sum_k c_k^2 z_kr^2; a unit vector beside dense ones, columns of A of very
// different size) would lose bits that the FP64 kernel keeps.  So S_r >= 2^-5 W is asked of
// every column that is not zero (the loss is then below 2^-53 S_r, the FP64 kernel's own
// rounding); the last CTA raises the pass's flag otherwise.  Random right-hand sides have S_r =
// W / 2, at least W / 6 (random clouds of 1,024 to 65,536 points, whose closest pairs weigh
// most).  The sums cost 3 us of 236 (complex128 A^H, 6,007 points, 3 right-hand sides), 7 of
// 1,354 (65,536 points, 16).
constexpr float kLightest = 1024.f;  // W^2 / S_r^2
constexpr int kXPrepThreads = 128;
template <int NT, int CW>
__global__ void __launch_bounds__(kXPrepThreads)
    dg_xprep_kernel(const double* __restrict__ X, uint64_t ldX, uint32_t n, uint32_t pc, const int* __restrict__ xmax,
                    const int* __restrict__ weight, int* __restrict__ xexp, unsigned char* __restrict__ z,
                    PassSums* __restrict__ sums, int* __restrict__ flag) {
  constexpr int NP = 8 * NT, kW = kXPrepThreads / 32;
  __shared__ float part[kW][NP + 1];
  const uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // unit of column col: 2^(xexp - 0), xexp = field - 1022 (complex: the column pair shares it)
  if (q < (uint64_t)NP) xexp[q] = q < pc ? xmax[q / CW] - 1022 : 0;
  const bool live = q < (uint64_t)n * CW;
  // e-major order: consecutive threads read consecutive rows of X
  const uint32_t e = live ? (uint32_t)(q / n) : 0u, i = live ? (uint32_t)(q - (uint64_t)e * n) : 0u;
  bool bad = false;
  auto val = [&](int col, int& sc) -> double {
    sc = __ldg(xmax + col / CW);
    double r;
    if (CW == 1) {
      r = __ldg(X + (uint64_t)col * ldX + i);
    } else {
      const double2 v = __ldg(reinterpret_cast<const double2*>(X) + (uint64_t)(col / 2) * ldX + i);
      r = e == 0 ? ((col & 1) ? v.y : v.x) : ((col & 1) ? v.x : -v.y);
    }
    // a subnormal entry counts as zero: only beside entries 2^99 times larger
    bad = bad || (sc < 100 && subnormal(r));
    return r;
  };
  float t[NP], all = 0.f;
#pragma unroll
  for (int j = 0; j < NP; ++j) t[j] = 0.f;
  if (live) {
    const int wt = max(__ldg(weight + i) - __ldg(weight + n), -4096);
    int m = kZeroZ;
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      if ((uint32_t)j < pc) {
        int sc;
        const double v = val(j, sc);
        const int x = ((uint32_t)__double2hiint(v) >> 20) & 0x7ffu;
        if (x) m = max(m, x - sc);
        const int s2 = 2 * (wt + x - sc);
        if (x && e == 0 && s2 >= -126) t[j] = __int_as_float((127 + min(s2, 0)) << 23);
        all = fmaxf(all, t[j]);
      }
    }
    unsigned char* const zq = z + ((uint64_t)CW * i + e) * (kPR<NT> * 16);
#pragma unroll
    for (int g = 0; g < NT; ++g) {
      uint32_t o[S][4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        Dig f[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const int j = 8 * g + 2 * u + w;
          int sc = 0;
          const double v = (uint32_t)j < pc ? val(j, sc) : 0.0;
          const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
          const int x = (hi >> 20) & 0x7ffu;
          f[w] = fix_f64(hi, lo, x ? (uint32_t)(m - (x - sc)) : 64u);
        }
        uint32_t d[S];
        digits(f[0], f[1], d);
#pragma unroll
        for (int k = 0; k < S; ++k) o[k][u] = d[k];
      }
#pragma unroll
      for (int k = 0; k < S; ++k)
        *reinterpret_cast<uint4*>(zq + (k * NT + g) * 16) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
    }
    *reinterpret_cast<uint4*>(zq + S * NT * 16) = make_uint4((uint32_t)(m * (1 << 20)), 0u, 0u, 0u);
    if (bad || (m != kZeroZ && (m < kZMin || m > kZMax))) atomicOr(flag, 1);
  }
  // ---- the columns' weights
  constexpr int kSh = NT == 1 ? 2 : 1;  // lanes that share a column's sum: 2^kSh
  const float cs = warp_sums<NP>(t, lane);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
  if ((lane & ((1u << kSh) - 1u)) == 0) part[warp][lane >> kSh] = cs;
  if (lane == 0) part[warp][NP] = all;
  __syncthreads();
  if (threadIdx.x <= NP) {
    float s = part[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < kW; ++w) s += part[w][threadIdx.x];
    if (s != 0.f) atomicAdd(threadIdx.x == NP ? &sums->all : &sums->col[threadIdx.x], s);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x != 0 || atomicAdd(&sums->ticket, 1u) != gridDim.x - 1) return;
  __threadfence();
  const float least = __ldcg(&sums->all) / kLightest;
  bool light = false;
  for (uint32_t c = 0; c < pc; c += CW) {
    float s = __ldcg(&sums->col[c]);
    if (CW == 2) s += __ldcg(&sums->col[c + 1]);
    light = light || (xmax[c / CW] != 0 && s < least);
  }
  if (light) atomicOr(flag, 1);
}

// T rows: a lane per column pair (a complex T entry), so that a row is read and each of
// its digit planes written by consecutive lanes; a thread per row left every access of a
// warp in 32 places (65,536 points, 16 right-hand sides: 81 -> 24 us).
template <int NT, int CW>
__global__ void __launch_bounds__(128) dg_tprep_kernel(const double* __restrict__ T, uint32_t t_rows, uint32_t pc,
                                                       unsigned char* __restrict__ z, int* __restrict__ flag) {
  constexpr uint32_t kL = 4 * NT;
  const uint64_t id = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, q = id / kL;
  const uint32_t l = (uint32_t)(id % kL), col = 2 * l;
  const bool live = q < (uint64_t)t_rows * CW;
  double v[2] = {0.0, 0.0};
  if (live && col < pc) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(T + q / CW * (8 * NT) + col));
    v[0] = CW == 2 && (q & 1) ? -t.y : t.x;
    v[1] = CW == 2 ? (q & 1 ? t.x : t.y) : col + 1 < pc ? t.y : 0.0;
  }
  int m = kZeroZ, ex[2];
  bool bad = false;
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    ex[w] = ((uint32_t)__double2hiint(v[w]) >> 20) & 0x7ffu;
    bad = bad || ex[w] == 0x7ff || subnormal(v[w]);
    if (ex[w]) m = max(m, ex[w] - 1022);
  }
#pragma unroll
  for (uint32_t o = 1; o < kL; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (!live) return;
  Dig f[2];
#pragma unroll
  for (int w = 0; w < 2; ++w)
    f[w] = fix_f64((uint32_t)__double2hiint(v[w]), (uint32_t)__double2loint(v[w]),
                   ex[w] ? (uint32_t)(m - (ex[w] - 1022)) : 64u);
  uint32_t d[S];
  digits(f[0], f[1], d);
  unsigned char* zq = z + q * (kPR<NT> * 16);
#pragma unroll
  for (int k = 0; k < S; ++k) *reinterpret_cast<uint32_t*>(zq + k * NT * 16 + l * 4) = d[k];
  if (l == 0) *reinterpret_cast<uint4*>(zq + S * NT * 16) = make_uint4((uint32_t)(m * (1 << 20)), 0u, 0u, 0u);
  if (bad || (m != kZeroZ && (m < kZMin || m > kZMax))) atomicOr(flag, 1);
}

__global__ void dg_expand_kernel(const DgSeg* __restrict__ segs, uint32_t nsegs, DgPos* __restrict__ pos) {
  const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, l = threadIdx.x & 7;
  if (s >= nsegs) return;
  const DgSeg g = segs[s];
  for (uint32_t k = l; k < g.kn; k += 8) pos[(uint64_t)g.pos0 + k] = DgPos{g.base + (uint64_t)k * g.ldk, g.z + k, g.rsf};
}

// exponent field of an element (complex: the larger of its parts'), 0 for zero; b |= it does not
// fit the digits
template <int CW>
__device__ __forceinline__ int leaf_exp(const uint2* a, uint64_t at, bool& b) {
  int m = 0;
#pragma unroll
  for (int c = 0; c < CW; ++c) {
    const uint2 u = __ldg(a + at * CW + c);
    const int e = (u.y >> 20) & 0x7ffu;
    if (((u.y << 1) | u.x) != 0) {
      b = b || e < kLeafMin || e > kLeafMax;
      m = max(m, e);
    }
  }
  return m;
}

// a CTA per leaf; see launch_dg_weigh
constexpr int kWeighThreads = 128;
template <int CW>
__global__ void __launch_bounds__(kWeighThreads)
    dg_weigh_kernel(const DgLeaf* __restrict__ leaves, const uint2* __restrict__ a, int* __restrict__ weight,
                    DgRange* __restrict__ range) {
  constexpr uint32_t kL = 32, kW = kWeighThreads / 32;
  __shared__ int ep[kL];
  const DgLeaf q = leaves[blockIdx.x];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  bool b = false;
  int most = kDgNoWeight, top = 0;
  auto look = [&](uint64_t at) -> int {
    const int e = leaf_exp<CW>(a, at, b);
    top = max(top, e);
    return e;
  };
  auto put = [&](uint32_t i, int w) {
    most = max(most, w);
    if (w > __ldcg(weight + i)) atomicMax(weight + i, w);
  };
  if (q.rank < 0) {
    if (q.mode == kDgN) {
      for (uint32_t j = warp; j < q.n2; j += kW) {
        int m = 0;
#pragma unroll 2
        for (uint32_t i = lane; i < q.n1; i += 32) m = max(m, look(q.off + (uint64_t)j * q.n1 + i));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0 && m) put(q.b2 + j, m - 1023);
      }
    } else {
      for (uint32_t i = tid; i < q.n1; i += kWeighThreads) {
        int m = 0;
#pragma unroll 4
        for (uint32_t j = 0; j < q.n2; ++j) m = max(m, look(q.off + (uint64_t)j * q.n1 + i));
        if (m) put(q.b1 + i, m - 1023);
      }
    }
  } else {
    const uint32_t k = (uint32_t)q.rank;
    const uint64_t u = q.off, v = q.off + (uint64_t)q.n1 * k;
    const bool fwd = q.mode == kDgN;
    const uint32_t in = fwd ? q.n2 : q.n1, on = fwd ? q.n1 : q.n2, ib = fwd ? q.b2 : q.b1;
    const uint64_t Q = fwd ? v : u, P = fwd ? u : v;
    for (uint32_t l0 = 0; l0 < k; l0 += kL) {
      const uint32_t ln = min(kL, k - l0);
      for (uint32_t l = warp; l < ln; l += kW) {
        int m = 0;
#pragma unroll 2
        for (uint32_t i = lane; i < on; i += 32) m = max(m, look(P + (uint64_t)(l0 + l) * on + i));
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) ep[l] = m;
      }
      __syncthreads();
      for (uint32_t j = tid; j < in; j += kWeighThreads) {
        int m = 0;
#pragma unroll 4
        for (uint32_t l = 0; l < ln; ++l) {
          const int e = look(Q + (uint64_t)(l0 + l) * in + j);
          if (e && ep[l]) m = max(m, e + ep[l]);
        }
        if (m) put(ib + j, m - 2046);
      }
      __syncthreads();
    }
  }
  most = __reduce_max_sync(0xffffffffu, most);
  top = __reduce_max_sync(0xffffffffu, top);
  const bool any = __any_sync(0xffffffffu, b);
  if (lane == 0) {
    if (most > __ldcg(&range->wmax)) atomicMax(&range->wmax, most);
    if (top && top - 1023 > __ldcg(&range->emax)) atomicMax(&range->emax, top - 1023);
    if (any) atomicOr(&range->bad, 1);
  }
}

__global__ void dg_drop_kernel(const int* __restrict__ weight, uint32_t n, DgRange* __restrict__ range) {
  const int wmax = range->wmax;
  int drop = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const int w = weight[i];
    if (w != kDgNoWeight) drop = max(drop, wmax - w);
  }
  drop = __reduce_max_sync(0xffffffffu, drop);
  if ((threadIdx.x & 31) == 0 && drop) atomicMax(&range->drop, drop);
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

struct Work {
  size_t sums, xmax, xexp, z, t, end;  // the passes' flags are at 0
};

// n-tiles of 8 columns per pass.  More than two per warp measured slower than
// more passes (64 right-hand sides, 65,536 points: 6.2 ms with four, 5.6 ms with
// two): their sums take the registers of half the warps.
constexpr uint32_t kMaxCols = dg_pass_cols(false);
int nt_of(uint32_t cols) { return cols <= 8 ? 1 : 2; }

Work work_of(bool cplx, uint32_t n, uint32_t t_rows, uint32_t p) {
  const size_t cw = cplx ? 2 : 1, nt = nt_of(p * (uint32_t)cw);
  Work w;
  const size_t per = dg_pass_cols(cplx);
  const size_t passes = ((size_t)p + per - 1) / per;
  w.sums = align256(passes * 4);
  w.xmax = align256(w.sums + passes * sizeof(PassSums));
  w.xexp = align256(w.xmax + (size_t)p * 4);
  w.z = align256(w.xexp + kMaxCols * 4);
  w.t = align256(w.z + ((size_t)n + t_rows) * cw * (S * nt + 1) * 16);
  w.end = align256(w.t + (size_t)t_rows * nt * 64);
  return w;
}

template <int NT, int CW, bool ROWS, bool RS1>
cudaError_t sweep(const KArgs& k, uint32_t n, cudaStream_t s) {
  if (!n) return cudaSuccess;
  auto f = dg_sweep_kernel<NT, CW, ROWS, RS1>;
  constexpr size_t smem = sizeof(Smem<NT, CW>);
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  f<<<n, kThreads, smem, s>>>(k);
  count_product_launches(1);
  return cudaGetLastError();
}

template <int NT, int CW>
cudaError_t run_pass(const DgPlan& pl, const DgArgs& a, const Work& w, uint32_t r0, uint32_t pr, cudaStream_t s) {
  unsigned char* wk = pl.work;
  int* flag = reinterpret_cast<int*>(wk) + r0 / dg_pass_cols(CW == 2);
  int* xmax = reinterpret_cast<int*>(wk + w.xmax) + r0;
  int* xexp = reinterpret_cast<int*>(wk + w.xexp);
  unsigned char* z = wk + w.z;
  double* T = reinterpret_cast<double*>(wk + w.t);
  const uint32_t pc = pr * CW;
  const double* X = static_cast<const double*>(a.X) + (uint64_t)r0 * a.ldX * CW;
  const uint64_t xr = (uint64_t)pl.n * CW, tr = (uint64_t)pl.t_rows * CW;
  PassSums* sums = reinterpret_cast<PassSums*>(wk + w.sums) + r0 / dg_pass_cols(CW == 2);
  dg_xprep_kernel<NT, CW><<<(unsigned)((xr + kXPrepThreads - 1) / kXPrepThreads), kXPrepThreads, 0, s>>>(
      X, a.ldX, pl.n, pc, xmax, pl.weight, xexp, z, sums, flag);
  KArgs k;
  k.arena = pl.arena;
  k.rowptr = pl.rowptr;
  k.pos = pl.pos;
  k.z = z;
  k.xexp = xexp;
  k.flag = flag;
  k.T = T;
  k.Y = static_cast<double*>(a.Y) + (uint64_t)r0 * a.ldY * CW;
  k.ldY = a.ldY;
  k.dre = a.dre;
  k.dim = a.dim;
  k.pc = pc;
  cudaError_t e;
  if (pl.nv) {
    if (pl.t_split && (e = cudaMemsetAsync(T, 0, (size_t)pl.t_split * NT * 64, s)) != cudaSuccess) return e;
    k.pieces = pl.vpieces;
    if ((e = sweep<NT, CW, false, false>(k, pl.nv, s)) != cudaSuccess) return e;
    dg_tprep_kernel<NT, CW><<<(unsigned)((tr * (4 * NT) + 127) / 128), 128, 0, s>>>(T, pl.t_rows, pc,
                                                                            z + xr * (kPR<NT> * 16), flag);
    count_product_launches(1);
  }
  k.pieces = pl.rpieces;
  e = pl.rs1 ? sweep<NT, CW, true, true>(k, pl.nr, s) : sweep<NT, CW, true, false>(k, pl.nr, s);
  if (e != cudaSuccess) return e;
  count_product_launches(1);
  return cudaGetLastError();
}

template <int CW>
cudaError_t run_all(const DgPlan& pl, const DgArgs& a, const Work& w, cudaStream_t s) {
  unsigned char* wk = pl.work;
  cudaError_t e;
  if ((e = cudaMemsetAsync(wk, 0, w.xexp, s)) != cudaSuccess) return e;  // flags, sums, column maxima
  const unsigned gx = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(((uint64_t)pl.n * CW + 1023) / 1024, 64));
  for (uint32_t r0 = 0; r0 < a.p; r0 += 65535) {
    const uint32_t pr = std::min<uint32_t>(a.p - r0, 65535);
    dg_xmax_kernel<CW><<<dim3(gx, pr), 256, 0, s>>>(static_cast<const double*>(a.X), a.ldX, pl.n, r0,
                                                    reinterpret_cast<int*>(wk + w.xmax), reinterpret_cast<int*>(wk));
  }
  count_product_launches(1);
  const uint32_t per = dg_pass_cols(CW == 2);
  for (uint32_t r0 = 0; r0 < a.p; r0 += per) {
    const uint32_t pr = std::min(per, a.p - r0);
    e = nt_of(pr * CW) == 1 ? run_pass<1, CW>(pl, a, w, r0, pr, s) : run_pass<2, CW>(pl, a, w, r0, pr, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

size_t dg_work_bytes(bool cplx, uint32_t n, uint32_t t_rows, uint32_t p) { return work_of(cplx, n, t_rows, p).end; }

cudaError_t launch_matvec_dg(const DgPlan& pl, const DgArgs& a, cudaStream_t s) {
  if (a.p == 0) return cudaSuccess;
  const Work w = work_of(a.cplx, pl.n, pl.t_rows, a.p);
  return a.cplx ? run_all<2>(pl, a, w, s) : run_all<1>(pl, a, w, s);
}

cudaError_t launch_dg_expand(const DgSeg* segs, uint32_t nsegs, DgPos* pos, cudaStream_t s) {
  if (!nsegs) return cudaSuccess;
  dg_expand_kernel<<<(unsigned)(((uint64_t)nsegs * 8 + 255) / 256), 256, 0, s>>>(segs, nsegs, pos);
  return cudaGetLastError();
}

cudaError_t launch_dg_weigh(const DgLeaf* leaves, uint32_t nleaves, bool cplx, const void* arena, int* weight,
                            uint32_t n, DgRange* range, cudaStream_t s) {
  if (!nleaves) return cudaSuccess;
  const uint2* a = static_cast<const uint2*>(arena);
  if (cplx) dg_weigh_kernel<2><<<nleaves, kWeighThreads, 0, s>>>(leaves, a, weight, range);
  else dg_weigh_kernel<1><<<nleaves, kWeighThreads, 0, s>>>(leaves, a, weight, range);
  dg_drop_kernel<<<std::min((n + 255) / 256, 152u), 256, 0, s>>>(weight, n, range);
  return cudaGetLastError();
}

// Two right-hand sides and 10^7 (elements x right-hand sides) on.  Below, the six
// launches of the sliced product (34 us at least) outlast the plain kernel: 1,000
// points (10^6 elements) take 35 us against 20 (p = 2), 38 against 41 (p = 8) and
// 43 against 69 (p = 16).  One right-hand side leaves the FP64 pipe less work per
// byte than the digits take: 0.99 ms against 0.64 ms (65,536 points; p = 2: 0.99
// against 1.11 ms, p = 8: 0.99 against 4.2, p = 16: 1.41 against 8.35).
// AHX_DG_MIN overrides the 10^7 (and lays out at the first product).
bool dg_wanted(uint64_t elems, uint32_t p) {
  const char* e = std::getenv("AHX_DG_MIN");
  const uint64_t least = e && *e ? std::strtoull(e, nullptr, 10) : 10000000ull;
  return p >= 2 && elems * p >= least;
}

// A single product gains less than the layout takes (about 0.3 ms and 55 ns per
// leaf: 1.9 ms in all against 1.1 ms of the plain kernel for 20,011 points and five
// right-hand sides, 25,000 leaves), so a handle that multiplies once stays with the
// plain kernel (2 p FP64 operations per element at 1 TFLOP/s); one that goes on
// never spends more than about twice the better choice.
bool dg_due(DgState& D, uint64_t elems, uint32_t p, size_t nleaves, const char* at_once) {
  if (D.valid || std::getenv(at_once)) return true;
  const double plain = 2e-6 * (double)elems * p, layout = 300.0 + 0.055 * (double)nleaves;
  if (D.spent + plain >= layout) return true;
  D.spent += plain;
  return false;
}

bool stream_captured(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return st != cudaStreamCaptureStatusNone;
}

static int build_state(DgState& D, const std::vector<DgLeaf>& leaves, uint32_t n, const void* arena, bool cplx,
                       int& finite, int device, cudaStream_t s) {
  int rc, sms = 0;
  AHX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  DgHost L;
  D.release();
  ScopedBuf segs, dl;
  if ((rc = upload(dl, leaves, s)) || (rc = D.weight.reserve((size_t)n * sizeof(int) + sizeof(DgRange)))) return rc;
  int* const w = D.weight.as<int>();
  DgRange* const range = reinterpret_cast<DgRange*>(w + n);
  D.range = DgRange{kDgNoWeight, 0, kDgNoWeight, 0};
  AHX_CUDA(cudaMemsetAsync(w, kDgNoWeight & 0xff, (size_t)n * sizeof(int), s));
  AHX_CUDA(cudaMemcpyAsync(range, &D.range, sizeof(DgRange), cudaMemcpyHostToDevice, s));
  AHX_CUDA(launch_dg_weigh(dl.as<DgLeaf>(), (uint32_t)leaves.size(), cplx, arena, w, n, range, s));
  const bool fits = build_dg_layout(leaves, n, (uint32_t)std::max(sms, 1) * 16, cplx ? kDgK / 2 : kDgK, L);
  AHX_CUDA(cudaMemcpyAsync(&D.range, range, sizeof(DgRange), cudaMemcpyDeviceToHost, s));
  AHX_CUDA(cudaStreamSynchronize(s));
  finite = D.range.bad ? 2 : 1;
  if (!fits) {
    D.valid = true;
    return AHX_OK;
  }
  if ((rc = upload(D.vpieces, L.vpieces, s))) return rc;
  if ((rc = upload(D.rpieces, L.rpieces, s))) return rc;
  if ((rc = upload(D.rowptr, L.rowptr, s))) return rc;
  if ((rc = upload(segs, L.segs, s))) return rc;
  if ((rc = D.pos.reserve(std::max<uint64_t>(L.npos, 1) * sizeof(DgPos)))) return rc;
  AHX_CUDA(launch_dg_expand(segs.as<DgSeg>(), (uint32_t)L.segs.size(), D.pos.as<DgPos>(), s));
  AHX_CUDA(cudaStreamSynchronize(s));
  D.nv = (uint32_t)L.vpieces.size();
  D.nr = (uint32_t)L.rpieces.size();
  D.t_rows = L.t_rows;
  D.t_split = L.t_split;
  D.rs1 = L.rs1;
  D.valid = D.usable = true;
  return AHX_OK;
}

int dg_prepare_state(DgState& D, const std::vector<DgLeaf>& leaves, uint32_t n, const void* arena, bool cplx,
                     int& finite, int device, cudaStream_t s) {
  if (D.valid) return AHX_OK;
  int rc;
  try {
    rc = build_state(D, leaves, n, arena, cplx, finite, device, s);
  } catch (const std::bad_alloc&) {
    rc = AHX_ERR_NOMEM;
  }
  if (rc == AHX_ERR_NOMEM) {
    // no room: the plain kernels, which need none, go on (and are counted from zero for the
    // next attempt)
    D.release();
    rc = AHX_OK;
  }
  return rc;
}

DgPlan dg_plan(const DgState& D, uint32_t n, const void* arena, const DevBuf& work) {
  DgPlan p;
  p.vpieces = D.vpieces.as<DgPiece>();
  p.rpieces = D.rpieces.as<DgPiece>();
  p.rowptr = D.rowptr.as<uint64_t>();
  p.pos = D.pos.as<DgPos>();
  p.weight = D.weight.as<int>();
  p.nv = D.nv;
  p.nr = D.nr;
  p.t_rows = D.t_rows;
  p.t_split = D.t_split;
  p.rs1 = D.rs1;
  p.n = n;
  p.arena = arena;
  p.work = static_cast<unsigned char*>(work.p);
  return p;
}

// ---- layout --------------------------------------------------------------

bool build_dg_layout(const std::vector<DgLeaf>& leaves, uint32_t n, uint32_t ctas, uint32_t kmax, DgHost& L) {
  L = DgHost();
  // the side a leaf reads (in) and writes (out), by its mode
  struct Side {
    uint32_t ib, in, ob, on;
    uint64_t q, p;  // factor on the input / output side
  };
  auto side = [](const DgLeaf& l) -> Side {
    const uint64_t u = l.off, v = l.off + (uint64_t)l.n1 * (uint32_t)std::max(l.rank, 0);
    return l.mode == kDgN ? Side{l.b2, l.n2, l.b1, l.n1, v, u} : Side{l.b1, l.n1, l.b2, l.n2, u, v};
  };
  const uint32_t nl = (uint32_t)leaves.size();
  std::vector<Side> sd(nl);
  for (uint32_t l = 0; l < nl; ++l) sd[l] = side(leaves[l]);
  // ---- V sweep: factor columns by column cluster, long clusters first (their
  // tiles are split along K, so their T rows come first).  Clusters are found by
  // their first row (a short list per row: one entry per level), the leaves of a
  // cluster stay in leaf order.
  struct Cluster {
    uint32_t ib, in, rows, next;  // next: the next cluster with this first row + 1
  };
  std::vector<Cluster> cl;
  std::vector<uint32_t> head(n, 0u), of(nl, 0u);
  uint64_t t_rows = 0, vwork = 0;
  for (uint32_t l = 0; l < nl; ++l) {
    if (leaves[l].rank <= 0) continue;
    const Side& q = sd[l];
    uint32_t c = head[q.ib];
    while (c && cl[c - 1].in != q.in) c = cl[c - 1].next;
    if (!c) {
      cl.push_back({q.ib, q.in, 0u, head[q.ib]});
      c = head[q.ib] = (uint32_t)cl.size();
    }
    of[l] = c - 1;
    cl[c - 1].rows += (uint32_t)leaves[l].rank;
    t_rows += (uint32_t)leaves[l].rank;
  }
  if (t_rows + n > 0x3fffffffull) return false;
  std::vector<uint32_t> ord(cl.size()), at(cl.size());
  for (uint32_t c = 0; c < ord.size(); ++c) ord[c] = c;
  std::sort(ord.begin(), ord.end(), [&](uint32_t x, uint32_t y) {
    return cl[x].in != cl[y].in ? cl[x].in > cl[y].in : cl[x].ib < cl[y].ib;
  });
  struct Tile {
    uint32_t row0, nrows, in0, K;
  };
  std::vector<Tile> vt;
  uint32_t t0 = 0;
  for (uint32_t c : ord) {
    at[c] = t0;
    for (uint32_t t = 0; t < cl[c].rows; t += kDgRows) {
      vt.push_back({t0 + t, std::min(kDgRows, cl[c].rows - t), cl[c].ib, cl[c].in});
      vwork += cl[c].in;
    }
    t0 += cl[c].rows;
  }
  std::vector<uint32_t> trow(nl, 0u);
  L.rowptr.resize(t_rows);
  for (uint32_t l = 0; l < nl; ++l) {
    const DgLeaf& q = leaves[l];
    if (q.rank <= 0) continue;
    const uint32_t t = trow[l] = at[of[l]];
    at[of[l]] += (uint32_t)q.rank;
    // U V^H: the input factor is conjugated unless the leaf acts transposed
    const uint64_t cj = q.mode == kDgT ? 0ull : kDgConj;
    for (int32_t k = 0; k < q.rank; ++k) L.rowptr[t + k] = (sd[l].q + (uint64_t)k * sd[l].in) | cj;
  }
  L.t_rows = (uint32_t)t_rows;
  // K range of a piece: enough pieces to fill the GPU several times over, long
  // enough that a piece's start-up and its additions to T or Y stay small
  auto piece_len = [&](uint64_t work) {
    const uint64_t k = work / std::max<uint32_t>(ctas, 1);
    // (the integer sums of a piece have room for 1024 real positions)
    return (uint32_t)std::min<uint64_t>(kmax, std::max<uint64_t>(std::min(256u, kmax), (k + 63) / 64 * 64));
  };
  const uint32_t kv = piece_len(vwork);
  for (const Tile& t : vt) {
    const uint32_t np = (t.K + kv - 1) / kv;
    if (np > 1) L.t_split = t.row0 + t.nrows;
    for (uint32_t p = 0; p < np; ++p) {
      const uint32_t k0 = p * kv;
      L.vpieces.push_back({t.row0, t.nrows, k0, std::min(kv, t.K - k0), t.in0, np > 1 ? 1u : 0u, {0, 0}});
    }
  }
  // ---- rows sweep: the finest row blocks, at most kDgRows rows each
  std::vector<uint32_t> blk(n + 1, 0u);  // first row of a block -> its number
  blk[0] = 1;
  for (uint32_t l = 0; l < nl; ++l)
    if (leaves[l].rank != 0) blk[sd[l].ob] = blk[sd[l].ob + sd[l].on] = 1;
  std::vector<uint32_t> bs;
  for (uint32_t r = 0; r < n;) {
    uint32_t e = r + 1;
    while (e < n && !blk[e]) ++e;
    // parts of whole 16-row fragments (only the last one ragged)
    const uint32_t len = e - r, np = (len + kDgRows - 1) / kDgRows, fr = ((len + 15) / 16 + np - 1) / np * 16;
    blk[r] = (uint32_t)bs.size();
    for (uint32_t q = 0; q < len; q += fr) bs.push_back(r + q);
    r = e;
  }
  const uint32_t nb = (uint32_t)bs.size();
  blk[n] = nb;
  bs.push_back(n);
  // segments and positions per block, by differences over the blocks of each leaf;
  // low-rank leaves first: the dense ones hold a row's largest entries, and what
  // a row has met before them keeps its own, finer scale
  std::vector<uint32_t> seg[2] = {std::vector<uint32_t>(nb + 1, 0u), std::vector<uint32_t>(nb + 1, 0u)};
  std::vector<uint64_t> kat[2] = {std::vector<uint64_t>(nb + 1, 0ull), std::vector<uint64_t>(nb + 1, 0ull)};
  auto kn_of = [](const DgLeaf& q) { return q.rank > 0 ? (uint32_t)q.rank : q.mode == kDgN ? q.n2 : q.n1; };
  for (uint32_t l = 0; l < nl; ++l) {
    const DgLeaf& q = leaves[l];
    if (q.rank == 0) continue;
    const uint32_t d = q.rank < 0, i0 = blk[sd[l].ob], i1 = blk[sd[l].ob + sd[l].on];
    ++seg[d][i0];
    --seg[d][i1];
    kat[d][i0] += kn_of(q);
    kat[d][i1] -= kn_of(q);
  }
  std::vector<uint64_t> bpos(nb + 1, 0ull);
  uint64_t npos = 0, nsegs = 0;
  uint32_t run[2] = {0u, 0u};
  uint64_t krun[2] = {0ull, 0ull};
  for (uint32_t i = 0; i < nb; ++i) {
    bpos[i] = npos;
    for (int d = 0; d < 2; ++d) {
      run[d] += seg[d][i];
      krun[d] += kat[d][i];
      seg[d][i] = (uint32_t)nsegs;
      kat[d][i] = npos;
      nsegs += run[d];
      npos += krun[d];
    }
    if (npos > 0xffffffffull) return false;
  }
  bpos[nb] = npos;
  L.npos = npos;
  L.segs.resize(nsegs);
  for (uint32_t l = 0; l < nl; ++l) {
    const DgLeaf& q = leaves[l];
    if (q.rank == 0) continue;
    const Side& s = sd[l];
    const uint32_t d = q.rank < 0, kn = kn_of(q), i1 = blk[s.ob + s.on];
    DgSeg g{};
    g.kn = kn;
    uint64_t step = 1;  // of base per row
    if (q.rank > 0) {
      // U V^H: only the transposed leaf conj(V) U^T conjugates its output factor
      g.base = s.p;
      g.ldk = s.on;
      g.rsf = 1u | (q.mode == kDgT ? 0x80000000u : 0u);
      g.z = n + trow[l];
    } else if (q.mode == kDgN) {
      g.base = q.off;
      g.ldk = q.n1;
      g.rsf = 1u;
      g.z = q.b2;
    } else {
      L.rs1 = false;
      g.base = q.off;
      g.ldk = 1u;
      g.rsf = q.n1 | (q.mode == kDgH ? 0x80000000u : 0u);
      g.z = q.b1;
      step = q.n1;
    }
    const uint64_t base = g.base;
    for (uint32_t i = blk[s.ob]; i < i1; ++i) {
      g.base = base + (bs[i] - s.ob) * step;
      g.pos0 = (uint32_t)kat[d][i];
      kat[d][i] += kn;
      L.segs[seg[d][i]++] = g;
    }
  }
  const uint32_t kr = piece_len(npos);
  for (uint32_t i = 0; i < nb; ++i)
    for (uint64_t k = bpos[i]; k < bpos[i + 1]; k += kr)
      L.rpieces.push_back({bs[i], bs[i + 1] - bs[i], (uint32_t)k, (uint32_t)std::min<uint64_t>(kr, bpos[i + 1] - k),
                           0u, 0u, {0, 0}});
  return true;
}

}  // namespace ahx

// Test hook (not part of the drop-in interface): Y += op(A) X through the layout
// of the digit-sliced product, evaluated on the host in FP64 piece by piece as the
// sweeps do.  leaves: 6 words per leaf (b1, n1, b2, n2, rank, DgMode), offs:
// element offsets, cplx: complex elements (re, im).  info[4] = {V pieces, rows
// pieces, T rows, rows of the widest tile}.
extern "C" int ahx_dg_host_product(uint32_t n, uint32_t nleaves, const uint32_t* leaves, const uint64_t* offs,
                                   const double* arena, int cplx, uint32_t p, const double* X, double* Y,
                                   uint64_t* info, uint32_t ctas) {
  if (!leaves || !offs || !arena || !X || !Y || !info) return 2;
  std::vector<ahx::DgLeaf> lv(nleaves);
  for (uint32_t l = 0; l < nleaves; ++l) {
    const uint32_t* w = leaves + 6 * (size_t)l;
    lv[l] = ahx::DgLeaf{w[0], w[1], w[2], w[3], (int32_t)w[4], w[5], offs[l]};
  }
  ahx::DgHost L;
  if (!ahx::build_dg_layout(lv, n, ctas, cplx ? ahx::kDgK / 2 : ahx::kDgK, L)) return 1;
  const uint32_t cw = cplx ? 2 : 1;
  // z (re, im) += op(element) * x, op: conjugation
  auto madd = [&](double* z, uint64_t e, bool cj, const double* x) {
    if (!cplx) {
      z[0] += arena[e] * x[0];
      return;
    }
    const double re = arena[2 * e], im = cj ? -arena[2 * e + 1] : arena[2 * e + 1];
    z[0] += re * x[0] - im * x[1];
    z[1] += re * x[1] + im * x[0];
  };
  std::vector<double> T((size_t)L.t_rows * p * cw, 0.0);
  std::vector<ahx::DgPos> pos(L.npos);
  for (const ahx::DgSeg& g : L.segs)
    for (uint32_t k = 0; k < g.kn; ++k) pos[g.pos0 + k] = ahx::DgPos{g.base + (uint64_t)k * g.ldk, g.z + k, g.rsf};
  for (const ahx::DgPiece& q : L.vpieces) {
    if (!q.add && q.row0 < L.t_split) return 3;  // rows that are stored, not added to
    for (uint32_t r = 0; r < q.nrows; ++r) {
      const uint64_t w = L.rowptr[q.row0 + r];
      for (uint32_t k = q.k0; k < q.k0 + q.kn; ++k)
        for (uint32_t j = 0; j < p; ++j)
          madd(&T[((size_t)(q.row0 + r) * p + j) * cw], (w & ~ahx::kDgConj) + k, (w & ahx::kDgConj) != 0,
               X + ((size_t)j * n + q.in0 + k) * cw);
    }
  }
  info[3] = 0;
  for (const ahx::DgPiece& q : L.rpieces) {
    info[3] = std::max<uint64_t>(info[3], q.nrows);
    for (uint32_t k = q.k0; k < q.k0 + q.kn; ++k)
      for (uint32_t r = 0; r < q.nrows; ++r)
        for (uint32_t j = 0; j < p; ++j) {
          const ahx::DgPos& P = pos[k];
          if (L.rs1 && (P.rsf & 0x7fffffffu) != 1) return 4;
          const double* x = P.z < n ? X + ((size_t)j * n + P.z) * cw : &T[((size_t)(P.z - n) * p + j) * cw];
          madd(Y + ((size_t)j * n + q.row0 + r) * cw, P.off + (uint64_t)r * (P.rsf & 0x7fffffffu), (P.rsf >> 31) != 0,
               x);
        }
  }
  info[0] = L.vpieces.size();
  info[1] = L.rpieces.size();
  info[2] = L.t_rows;
  return 0;
}
