// H-matrix product with several right-hand sides on the warp-level tensor
// cores, at the accuracy of the leaves' own storage (ahx_matvec_dg.cu).
//
// GB300 runs one FP64 multiply-add for every 240 of its FP16 tensor products,
// so a product with p right-hand sides that does 2p FP64 operations per 8
// stored bytes is bound by the FP64 pipe from p = 1 on.  Here every stored
// value and every vector entry is cut into digits that FP16 holds exactly, the
// tensor cores multiply digits by digits, and the partial sums that carry the
// leading bits are kept as integers, exactly.
//
//   value = sign * m * 2^e -> fixed point relative to a power of two 2^E
//           (E: the largest exponent its output row has met so far)
//         = 2^E * (d0 2^-8 + d1 2^-17 + d2 2^-26 + d3 2^-35 + d4 2^-45 + d5 2^-55)
//
// with balanced digits (|d0| <= 256, d1..d3 in [-256, 255], d4, d5 in
// [-512, 511]): 57 bits of a double relative to its row's largest term.  The
// digits of the vectors are laid out once per product (the "Z rows": X rows, then
// T = V^T X rows), those of the leaves are cut in registers from the arena
// itself: no second copy of the leaves exists.
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "ahx_matvec.cuh"

namespace ahx {

// How a leaf acts: as stored, transposed, or adjoint (complex; real: transposed)
enum DgMode : uint32_t { kDgN = 0, kDgT = 1, kDgH = 2 };

struct DgLeaf {
  uint32_t b1, n1, b2, n2;
  int32_t rank;
  uint32_t mode;
  uint64_t off;
};

// One K position of the rows sweep: element (row r of its tile) is
// arena[off + r * rs], multiplied with Z row z.  rsf: rs | conjugate << 31.
struct DgPos {
  uint64_t off;
  uint32_t z;
  uint32_t rsf;
};
static_assert(sizeof(DgPos) == 16, "copied 16 bytes at a time");

// kn consecutive positions of one leaf in one row tile: off = base + k * ldk, z + k
struct DgSeg {
  uint64_t base;
  uint32_t ldk, rsf, kn, z, pos0, pad;
};

// One CTA's work: a tile of <= 48 output rows over a range of K.
//   V sweep:    T rows row0 .. (factor columns, see DgHost::rowptr), input rows k0 ..
//   rows sweep: Y rows row0 .., positions k0 .. of the position table
struct DgPiece {
  uint32_t row0, nrows, k0, kn;
  uint32_t in0;  // V sweep: first input (Z) row of the tile's column cluster
  uint32_t add;  // V sweep: 1 when several pieces share the tile (T is added to)
  uint32_t pad[2];
};

constexpr uint32_t kDgK = 1024;
constexpr uint32_t kDgRows = 48;            // rows of a tile
constexpr uint64_t kDgConj = 1ull << 63;    // rowptr flag: conjugated factor column

struct DgHost {
  std::vector<DgPiece> vpieces, rpieces;
  std::vector<uint64_t> rowptr;  // per T row: element offset of its factor column | kDgConj
  std::vector<DgSeg> segs;
  uint32_t t_rows = 0, t_split = 0;  // T rows [0, t_split) are added to by several pieces
  bool rs1 = true;  // every rs is 1
  uint64_t npos = 0;
};

// False when the layout's indices would not fit (the plain kernels take over).
// ctas: how many pieces the sweeps should have at least, where the work allows it;
// kmax: longest K range of a piece (kDgK real positions; half of it for complex leaves).
bool build_dg_layout(const std::vector<DgLeaf>& leaves, uint32_t n, uint32_t ctas, uint32_t kmax, DgHost& L);

struct DgPlan {
  const DgPiece* vpieces;
  const DgPiece* rpieces;
  const uint64_t* rowptr;
  const DgPos* pos;
  uint32_t nv, nr, t_rows, t_split, n;
  bool rs1;
  const int* weight;  // per X row, then their maximum (DgState::weight)
  const void* arena;
  // work buffers of one product (dg_work_bytes)
  unsigned char* work;
};

struct DgArgs {
  bool cplx;  // complex128 leaves and vectors, else double
  double dre, dim;
  uint32_t p;
  const void* X;  // column-major, double (real) or double2
  uint64_t ldX;
  void* Y;
  uint64_t ldY;
};

// Bytes of the work buffer for p right-hand sides.  dg_flags: a word per pass of
// dg_pass_cols right-hand sides, non-zero after a product in which those columns of X (or
// of V^T X) do not fit the digits: an entry is not finite, the largest entry of a row is
// below 2^-200 of its column's largest, a column is subnormal, or one column weighs too
// little against the others (dg_xprep_kernel).  Their columns of Y were then left as they were.
size_t dg_work_bytes(bool cplx, uint32_t n, uint32_t t_rows, uint32_t p);
constexpr uint32_t dg_pass_cols(bool cplx) { return cplx ? 8u : 16u; }
inline const int* dg_flags(const DgPlan& pl) { return reinterpret_cast<const int*>(pl.work); }

cudaError_t launch_dg_expand(const DgSeg* segs, uint32_t nsegs, DgPos* pos, cudaStream_t s);
// Looks at every element of the leaves.  weight[i] (n of them, kDgNoWeight to begin with): the
// binary exponent of the largest entry that meets input row i, of a low-rank leaf P Q^H the
// largest |Q_il| max |P_l|.
constexpr int kDgNoWeight = (int)0x80808080;
struct DgRange {
  int wmax;  // largest weight (kDgNoWeight to begin with)
  int bad;   // an element is not finite, or not zero and outside [2^-500, 2^500] (0)
  int emax;  // largest exponent of an element (kDgNoWeight; 1024: not finite)
  int drop;  // wmax - smallest weight other than kDgNoWeight (0)
};
cudaError_t launch_dg_weigh(const DgLeaf* leaves, uint32_t nleaves, bool cplx, const void* arena, int* weight,
                            uint32_t n, DgRange* range, cudaStream_t s);
cudaError_t launch_matvec_dg(const DgPlan& pl, const DgArgs& a, cudaStream_t s);
// FP64 leaves and one right-hand side over the same layout (ahx_matvec_f1.cu); pl.work:
// dg_work_bytes
cudaError_t launch_matvec_f1(const DgPlan& pl, double d, const double* X, double* Y, cudaStream_t s);
bool f1_wanted(uint64_t elems, bool transposed);
// complex64 leaves over the same layout (ahx_matvec_zt.cu; X, Y complex128): pl.arena the
// complex64 copy, pl.work of zt_work_bytes, control: zt_control_bytes, zero before the first
// product (each leaves its counters zero).  Every kZtPassWords words of it belong to a pass of
// kZtPassCols right-hand sides; the one at kZtFlagAt is as dg_flags (out of the range in which
// split operands are exact to FP32).
constexpr uint32_t kZtPassCols = 16, kZtPassWords = kZtPassCols + 2, kZtFlagAt = kZtPassCols + 1;
size_t zt_control_bytes(uint32_t p);
bool zt_fits(const DgRange& r);  // whether the leaves' elements are in that range
size_t zt_work_bytes(uint32_t n, uint32_t t_rows, uint32_t p);
cudaError_t launch_matvec_zt(const DgPlan& pl, const DgArgs& a, int* control, cudaStream_t s);
bool zt_wanted(uint64_t elems, uint32_t p);

}  // namespace ahx
