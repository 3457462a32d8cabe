// Batched ACA assembly of admissible leaves with SVD recompression, and the
// dense fill of inadmissible leaves (FP64 throughout).
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "ahx_device.cuh"
#include "ahx_tree.hpp"

namespace ahx {

// One admissible leaf to approximate, with the capacity kcap of its cross columns.
struct AcaTask {
  uint32_t b1, n1, b2, n2;
  uint32_t i0, kmax, kcap, leaf;
};

enum AcaStatus : int32_t { kAcaFail = 0, kAcaOk = 1, kAcaOverflow = 2, kAcaNoSpace = 3 };

// ACA of the general assembly (Include/ACA.h:217-350) or ACAr of the symmetric one
// (Include/ACA.h:657-720, Include/apprx.h:86-132)
enum AcaVariant : int32_t { kAcaVariantGeneral = 0, kAcaVariantSym = 1 };

struct AcaResult {
  int32_t status;
  uint32_t k_aca;  // rank returned by ACA (before recompression)
  uint32_t kt;     // rank after recompression
  uint32_t pad;
  uint64_t off;    // element offset of the factors (U, then V) in the arena
};

// Workspace of a leaf (ahx_lowrank.cuh): elements U[n1 kcap] V[n2 kcap], four squares of
// kw x kw, tau[2 kw]; doubles [5 kw]; ints Z[n1] S[n2] (ACA.h:38-42 row/column success
// counters).  kw bounds the crosses of a block: every cross uses up a row (row steps) or
// a column, one more may follow the last row.  64-bit throughout.
__host__ __device__ inline uint32_t aca_work_k(uint32_t n1, uint32_t n2, uint32_t kcap) {
  const uint32_t n = n1 > n2 ? n1 : n2;
  return kcap <= n ? kcap : n + 1u;
}
inline uint64_t aca_ws_bytes(uint32_t n1, uint32_t n2, uint32_t kcap, size_t elem) {
  const uint64_t n = (uint64_t)n1 + n2, kw = aca_work_k(n1, n2, kcap);
  return ((n * kcap + 4ull * kw * kw + 2ull * kw) * elem + 40ull * kw + 4ull * n + 255u) & ~255ull;
}

// Agglomeration's workspace: U[n1 k] V[n2 k] Un[n1 k] Vn[n2 k] R[k k] Vs[k k] sig[k] tau[2 k]
inline uint64_t aca_ws_doubles(uint32_t n1, uint32_t n2, uint32_t kcap) {
  const uint64_t n = (uint64_t)n1 + n2, k = kcap;
  return 2ull * n * k + 2ull * k * k + 3ull * k;
}

// One launch over all leaves: the first nlarge tasks by a CTA each, the rest by a warp
// each, by as many resident teams as there are slots; slots[i]: byte offset of a team's
// workspace (large teams first).
constexpr int kAcaThreads = 128;
struct AcaParams {
  PointsSoA pts;
  double diag;  // Laplace: 1/(4 pi h)
  double k, h;  // Helmholtz
  double eps;
  const AcaTask* tasks;
  AcaResult* res;
  const uint64_t* slots;
  unsigned char* ws;
  void* arena;
  unsigned long long* used;  // arena elements taken
  uint32_t* ctr;             // two task counters
  uint64_t cap;              // arena capacity in elements
  uint32_t nlarge, nsmall, nslot_l, nslot_s;
  int32_t variant;
};

cudaError_t launch_aca(const AcaParams& p, uint32_t grid, cudaStream_t s);   // Laplace (ahx_aca.cu)
cudaError_t launch_zaca(const AcaParams& p, uint32_t grid, cudaStream_t s);  // Helmholtz (ahx_aca_helm.cu)
cudaError_t resident_aca(int device, uint32_t& ctas);
cudaError_t resident_zaca(int device, uint32_t& ctas);

// Dense leaves: fill n1 x n2 column-major blocks of the generator.  The generators are
// symmetric, entry for entry: where the tree also has the block's mirror image, one task
// writes both.
constexpr uint64_t kNoMirror = ~0ull;
struct DenseTask {
  uint32_t b1, n1, b2, n2;
  uint64_t off, mirror;  // element offsets in the arena
};
// The tasks of `leaves` (indices, ascending; off: their offsets), mirror images joined.
std::vector<DenseTask> dense_tasks(const std::vector<Leaf>& Ls, uint32_t n, const std::vector<uint32_t>& leaves,
                                   const std::vector<uint64_t>& off);
cudaError_t launch_dense_fill(const PointsSoA& pts, double diag, const DenseTask* tasks,
                              uint32_t ntasks, double* arena, cudaStream_t s);

// Mirror image of an upper block of a symmetric H-matrix into the same arena:
// rank > 0: U (n1 x rank), V (n2 x rank) at src -> V, U at dst (the leaf V U^T);
// rank < 0: the n1 x n2 block at src -> its transpose (n2 x n1) at dst.
struct MirrorTask {
  uint64_t src, dst;
  uint32_t n1, n2;
  int32_t rank;
  uint32_t pad;
};
cudaError_t launch_mirror(const MirrorTask* tasks, uint32_t ntasks, double* arena, cudaStream_t s);

// Agglomeration: recompression of merged sibling blocks.  Workspace at `ws`
// (doubles, aca_ws_doubles(m, n, k) + merge_qrcp_doubles(k)): U (m x k) and V
// (n x k) hold the gathered factors; Un, Vn receive the result; `zs` (ints):
// m + n + 1 scratch.
inline uint64_t merge_qrcp_doubles(uint32_t k) { return (uint64_t)k * k + 3ull * k; }
struct MergeTask {
  uint32_t m, n, k, pad;
  uint64_t ws, zs;
};
struct MergeParams {
  const MergeTask* tasks;
  uint32_t ntasks;
  double* ws;
  int* zs;
  double eps;
  AcaResult* res;  // k_aca = k, kt = recompressed rank
};
// large: one CTA per task (m or n above 4096), else one warp
cudaError_t launch_merge(const MergeParams& p, bool large, cudaStream_t s);
// Complex unions (ahx_aca_helm.cu): the same tasks and workspace layout in complex
// elements (MergeParams::ws holds them as interleaved doubles), one warp per union.
cudaError_t launch_zmerge(const MergeParams& p, cudaStream_t s);
// dst[s.dst + c * ld_dst + r] = src[s.src + c * nrows + r], r < nrows, c < ncols;
// src == kSegIdentity: ones on the diagonal (r == c) of the zeroed destination,
// at dst[s.dst + c * ld_dst + c * (1 + cplx)] (cplx = 1: the real parts of a
// complex identity stored as interleaved doubles)
constexpr uint64_t kSegIdentity = ~0ull;
struct Seg2D {
  uint64_t src, dst;
  uint32_t nrows, ncols, ld_dst, cplx;
};
cudaError_t launch_copy2d(const Seg2D* segs, uint32_t nsegs, const double* src, double* dst, cudaStream_t s);

// Copy recompressed factors (Un, Vn, kt columns) from the workspace into the arena.
struct CopyTask {
  uint64_t src_u, src_v;  // workspace offsets (doubles)
  uint64_t dst;           // arena offset
  uint32_t n1, n2, kt, pad;
};
cudaError_t launch_copy_factors(const CopyTask* tasks, uint32_t ntasks, const double* ws,
                                double* arena, cudaStream_t s);

}  // namespace ahx
