// Laplace assembly: the ACA launch over admissible leaves (ahx_lowrank.cuh; leaf policy
// Include/apprx.h:136-172), dense and mirrored leaves, the recompression of unions of
// leaves (agglomeration), and the ACA of one block without device allocation.
#include <climits>
#include <mutex>
#include <string>

#include "ahx_aca.cuh"
#include "ahx_hmat.hpp"
#include "ahx_lowrank.cuh"

namespace ahx {
namespace {

constexpr int KSM = 32;        // ranks up to KSM keep the k x k SVD in shared memory
constexpr int LDS = KSM + 1;   // padded row stride of the shared k x k arrays

// per-group shared scratch (doubles)
constexpr int kSmemPerGroup = 2 * KSM * LDS + KSM + 2 * KSM + KSM;

// In-place Householder QR of A (m x k, column-major) by the group; tau[k].
template <int G, class Grp>
__device__ void group_qr(const Grp& g, uint32_t m, uint32_t k, double* A, double* tau) {
  const uint32_t kk = min(m, k);
  for (uint32_t c = 0; c < kk; ++c) {
    double* a = A + (size_t)c * m;
    double xn2 = 0.0, alpha = 0.0;
    for (uint32_t i = g.rank; i < m; i += G) {
      if (i > c) xn2 += a[i] * a[i];
      else if (i == c) alpha = a[i];
    }
    g.sum2(xn2, alpha);
    if (xn2 == 0.0) {
      if (g.rank == 0) tau[c] = 0.0;
      continue;
    }
    const double nrm = sqrt(alpha * alpha + xn2);
    const double beta = alpha >= 0.0 ? -nrm : nrm;
    const double t = (beta - alpha) / beta;
    const double sc = 1.0 / (alpha - beta);
    if (g.rank == 0) tau[c] = t;
    for (uint32_t i = g.rank; i < m; i += G) {
      if (i > c) a[i] *= sc;
      else if (i == c) a[i] = beta;
    }
    for (uint32_t q = c + 1; q < k; ++q) {
      double* b = A + (size_t)q * m;
      double s = 0.0;
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i > c) s += a[i] * b[i];
        else if (i == c) s += b[i];
      }
      s = g.sum(s) * t;
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i > c) b[i] -= s * a[i];
        else if (i == c) b[i] -= s;
      }
    }
  }
}

// C (m x nc, column-major, ldc m) := Q C, Q = H_0 ... H_{kr-1} stored in A/tau.
// Rows of C are owned like rows of A; tau is read from memory written by rank 0
// before a group barrier.
template <int G, class Grp>
__device__ void group_apply_q(const Grp& g, uint32_t m, uint32_t kr, const double* A,
                              const double* tau, uint32_t nc, double* C) {
  for (int c = (int)kr - 1; c >= 0; --c) {
    const double t = tau[c];
    if (t == 0.0) continue;
    const double* a = A + (size_t)c * m;
    for (uint32_t q = 0; q < nc; ++q) {
      double* b = C + (size_t)q * m;
      double s = 0.0;
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i > (uint32_t)c) s += a[i] * b[i];
        else if (i == (uint32_t)c) s += b[i];
      }
      s = g.sum(s) * t;
      for (uint32_t i = g.rank; i < m; i += G) {
        if (i > (uint32_t)c) b[i] -= s * a[i];
        else if (i == (uint32_t)c) b[i] -= s;
      }
    }
  }
}

// One-sided Jacobi on the columns of R (m x n, m, n <= 16) by one warp, in
// tournament order (Brent-Luk round robin): every round rotates n/2 disjoint
// column pairs at once, one group of 4 lanes per pair, each lane holding rows
// sub, sub + 4, sub + 8, sub + 12.  Rotations are accumulated in Vs (n x n).
__device__ void jacobi_warp16(uint32_t m, uint32_t n, double* R, double* Vs, uint32_t ld) {
  const uint32_t lane = threadIdx.x & 31, grp = lane >> 2, sub = lane & 3;
  const uint32_t ne = n + (n & 1);  // a dummy column when n is odd
  for (int sweep = 0; sweep < 40; ++sweep) {
    bool rotated = false;
    for (uint32_t r = 0; r + 1 < ne; ++r) {
      __syncwarp();
      uint32_t a = 0, b = 0;
      bool live = grp < ne / 2;
      if (live) {
        const uint32_t pa = grp, pb = ne - 1 - grp;
        a = pa == 0 ? 0 : 1 + (pa - 1 + r) % (ne - 1);
        b = pb == 0 ? 0 : 1 + (pb - 1 + r) % (ne - 1);
        if (a > b) {
          const uint32_t t = a;
          a = b;
          b = t;
        }
        live = b < n;
      }
      double al = 0.0, be = 0.0, ga = 0.0;
      if (live) {
        for (uint32_t i = sub; i < m; i += 4) {
          const double x = R[i * ld + a], y = R[i * ld + b];
          al = fma(x, x, al);
          be = fma(y, y, be);
          ga = fma(x, y, ga);
        }
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        al += __shfl_xor_sync(0xffffffffu, al, o);
        be += __shfl_xor_sync(0xffffffffu, be, o);
        ga += __shfl_xor_sync(0xffffffffu, ga, o);
      }
      // rotate unless |ga| <= 1e-15 sqrt(al be)  (tested without a square root)
      const bool rot = live && ga != 0.0 && ga * ga > 1e-30 * (al * be);
      if (rot) {
        const double zeta = (be - al) / (2.0 * ga);
        const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0)));
        const double c = rsqrt(fma(t, t, 1.0));
        const double s = c * t;
        for (uint32_t i = sub; i < m; i += 4) {
          const double x = R[i * ld + a], y = R[i * ld + b];
          R[i * ld + a] = c * x - s * y;
          R[i * ld + b] = s * x + c * y;
        }
        for (uint32_t i = sub; i < n; i += 4) {
          const double x = Vs[i * ld + a], y = Vs[i * ld + b];
          Vs[i * ld + a] = c * x - s * y;
          Vs[i * ld + b] = s * x + c * y;
        }
      }
      rotated |= rot;
    }
    if (!__any_sync(0xffffffffu, rotated)) break;
  }
  __syncwarp();
}

// One-sided Jacobi (Hestenes) on the columns of R (mmin x nmin, column-major with
// stride ld), rotations accumulated in Vs: the column pairs of a round-robin
// tournament (circle method) rotate in parallel, one warp per pair, so that a
// whole CTA works on one wide SVD.  Same rotation formulas and stopping rule as
// the serial sweeps; the pair order differs.
__device__ void jacobi_cta(uint32_t mmin, uint32_t nmin, double* R, double* Vs, uint32_t ld) {
  __shared__ int rotated;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const uint32_t np = (nmin + 1) & ~1u;  // players: a dummy one when nmin is odd
  for (int sweep = 0; sweep < 40; ++sweep) {
    __syncthreads();
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (uint32_t r = 0; r + 1 < np; ++r) {
      for (uint32_t k = warp; k < np / 2; k += nw) {
        const uint32_t pa = k, pb = np - 1 - k;
        const uint32_t a = pa == 0 ? 0 : (pa - 1 + r) % (np - 1) + 1;
        const uint32_t b = pb == 0 ? 0 : (pb - 1 + r) % (np - 1) + 1;
        const uint32_t p = min(a, b), q = max(a, b);
        if (q >= nmin) continue;  // the dummy's pair
        double* cp = R + (size_t)p * ld;
        double* cq = R + (size_t)q * ld;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (uint32_t i = lane; i < mmin; i += 32) {
          const double x = cp[i], y = cq[i];
          al += x * x;
          be += y * y;
          ga += x * y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          al += __shfl_xor_sync(0xffffffffu, al, o);
          be += __shfl_xor_sync(0xffffffffu, be, o);
          ga += __shfl_xor_sync(0xffffffffu, ga, o);
        }
        if (ga == 0.0 || fabs(ga) <= 1e-15 * sqrt(al * be)) continue;
        if (lane == 0) rotated = 1;
        const double zeta = (be - al) / (2.0 * ga);
        const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double c = 1.0 / sqrt(1.0 + t * t);
        const double s = c * t;
        for (uint32_t i = lane; i < mmin; i += 32) {
          const double x = cp[i], y = cq[i];
          cp[i] = c * x - s * y;
          cq[i] = s * x + c * y;
        }
        double* vp = Vs + (size_t)p * ld;
        double* vq = Vs + (size_t)q * ld;
        for (uint32_t i = lane; i < nmin; i += 32) {
          const double x = vp[i], y = vq[i];
          vp[i] = c * x - s * y;
          vq[i] = s * x + c * y;
        }
      }
      __syncthreads();
    }
    if (!rotated) break;
  }
  __syncthreads();
}

// addtrll (H/mblock_D.cpp:356-465) for a fresh low-rank block: recompress U V^T
// of rank k to kt <= k columns (relative threshold delta, absolute 1e-64).
// Results in Un (n1 x kt) and Vn (n2 x kt).
template <int G, class Grp>
__device__ uint32_t recompress(const Grp& g, uint32_t n1, uint32_t n2, uint32_t k, double* U,
                               double* V, double* Un, double* Vn, double delta, double* R,
                               double* Vs, uint32_t ld, double* sig, double* tau, int* perm, bool cm = false) {
  if (k == 0) return 0;
  // R and Vs: row-major with a padded stride in shared memory, column-major (the
  // Jacobi sweeps read columns) in the global workspace
  auto ix = [&](uint32_t i, uint32_t j) -> size_t { return cm ? (size_t)j * ld + i : (size_t)i * ld + j; };
  const uint32_t mmin = min(n1, k), nmin = min(n2, k), amin = min(mmin, nmin);
  double* tau1 = tau;
  double* tau2 = tau + k;
  group_qr<G>(g, n1, k, U, tau1);
  group_qr<G>(g, n2, k, V, tau2);
  g.sync();
  // R = R1 R2^T (Include/blas.h:2767-2781), rows owned by i % G
  double fro = 0.0;
  for (uint32_t i = g.rank; i < mmin; i += G) {
    for (uint32_t j = 0; j < nmin; ++j) {
      double d = 0.0;
      for (uint32_t l = max(i, j); l < k; ++l) d += U[i + (size_t)l * n1] * V[j + (size_t)l * n2];
      R[ix(i, j)] = d;
      fro += d * d;
    }
  }
  fro = g.sum(fro);
  const double thresh = delta * sqrt(fro) / (double)sqrtf((float)mmin * (float)nmin);
  for (uint32_t i = g.rank; i < mmin; i += G)
    for (uint32_t j = 0; j < nmin; ++j)
      if (fabs(R[ix(i, j)]) < thresh) R[ix(i, j)] = 0.0;
  for (uint32_t i = g.rank; i < nmin; i += G)
    for (uint32_t j = 0; j < nmin; ++j) Vs[ix(i, j)] = (i == j) ? 1.0 : 0.0;
  // one-sided Jacobi on the columns of R (Hestenes), rotations accumulated in Vs
  if (G == 32 && !cm && mmin <= 16 && nmin <= 16) {
    g.sync();
    jacobi_warp16(mmin, nmin, R, Vs, ld);
  } else if (G > 32 && cm) {
    g.sync();
    jacobi_cta(mmin, nmin, R, Vs, ld);
  } else
  for (int sweep = 0; sweep < 40; ++sweep) {
    bool rotated = false;
    for (uint32_t p = 0; p + 1 < nmin; ++p) {
      for (uint32_t q = p + 1; q < nmin; ++q) {
        double al = 0.0, be = 0.0, ga = 0.0;
        for (uint32_t i = g.rank; i < mmin; i += G) {
          const double x = R[ix(i, p)], y = R[ix(i, q)];
          al += x * x;
          be += y * y;
          ga += x * y;
        }
        g.sum3(al, be, ga);
        if (ga == 0.0 || fabs(ga) <= 1e-15 * sqrt(al * be)) continue;
        rotated = true;
        const double zeta = (be - al) / (2.0 * ga);
        const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double c = 1.0 / sqrt(1.0 + t * t);
        const double s = c * t;
        for (uint32_t i = g.rank; i < mmin; i += G) {
          const double x = R[ix(i, p)], y = R[ix(i, q)];
          R[ix(i, p)] = c * x - s * y;
          R[ix(i, q)] = s * x + c * y;
        }
        for (uint32_t i = g.rank; i < nmin; i += G) {
          const double x = Vs[ix(i, p)], y = Vs[ix(i, q)];
          Vs[ix(i, p)] = c * x - s * y;
          Vs[ix(i, q)] = s * x + c * y;
        }
      }
    }
    if (!rotated) break;
  }
  g.sync();
  for (uint32_t j = 0; j < nmin; ++j) {
    double s = 0.0;
    for (uint32_t i = g.rank; i < mmin; i += G) s += R[ix(i, j)] * R[ix(i, j)];
    s = g.sum(s);
    if (g.rank == 0) sig[j] = sqrt(s);
  }
  g.sync();
  if (g.rank == 0) {
    for (uint32_t j = 0; j < nmin; ++j) perm[j] = (int)j;
    for (uint32_t j = 0; j < nmin; ++j) {
      uint32_t b = j;
      for (uint32_t q = j + 1; q < nmin; ++q)
        if (sig[perm[q]] > sig[perm[b]]) b = q;
      const int t = perm[j];
      perm[j] = perm[b];
      perm[b] = t;
    }
    uint32_t kt = min(amin, k);
    const double s0 = sig[perm[0]];
    while (kt > 0 && (sig[perm[kt - 1]] <= delta * s0 || sig[perm[kt - 1]] < 1e-64)) --kt;
    perm[nmin] = (int)kt;  // the slot after the permutation holds kt
  }
  g.sync();
  const uint32_t kt = (uint32_t)perm[nmin];
  // Un = Q1 [R(:, perm[:kt]); 0],  Vn = Q2 [Vs(:, perm[:kt]); 0]
  for (uint32_t j = 0; j < kt; ++j) {
    const int pj = perm[j];
    for (uint32_t i = g.rank; i < n1; i += G) Un[i + (size_t)j * n1] = i < mmin ? R[ix(i, pj)] : 0.0;
    for (uint32_t i = g.rank; i < n2; i += G) Vn[i + (size_t)j * n2] = i < nmin ? Vs[ix(i, pj)] : 0.0;
  }
  group_apply_q<G>(g, n1, mmin, U, tau1, kt, Un);
  group_apply_q<G>(g, n2, nmin, V, tau2, kt, Vn);
  return kt;
}

// Recompression of a wide union (agglomeration) by a warp or a whole CTA.  The steps of
// recompress up to R = R1 R2^T (QR of both factors, small entries dropped), then
// a column-pivoted Householder QR of R that stops once the trailing columns'
// Frobenius norm is at most 1e-2 delta max_j |R(:, j)| (<= 1e-2 delta sigma_0,
// so no singular value moves by more than that), then one-sided Jacobi on the
// transpose of the kept rows: rr columns instead of nmin, and the pivoted
// triangle converges in fewer sweeps.  R = Qr T P^T, T^T Z = W S gives
// R = (Qr Z) S (P W)^T.  Workspaces (column-major, stride ld): R (mmin x nmin,
// later the reflectors), Tt (nmin x rr), Z (rr x rr); cn, qtau: nmin doubles;
// cperm: nmin ints; perm: rr + 1 ints.
template <int G, class Grp>
__device__ uint32_t recompress_qrcp(const Grp& g, uint32_t n1, uint32_t n2, uint32_t k, double* U, double* V,
                                    double* Un, double* Vn, double delta, double* R, double* Tt, double* Z,
                                    uint32_t ld, double* sig, double* tau, double* cn, double* qtau, int* cperm,
                                    int* perm) {
  if (k == 0) return 0;
  constexpr uint32_t NW = G / 32;
  const uint32_t warp = g.rank >> 5, lane = g.rank & 31;
  const uint32_t mmin = min(n1, k), nmin = min(n2, k), amin = min(mmin, nmin);
  double* tau1 = tau;
  double* tau2 = tau + k;
  group_qr<G>(g, n1, k, U, tau1);
  group_qr<G>(g, n2, k, V, tau2);
  g.sync();
  double fro = 0.0;
  for (uint32_t i = g.rank; i < mmin; i += G) {
    for (uint32_t j = 0; j < nmin; ++j) {
      double d = 0.0;
      for (uint32_t l = max(i, j); l < k; ++l) d += U[i + (size_t)l * n1] * V[j + (size_t)l * n2];
      R[i + (size_t)j * ld] = d;
      fro += d * d;
    }
  }
  fro = g.sum(fro);
  const double thresh = delta * sqrt(fro) / (double)sqrtf((float)mmin * (float)nmin);
  for (uint32_t i = g.rank; i < mmin; i += G)
    for (uint32_t j = 0; j < nmin; ++j)
      if (fabs(R[i + (size_t)j * ld]) < thresh) R[i + (size_t)j * ld] = 0.0;
  g.sync();
  // column norms
  for (uint32_t j = warp; j < nmin; j += NW) {
    double s = 0.0;
    for (uint32_t i = lane; i < mmin; i += 32) {
      const double x = R[i + (size_t)j * ld];
      s += x * x;
    }
    s = Group<32>::sum(s);
    if (lane == 0) {
      cn[j] = s;
      cperm[j] = (int)j;
    }
  }
  g.sync();
  ArgMax cm{0.0, 0xffffffffu, 0.0};
  for (uint32_t j = g.rank; j < nmin; j += G)
    if (gt_nonneg(cn[j], cm.v)) cm = ArgMax{cn[j], j, 0.0};
  cm = g.argmax(cm);
  const double tol2 = (1e-2 * delta) * (1e-2 * delta) * cm.v;
  // column-pivoted QR, stopped at the trailing norm tol
  uint32_t rr = amin;
  for (uint32_t c = 0; c < amin; ++c) {
    double tot = 0.0;
    ArgMax am{0.0, 0xffffffffu, 0.0};
    for (uint32_t j = c + g.rank; j < nmin; j += G) {
      const double v = cn[j];
      tot += v;
      if (gt_nonneg(v, am.v)) am = ArgMax{v, j, 0.0};
    }
    tot = g.sum(tot);
    am = g.argmax(am);
    if (tot <= tol2 || am.idx >= nmin) {
      rr = c;
      break;
    }
    const uint32_t p = am.idx;
    if (p != c) {
      for (uint32_t i = g.rank; i < mmin; i += G) {
        const double x = R[i + (size_t)c * ld];
        R[i + (size_t)c * ld] = R[i + (size_t)p * ld];
        R[i + (size_t)p * ld] = x;
      }
      if (g.rank == 0) {
        const double x = cn[c];
        cn[c] = cn[p];
        cn[p] = x;
        const int q = cperm[c];
        cperm[c] = cperm[p];
        cperm[p] = q;
      }
    }
    g.sync();
    double* a = R + (size_t)c * ld;
    double xn2 = 0.0, alpha = 0.0;
    for (uint32_t i = g.rank; i < mmin; i += G) {
      if (i > c) xn2 += a[i] * a[i];
      else if (i == c) alpha = a[i];
    }
    g.sum2(xn2, alpha);
    double t = 0.0;
    if (xn2 != 0.0) {
      const double nrm = sqrt(alpha * alpha + xn2);
      const double beta = alpha >= 0.0 ? -nrm : nrm;
      t = (beta - alpha) / beta;
      const double sc = 1.0 / (alpha - beta);
      for (uint32_t i = g.rank; i < mmin; i += G) {
        if (i > c) a[i] *= sc;
        else if (i == c) a[i] = beta;
      }
    }
    if (g.rank == 0) qtau[c] = t;
    g.sync();
    // the trailing columns: b -= t v (v^T b), then their norms below row c
    for (uint32_t j = c + 1 + warp; j < nmin; j += NW) {
      double* b = R + (size_t)j * ld;
      if (t != 0.0) {
        double s = 0.0;
        for (uint32_t i = c + lane; i < mmin; i += 32) s += (i == c ? 1.0 : a[i]) * b[i];
        s = Group<32>::sum(s) * t;
        for (uint32_t i = c + lane; i < mmin; i += 32) b[i] -= s * (i == c ? 1.0 : a[i]);
      }
      double s2 = 0.0;
      for (uint32_t i = c + lane; i < mmin; i += 32)
        if (i > c) s2 += b[i] * b[i];
      s2 = Group<32>::sum(s2);
      if (lane == 0) cn[j] = s2;
    }
    g.sync();
  }
  // Tt = T^T (T = the first rr rows of the triangle, pivoted column order), Z = I
  for (uint32_t e = g.rank; e < nmin * rr; e += G) {
    const uint32_t i = e / nmin, j = e - i * nmin;
    Tt[j + (size_t)i * ld] = j >= i ? R[i + (size_t)j * ld] : 0.0;
  }
  for (uint32_t e = g.rank; e < rr * rr; e += G) {
    const uint32_t i = e % rr, j = e / rr;
    Z[i + (size_t)j * ld] = i == j ? 1.0 : 0.0;
  }
  g.sync();
  if (rr > 1) jacobi_cta(nmin, rr, Tt, Z, ld);
  for (uint32_t j = warp; j < rr; j += NW) {
    double s = 0.0;
    for (uint32_t i = lane; i < nmin; i += 32) {
      const double x = Tt[i + (size_t)j * ld];
      s += x * x;
    }
    s = Group<32>::sum(s);
    if (lane == 0) sig[j] = sqrt(s);
  }
  g.sync();
  if (g.rank == 0) {
    for (uint32_t j = 0; j < rr; ++j) perm[j] = (int)j;
    for (uint32_t j = 0; j < rr; ++j) {
      uint32_t b = j;
      for (uint32_t q = j + 1; q < rr; ++q)
        if (sig[perm[q]] > sig[perm[b]]) b = q;
      const int t = perm[j];
      perm[j] = perm[b];
      perm[b] = t;
    }
    uint32_t kt = rr;
    const double s0 = rr ? sig[perm[0]] : 0.0;
    while (kt > 0 && (sig[perm[kt - 1]] <= delta * s0 || sig[perm[kt - 1]] < 1e-64)) --kt;
    perm[rr] = (int)kt;
  }
  g.sync();
  const uint32_t kt = (uint32_t)perm[rr];
  // Un = Q1 [Qr [Z(:, p) s_p; 0]; 0],  Vn = Q2 [P W(:, p); 0]
  for (uint32_t j = 0; j < kt; ++j) {
    const int pj = perm[j];
    const double sj = sig[pj];
    for (uint32_t i = g.rank; i < n1; i += G) Un[i + (size_t)j * n1] = i < rr ? Z[i + (size_t)pj * ld] * sj : 0.0;
    for (uint32_t i = g.rank; i < n2; i += G) {
      if (i < nmin) Vn[(uint32_t)cperm[i] + (size_t)j * n2] = Tt[i + (size_t)pj * ld] / sj;
      else Vn[i + (size_t)j * n2] = 0.0;
    }
  }
  g.sync();
  for (int c = (int)rr - 1; c >= 0; --c) {
    const double t = qtau[c];
    if (t != 0.0) {
      const double* a = R + (size_t)c * ld;
      for (uint32_t j = warp; j < kt; j += NW) {
        double* b = Un + (size_t)j * n1;
        double s = 0.0;
        for (uint32_t i = (uint32_t)c + lane; i < mmin; i += 32) s += (i == (uint32_t)c ? 1.0 : a[i]) * b[i];
        s = Group<32>::sum(s) * t;
        for (uint32_t i = (uint32_t)c + lane; i < mmin; i += 32) b[i] -= s * (i == (uint32_t)c ? 1.0 : a[i]);
      }
    }
    g.sync();
  }
  group_apply_q<G>(g, n1, mmin, U, tau1, kt, Un);
  group_apply_q<G>(g, n2, nmin, V, tau2, kt, Vn);
  return kt;
}

// Agglomeration (H/agglH.cpp:14-107): the concatenated factors of sibling
// low-rank blocks (gathered into the task's workspace, zero elsewhere)
// recompressed to the parent's rank with the relative threshold of
// mblock::unify_cols / unify_rows (H/mblock_D.cpp:662-862).
template <int G, class Grp>
__device__ void merge_task(const Grp& g, const MergeParams& p, uint32_t ti, double* smem) {
  const MergeTask t = p.tasks[ti];
  const uint32_t m = t.m, n = t.n, kc = t.k;
  double* U = p.ws + t.ws;
  double* V = U + (size_t)m * kc;
  double* Un = V + (size_t)n * kc;
  double* Vn = Un + (size_t)m * kc;
  double* Rg = Vn + (size_t)n * kc;
  double* Vsg = Rg + (size_t)kc * kc;
  double* sigg = Vsg + (size_t)kc * kc;
  double* taug = sigg + kc;
  uint32_t kt = 0;
  if (kc > 0) {
    const bool sm = kc <= (uint32_t)KSM;
    double* R = sm ? smem : Rg;
    double* Vs = sm ? smem + KSM * LDS : Vsg;
    double* sig = sm ? smem + 2 * KSM * LDS : sigg;
    double* tau = sm ? smem + 2 * KSM * LDS + KSM : taug;
    int* perm = sm ? reinterpret_cast<int*>(smem + 2 * KSM * LDS + 3 * KSM) : p.zs + t.zs;
    g.sync();
    if (!sm) {
      // k x k beyond shared memory: pivoted QR first; Z, cn, qtau, cperm follow tau
      double* Z = taug + 2 * (size_t)kc;
      double* cn = Z + (size_t)kc * kc;
      double* qtau = cn + kc;
      int* cperm = reinterpret_cast<int*>(qtau + kc);
      kt = recompress_qrcp<G>(g, m, n, kc, U, V, Un, Vn, p.eps, R, Vs, Z, kc, sig, tau, cn, qtau, cperm, perm);
    } else {
      kt = recompress<G>(g, m, n, kc, U, V, Un, Vn, p.eps, R, Vs, sm ? LDS : kc, sig, tau, perm, !sm);
    }
  }
  if (g.rank == 0) p.res[ti] = AcaResult{kAcaOk, kc, kt, 0u};
}

// one warp per CTA: consecutive (similarly costly) unions go to different SMs
__global__ void __launch_bounds__(32) merge_small_kernel(MergeParams p) {
  extern __shared__ double smem_all[];
  const uint32_t task = blockIdx.x;
  if (task >= p.ntasks) return;
  Group<32> g(threadIdx.x & 31);
  merge_task<32>(g, p, task, smem_all);
}

__global__ void copy2d_kernel(const Seg2D* __restrict__ segs, const double* __restrict__ src,
                              double* __restrict__ dst) {
  const Seg2D s = segs[blockIdx.x];
  if (s.src == kSegIdentity) {
    for (uint32_t c = threadIdx.x; c < s.ncols; c += blockDim.x)
      dst[s.dst + (uint64_t)c * s.ld_dst + (uint64_t)c * (1 + s.cplx)] = 1.0;
    return;
  }
  const uint64_t cnt = (uint64_t)s.nrows * s.ncols;
  for (uint64_t e = threadIdx.x; e < cnt; e += blockDim.x) {
    const uint64_t c = e / s.nrows, r = e - c * s.nrows;
    dst[s.dst + c * s.ld_dst + r] = src[s.src + e];
  }
}

constexpr int kLargeThreads = 256;

__global__ void __launch_bounds__(kLargeThreads) merge_large_kernel(MergeParams p) {
  extern __shared__ double smem_all[];
  const uint32_t task = blockIdx.x;
  if (task >= p.ntasks) return;
  Group<kLargeThreads> g(threadIdx.x, smem_all + kSmemPerGroup);
  merge_task<kLargeThreads>(g, p, task, smem_all);
}

__global__ void dense_fill_kernel(PointsSoA P, double diag, const DenseTask* __restrict__ tasks,
                                  double* __restrict__ arena) {
  const DenseTask t = tasks[blockIdx.x];
  double* out = arena + t.off;
  const uint32_t si = blockDim.x % t.n1, sj = blockDim.x / t.n1;
  for (uint32_t i = threadIdx.x % t.n1, j = threadIdx.x / t.n1; j < t.n2;) {
    const uint32_t gj = t.b2 + j;
    const double v = lap_entry(P, gj, t.b1 + i, P.x[gj], P.y[gj], P.z[gj], diag);
    out[(uint64_t)j * t.n1 + i] = v;
    if (t.mirror != kNoMirror) arena[t.mirror + (uint64_t)i * t.n2 + j] = v;
    i += si;
    j += sj;
    if (i >= t.n1) {
      i -= t.n1;
      ++j;
    }
  }
}

// Mirror images of upper blocks: V U^T (the factors swapped) or D^T.
__global__ void mirror_kernel(const MirrorTask* __restrict__ tasks, double* __restrict__ arena) {
  const MirrorTask t = tasks[blockIdx.x];
  const double* src = arena + t.src;
  double* dst = arena + t.dst;
  if (t.rank > 0) {
    const uint64_t nu = (uint64_t)t.n1 * t.rank, nv = (uint64_t)t.n2 * t.rank;
    for (uint64_t e = threadIdx.x; e < nv; e += blockDim.x) dst[e] = src[nu + e];
    for (uint64_t e = threadIdx.x; e < nu; e += blockDim.x) dst[nv + e] = src[e];
  } else {
    const uint64_t cnt = (uint64_t)t.n1 * t.n2;
    for (uint64_t e = threadIdx.x; e < cnt; e += blockDim.x) {
      const uint32_t j = (uint32_t)(e % t.n2), i = (uint32_t)(e / t.n2);  // D^T(j, i) = D(i, j)
      dst[e] = src[i + (uint64_t)j * t.n1];
    }
  }
}

__global__ void copy_factors_kernel(const CopyTask* __restrict__ tasks, const double* __restrict__ ws,
                                    double* __restrict__ arena) {
  const CopyTask t = tasks[blockIdx.x];
  const uint64_t nu = (uint64_t)t.n1 * t.kt, nv = (uint64_t)t.n2 * t.kt;
  double* dst = arena + t.dst;
  for (uint64_t e = threadIdx.x; e < nu; e += blockDim.x) dst[e] = ws[t.src_u + e];
  for (uint64_t e = threadIdx.x; e < nv; e += blockDim.x) dst[nu + e] = ws[t.src_v + e];
}

}  // namespace

cudaError_t launch_aca(const AcaParams& p, uint32_t grid, cudaStream_t s) {
  return lowrank::launch_aca_kernel(lowrank::LapGen{p.pts, p.diag}, p, grid, s);
}
cudaError_t resident_aca(int device, uint32_t& ctas) { return lowrank::resident_aca_kernel<lowrank::LapGen>(device, ctas); }

cudaError_t launch_dense_fill(const PointsSoA& pts, double diag, const DenseTask* tasks,
                              uint32_t ntasks, double* arena, cudaStream_t s) {
  if (ntasks == 0) return cudaSuccess;
  dense_fill_kernel<<<ntasks, 256, 0, s>>>(pts, diag, tasks, arena);
  return cudaGetLastError();
}

cudaError_t launch_merge(const MergeParams& p, bool large, cudaStream_t s) {
  if (p.ntasks == 0) return cudaSuccess;
  if (!large) {
    const size_t smem = sizeof(double) * kSmemPerGroup;
    cudaError_t e = cudaFuncSetAttribute(merge_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    merge_small_kernel<<<p.ntasks, 32, smem, s>>>(p);
  } else {
    const size_t smem = sizeof(double) * (kSmemPerGroup + 3 * (kLargeThreads / 32) + 8);
    cudaError_t e = cudaFuncSetAttribute(merge_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    merge_large_kernel<<<p.ntasks, kLargeThreads, smem, s>>>(p);
  }
  return cudaGetLastError();
}

cudaError_t launch_copy2d(const Seg2D* segs, uint32_t nsegs, const double* src, double* dst, cudaStream_t s) {
  if (nsegs == 0) return cudaSuccess;
  copy2d_kernel<<<nsegs, 256, 0, s>>>(segs, src, dst);
  return cudaGetLastError();
}

cudaError_t launch_mirror(const MirrorTask* tasks, uint32_t ntasks, double* arena, cudaStream_t s) {
  if (ntasks == 0) return cudaSuccess;
  mirror_kernel<<<ntasks, 256, 0, s>>>(tasks, arena);
  return cudaGetLastError();
}

cudaError_t launch_copy_factors(const CopyTask* tasks, uint32_t ntasks, const double* ws,
                                double* arena, cudaStream_t s) {
  if (ntasks == 0) return cudaSuccess;
  copy_factors_kernel<<<ntasks, 256, 0, s>>>(tasks, ws, arena);
  return cudaGetLastError();
}

}  // namespace ahx

// ---------------------------------------------------------------------------
// ACA of one block with no device allocation.
//
// Some callers cannot call cudaMalloc: code that runs while a framework's
// caching allocator has reserved the device memory, latency-critical paths
// where the implicit device synchronisation of cudaMalloc/cudaFree is not
// acceptable, or hosts that own every device allocation themselves and only
// hand out buffers.  For them, ahx_aca_block_noalloc approximates one
// admissible block with the same kernel code as ahx_assemble, taking its
// scratch (the ACA columns, the row/column counters and the recompression
// work arrays) from the file-scope array below instead of an allocation.
//
// The array is 11 MiB and lives on every GPU that loads the library until the
// process exits.  Every call shares it and it keeps the last call's contents;
// the kernel rewrites every word it reads (the counters are set to zero by the
// ACA itself), so nothing carries over between calls.  Calls whose kernels
// overlap on the GPU (on different streams) race on the array: serialise them.

namespace ahx {
namespace {

constexpr size_t kNoAllocScratchBytes = (size_t)8 << 20;
constexpr size_t kNoAllocHeader = 256;

// Blocks are accepted by the size formula of noalloc_bytes, up to 8 MiB.  The workspace
// of a leaf (aca_ws_bytes) can be larger where the rank bound reaches the block's sides:
// with n = n1 + n2 and c columns it is at most n c + 4 min(c, n)^2 + O(n + c) elements,
// and 2 n c + 2 c^2 elements fit 8 MiB: at most 10 MiB, at n = c = 512, and O(n + c)
// (c <= n, or the formula's own 2 c^2 is the larger).
constexpr size_t kNoAllocArrayBytes = (size_t)11 << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocArrayBytes];

// Blocks beyond this many rows or columns, or rank bounds beyond kNoAllocMaxK,
// are refused before any size arithmetic (they could never fit the array).
constexpr uint32_t kNoAllocMaxDim = 1u << 20;
constexpr uint32_t kNoAllocMaxK = 1u << 16;

// bytes of scratch for a block; the ACA columns have the reference's kmax + 1
// capacity (Include/ACA.h:231-232).  64-bit arithmetic throughout.
uint64_t noalloc_bytes(uint32_t n1, uint32_t n2, uint32_t kmax) {
  const uint64_t ws = aca_ws_doubles(n1, n2, kcap_limit(kmax)) * sizeof(double);
  return kNoAllocHeader + ws + ((uint64_t)n1 + n2) * sizeof(int);
}

template <int W>
__global__ void __launch_bounds__(32 * W)
    aca_noalloc_kernel(AcaTask t, PointsSoA P, double diag, double eps, unsigned char* scratch,
                       double* __restrict__ Uout, double* __restrict__ Vout, int32_t* info) {
  extern __shared__ __align__(16) unsigned char smem_na[];
  double* const sm = reinterpret_cast<double*>(smem_na);
  lowrank::Team<W> g(threadIdx.x, reinterpret_cast<double*>(smem_na + lowrank::team_smem<double>()));
  int st;
  uint32_t k, kt;
  lowrank::leaf(g, lowrank::LapGen{P, diag}, t, eps, kAcaVariantGeneral, scratch, sm,
                [&](uint32_t, double*& Un, double*& Vn) {
                  Un = Uout;
                  Vn = Vout;
                  return true;
                },
                st, k, kt);
  if (threadIdx.x == 0) {
    info[0] = st;
    info[1] = (int32_t)k;
    info[2] = (int32_t)kt;
  }
}

// Device address of the scratch array, looked up once per device and context:
// a context torn down and created again (cudaDeviceReset) loads the module
// again, so an address resolved in the old context is not reused.
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[256] = {};
void* g_noalloc_ctx[256] = {};

// the calling thread's current driver context (cuCtxGetCurrent through the
// runtime's entry-point query, so that the library needs no -lcuda)
void* current_context() {
  using Fn = int (*)(void**);
  static Fn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Fn>(f);
  }();
  void* ctx = nullptr;
  if (fn && fn(&ctx) != 0) ctx = nullptr;
  return ctx;
}

}  // namespace
}  // namespace ahx

extern "C" int ahx_aca_block_noalloc(const double* px, const double* py, const double* pz,
                                     uint32_t b1, uint32_t n1, uint32_t b2, uint32_t n2,
                                     uint32_t i0, double h, double eps, uint32_t kmax, double* U,
                                     double* V, int32_t* info, void* stream) {
  using namespace ahx;
  if (!px || !py || !pz || !U || !V || !info || n1 == 0 || n2 == 0 || i0 >= n1 || kmax == 0 ||
      !(h > 0.0) || !(eps > 0.0)) {
    set_error("ahx_aca_block_noalloc: invalid argument");
    return AHX_ERR_ARG;
  }
  if (n1 > kNoAllocMaxDim || n2 > kNoAllocMaxDim || kmax > kNoAllocMaxK) {
    set_error("ahx_aca_block_noalloc: block " + std::to_string(n1) + " x " + std::to_string(n2) +
              " with kmax " + std::to_string(kmax) + " exceeds the fixed scratch array (" +
              std::to_string(kNoAllocScratchBytes) + " bytes)");
    return AHX_ERR_ARG;
  }
  const uint64_t need = noalloc_bytes(n1, n2, kmax);
  if (need > kNoAllocScratchBytes) {
    set_error("ahx_aca_block_noalloc: block " + std::to_string(n1) + " x " + std::to_string(n2) +
              " with kmax " + std::to_string(kmax) + " needs " + std::to_string(need) +
              " bytes of scratch; the fixed scratch array holds " +
              std::to_string(kNoAllocScratchBytes) + " bytes");
    return AHX_ERR_ARG;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= 256) {
    set_error("ahx_aca_block_noalloc: device ordinal out of range");
    return AHX_ERR_ARG;
  }
  void* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    void* ctx = current_context();
    if (!g_noalloc_ptr[dev] || ctx != g_noalloc_ctx[dev]) {
      // first call on this device (or in a new context): resolve the array's
      // device address; the current device is the one the kernel will run on
      void* ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if (e != cudaSuccess) {
        g_noalloc_ptr[dev] = nullptr;
        return cuda_fail(e, "cudaGetSymbolAddress(scratch)");
      }
      g_noalloc_ptr[dev] = ptr;
      g_noalloc_ctx[dev] = current_context();
    }
    scratch = g_noalloc_ptr[dev];
  }
  AcaTask t{};
  t.b1 = b1;
  t.n1 = n1;
  t.b2 = b2;
  t.n2 = n2;
  t.i0 = i0;
  t.kmax = kmax;
  t.kcap = kcap_limit(kmax);  // never overflows: status is 1 or 0
  t.leaf = 0;
  const PointsSoA P{px, py, pz};
  const double diag = 1.0 / (kFourPi * h);
  if (aca_ws_bytes(n1, n2, t.kcap, sizeof(double)) > kNoAllocArrayBytes) {
    set_error("ahx_aca_block_noalloc: workspace beyond the fixed scratch array");
    return AHX_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (std::max(n1, n2) > 256) {
    const size_t smem = lowrank::team_smem<double>() + 64 * sizeof(double);
    aca_noalloc_kernel<4><<<1, 128, smem, s>>>(t, P, diag, eps, (unsigned char*)scratch, U, V, info);
  } else {
    aca_noalloc_kernel<1><<<1, 32, lowrank::team_smem<double>(), s>>>(t, P, diag, eps, (unsigned char*)scratch, U, V,
                                                                      info);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "aca_noalloc_kernel launch");
  return AHX_OK;
}
