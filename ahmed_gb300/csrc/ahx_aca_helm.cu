// Helmholtz single-layer matrix exp(i k r) / (4 pi r) (diagonal exp(i k h) /
// (4 pi h)) on the GPU: the reference's ACA with T = dcomp (Include/ACA.h:46-350;
// complex arithmetic of Include/cmplx.h:80-245: |z| = sqrt(re^2 + im^2), a / z
// = a / |z|^2 * conj(z), scpr = sum conj(x) y), one warp per admissible leaf,
// every leaf with the reference's stopping rule and counters.
//   ahx_helm_aca_ranks: the ACA rank per leaf only (training data and
//     verification of the rank predictor on oscillatory kernels);
//   ahx_helm_assemble: the complex H-matrix (apprx_unsym, Include/apprx.h:136-172,
//     with T = dcomp): ACA, recompression as mblock<dcomp>::addtrll
//     (H/mblock_Z.cpp:200-300), dense leaves where ACA fails or the block is
//     inadmissible; leaves in the mblock<dcomp> layout in a complex arena.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ahx_aca.cuh"
#include "ahx_hmat.hpp"
#include "ahx_lowrank.cuh"

namespace ahx {
namespace {

constexpr int kWarps = 4;  // leaves per CTA

using lowrank::HelmGen;
using lowrank::Team;

__device__ __forceinline__ double cabs2(Cx a) { return __dadd_rn(__dmul_rn(a.re, a.re), __dmul_rn(a.im, a.im)); }
__device__ __forceinline__ double cabs(Cx a) { return __dsqrt_rn(cabs2(a)); }
__device__ __forceinline__ Cx cconj(Cx a) { return Cx{a.re, -a.im}; }

// entry of a dense leaf, r and 1 / (4 pi r) rounded as on the host
__device__ __forceinline__ Cx helm_entry(const PointsSoA& P, double k, double h, uint32_t i, uint32_t j) {
  double r = h, s;
  if (i != j) rounded_r_s(rounded_r2(P.x[i], P.y[i], P.z[i], P.x[j], P.y[j], P.z[j]), r, s);
  else s = __ddiv_rn(1.0, __dmul_rn(kFourPi, r));
  double sn, cs;
  sincos(__dmul_rn(k, r), &sn, &cs);
  return Cx{__dmul_rn(cs, s), __dmul_rn(sn, s)};
}

using G32 = Group<32>;

// ---------------------------------------------------------------------------
// Unions of complex low-rank blocks, by one warp.  The row i of every column belongs
// to lane i % 32.

__device__ __forceinline__ Cx cmul(Cx a, Cx b) { return Cx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
// conj(a) b
__device__ __forceinline__ Cx cmulc(Cx a, Cx b) { return Cx{a.re * b.re + a.im * b.im, a.re * b.im - a.im * b.re}; }
__device__ __forceinline__ Cx cinv(Cx a) {
  const double s = 1.0 / (a.re * a.re + a.im * a.im);
  return Cx{a.re * s, -a.im * s};
}

// Householder QR of A (m x k, column-major) in LAPACK's zgeqrf form:
// H_c = I - tau_c v_c v_c^H with v_c(c) = 1, a real diagonal beta in R.
__device__ void zqr(const G32& g, uint32_t m, uint32_t k, Cx* A, Cx* tau) {
  const uint32_t kk = min(m, k);
  for (uint32_t c = 0; c < kk; ++c) {
    Cx* a = A + (size_t)c * m;
    double xn2 = 0.0, ar = 0.0, ai = 0.0;
    for (uint32_t i = g.rank; i < m; i += 32) {
      const Cx v = a[i];
      if (i > c) xn2 += v.re * v.re + v.im * v.im;
      else if (i == c) {
        ar = v.re;
        ai = v.im;
      }
    }
    G32::sum3(xn2, ar, ai);
    if (xn2 == 0.0 && ai == 0.0) {
      if (g.rank == 0) tau[c] = Cx{0.0, 0.0};
      continue;
    }
    const double nrm = sqrt(ar * ar + ai * ai + xn2);
    const double beta = ar >= 0.0 ? -nrm : nrm;
    const Cx t{(beta - ar) / beta, -ai / beta};
    const Cx sc = cinv(Cx{ar - beta, ai});
    if (g.rank == 0) tau[c] = t;
    for (uint32_t i = g.rank; i < m; i += 32) {
      if (i > c) a[i] = cmul(a[i], sc);
      else if (i == c) a[i] = Cx{beta, 0.0};
    }
    // the remaining columns: b -= conj(tau) v (v^H b)
    const Cx tc = cconj(t);
    for (uint32_t q = c + 1; q < k; ++q) {
      Cx* b = A + (size_t)q * m;
      double sr = 0.0, si = 0.0;
      for (uint32_t i = g.rank; i < m; i += 32) {
        if (i > c) {
          const Cx z = cmulc(a[i], b[i]);
          sr += z.re;
          si += z.im;
        } else if (i == c) {
          sr += b[i].re;
          si += b[i].im;
        }
      }
      G32::sum2(sr, si);
      const Cx f = cmul(tc, Cx{sr, si});
      for (uint32_t i = g.rank; i < m; i += 32) {
        if (i > c) {
          const Cx z = cmul(f, a[i]);
          b[i].re -= z.re;
          b[i].im -= z.im;
        } else if (i == c) {
          b[i].re -= f.re;
          b[i].im -= f.im;
        }
      }
    }
  }
}

// C (m x nc, ld m) := Q C with Q = H_0 ... H_{kr-1} from zqr (tau read after a
// warp barrier).
__device__ void zapply_q(const G32& g, uint32_t m, uint32_t kr, const Cx* A, const Cx* tau, uint32_t nc, Cx* C) {
  for (int c = (int)kr - 1; c >= 0; --c) {
    const Cx t = tau[c];
    if (t.re == 0.0 && t.im == 0.0) continue;
    const Cx* a = A + (size_t)c * m;
    for (uint32_t q = 0; q < nc; ++q) {
      Cx* b = C + (size_t)q * m;
      double sr = 0.0, si = 0.0;
      for (uint32_t i = g.rank; i < m; i += 32) {
        if (i > (uint32_t)c) {
          const Cx z = cmulc(a[i], b[i]);
          sr += z.re;
          si += z.im;
        } else if (i == (uint32_t)c) {
          sr += b[i].re;
          si += b[i].im;
        }
      }
      G32::sum2(sr, si);
      const Cx f = cmul(t, Cx{sr, si});
      for (uint32_t i = g.rank; i < m; i += 32) {
        if (i > (uint32_t)c) {
          const Cx z = cmul(f, a[i]);
          b[i].re -= z.re;
          b[i].im -= z.im;
        } else if (i == (uint32_t)c) {
          b[i].re -= f.re;
          b[i].im -= f.im;
        }
      }
    }
  }
}

// Recompression of a union of complex low-rank blocks (agglomeration of mblock<dcomp>
// leaves, H/agglH.cpp:14-107 with T = dcomp) by one warp: QR of both factors,
// R = R1 R2^H, small entries dropped as in addtrll, then a column-pivoted
// Householder QR of R stopped once the trailing columns' Frobenius norm is at most
// 1e-2 delta max_j |R(:, j)|, one-sided Jacobi on Tt = T^H of the kept rows T
// (T^H Z = W S), and R = (Qr Z S) (P W)^H.  Workspaces as the real union's
// (complex elements): R (mmin x nmin, stride ld, then the reflectors), Tt
// (nmin x rr), Z (rr x rr); cn: nmin doubles; qtau: nmin; cperm: nmin ints;
// perm: rr + 1 ints.
__device__ uint32_t zrecompress_qrcp(const G32& g, uint32_t n1, uint32_t n2, uint32_t k, Cx* U, Cx* V, Cx* Un,
                                     Cx* Vn, double delta, Cx* R, Cx* Tt, Cx* Z, uint32_t ld, double* sig, Cx* tau,
                                     double* cn, Cx* qtau, int* cperm, int* perm) {
  if (k == 0) return 0;
  const uint32_t lane = g.rank;
  const uint32_t mmin = min(n1, k), nmin = min(n2, k), amin = min(mmin, nmin);
  Cx* tau1 = tau;
  Cx* tau2 = tau + k;
  zqr(g, n1, k, U, tau1);
  zqr(g, n2, k, V, tau2);
  __syncwarp();
  double fro = 0.0;
  for (uint32_t i = lane; i < mmin; i += 32) {
    for (uint32_t j = 0; j < nmin; ++j) {
      double dr = 0.0, di = 0.0;
      for (uint32_t l = max(i, j); l < k; ++l) {
        const Cx u = U[i + (size_t)l * n1], v = V[j + (size_t)l * n2];
        dr += u.re * v.re + u.im * v.im;
        di += u.im * v.re - u.re * v.im;
      }
      R[i + (size_t)j * ld] = Cx{dr, di};
      fro += dr * dr + di * di;
    }
  }
  fro = G32::sum(fro);
  const double thresh = delta * sqrt(fro) / (double)sqrtf((float)mmin * (float)nmin);
  for (uint32_t i = lane; i < mmin; i += 32)
    for (uint32_t j = 0; j < nmin; ++j)
      if (cabs(R[i + (size_t)j * ld]) < thresh) R[i + (size_t)j * ld] = Cx{0.0, 0.0};
  __syncwarp();
  ArgMax cm{0.0, 0xffffffffu, 0.0};
  for (uint32_t j = 0; j < nmin; ++j) {
    double sj = 0.0;
    for (uint32_t i = lane; i < mmin; i += 32) sj += cabs2(R[i + (size_t)j * ld]);
    sj = G32::sum(sj);
    if (lane == 0) {
      cn[j] = sj;
      cperm[j] = (int)j;
    }
    if (gt_nonneg(sj, cm.v)) cm = ArgMax{sj, j, 0.0};
  }
  __syncwarp();
  const double tol2 = (1e-2 * delta) * (1e-2 * delta) * cm.v;
  uint32_t rr = amin;
  for (uint32_t c = 0; c < amin; ++c) {
    double tot = 0.0;
    ArgMax am{0.0, 0xffffffffu, 0.0};
    for (uint32_t j = c + lane; j < nmin; j += 32) {
      const double v = cn[j];
      tot += v;
      if (gt_nonneg(v, am.v)) am = ArgMax{v, j, 0.0};
    }
    tot = G32::sum(tot);
    am = G32::argmax(am);
    if (tot <= tol2 || am.idx >= nmin) {
      rr = c;
      break;
    }
    const uint32_t p = am.idx;
    __syncwarp();
    if (p != c) {
      for (uint32_t i = lane; i < mmin; i += 32) {
        const Cx x = R[i + (size_t)c * ld];
        R[i + (size_t)c * ld] = R[i + (size_t)p * ld];
        R[i + (size_t)p * ld] = x;
      }
      if (lane == 0) {
        const double x = cn[c];
        cn[c] = cn[p];
        cn[p] = x;
        const int q = cperm[c];
        cperm[c] = cperm[p];
        cperm[p] = q;
      }
    }
    __syncwarp();
    Cx* a = R + (size_t)c * ld;
    double xn2 = 0.0, ar = 0.0, ai = 0.0;
    for (uint32_t i = lane; i < mmin; i += 32) {
      const Cx v = a[i];
      if (i > c) xn2 += v.re * v.re + v.im * v.im;
      else if (i == c) {
        ar = v.re;
        ai = v.im;
      }
    }
    G32::sum3(xn2, ar, ai);
    Cx t{0.0, 0.0};
    if (!(xn2 == 0.0 && ai == 0.0)) {
      const double nrm = sqrt(ar * ar + ai * ai + xn2);
      const double beta = ar >= 0.0 ? -nrm : nrm;
      t = Cx{(beta - ar) / beta, -ai / beta};
      const Cx sc = cinv(Cx{ar - beta, ai});
      for (uint32_t i = lane; i < mmin; i += 32) {
        if (i > c) a[i] = cmul(a[i], sc);
        else if (i == c) a[i] = Cx{beta, 0.0};
      }
    }
    if (lane == 0) qtau[c] = t;
    __syncwarp();
    // trailing columns: b -= conj(t) v (v^H b), then their norms below row c
    const Cx tc = cconj(t);
    for (uint32_t j = c + 1; j < nmin; ++j) {
      Cx* b = R + (size_t)j * ld;
      if (t.re != 0.0 || t.im != 0.0) {
        double sr = 0.0, si = 0.0;
        for (uint32_t i = c + lane; i < mmin; i += 32) {
          if (i > c) {
            const Cx z = cmulc(a[i], b[i]);
            sr += z.re;
            si += z.im;
          } else {
            sr += b[i].re;
            si += b[i].im;
          }
        }
        G32::sum2(sr, si);
        const Cx f = cmul(tc, Cx{sr, si});
        for (uint32_t i = c + lane; i < mmin; i += 32) {
          if (i > c) {
            const Cx z = cmul(f, a[i]);
            b[i].re -= z.re;
            b[i].im -= z.im;
          } else {
            b[i].re -= f.re;
            b[i].im -= f.im;
          }
        }
      }
      double s2 = 0.0;
      for (uint32_t i = c + lane; i < mmin; i += 32)
        if (i > c) s2 += cabs2(b[i]);
      s2 = G32::sum(s2);
      if (lane == 0) cn[j] = s2;
    }
    __syncwarp();
  }
  // Tt = T^H (nmin x rr), Z = I (rr x rr)
  for (uint32_t e = lane; e < nmin * rr; e += 32) {
    const uint32_t i = e / nmin, j = e - i * nmin;
    Tt[j + (size_t)i * ld] = j >= i ? cconj(R[i + (size_t)j * ld]) : Cx{0.0, 0.0};
  }
  for (uint32_t e = lane; e < rr * rr; e += 32) {
    const uint32_t i = e % rr, j = e / rr;
    Z[i + (size_t)j * ld] = Cx{i == j ? 1.0 : 0.0, 0.0};
  }
  __syncwarp();
  // one-sided Jacobi on the columns of Tt (the rotations of zrecompress)
  for (int sweep = 0; sweep < 40; ++sweep) {
    bool rotated = false;
    for (uint32_t p = 0; p + 1 < rr; ++p) {
      for (uint32_t q = p + 1; q < rr; ++q) {
        double al = 0.0, be = 0.0, gr = 0.0, gi = 0.0;
        for (uint32_t i = lane; i < nmin; i += 32) {
          const Cx x = Tt[i + (size_t)p * ld], y = Tt[i + (size_t)q * ld];
          al += x.re * x.re + x.im * x.im;
          be += y.re * y.re + y.im * y.im;
          const Cx z = cmulc(x, y);
          gr += z.re;
          gi += z.im;
        }
        G32::sum2(al, be);
        G32::sum2(gr, gi);
        const double ga = sqrt(gr * gr + gi * gi);
        if (ga == 0.0 || ga <= 1e-15 * sqrt(al * be)) continue;
        rotated = true;
        const double zeta = (be - al) / (2.0 * ga);
        const double tt = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double cs = 1.0 / sqrt(1.0 + tt * tt);
        const double sn = cs * tt;
        const Cx e{gr / ga, -gi / ga};
        for (uint32_t i = lane; i < nmin; i += 32) {
          const Cx x = Tt[i + (size_t)p * ld], ey = cmul(e, Tt[i + (size_t)q * ld]);
          Tt[i + (size_t)p * ld] = Cx{cs * x.re - sn * ey.re, cs * x.im - sn * ey.im};
          Tt[i + (size_t)q * ld] = Cx{sn * x.re + cs * ey.re, sn * x.im + cs * ey.im};
        }
        for (uint32_t i = lane; i < rr; i += 32) {
          const Cx x = Z[i + (size_t)p * ld], ey = cmul(e, Z[i + (size_t)q * ld]);
          Z[i + (size_t)p * ld] = Cx{cs * x.re - sn * ey.re, cs * x.im - sn * ey.im};
          Z[i + (size_t)q * ld] = Cx{sn * x.re + cs * ey.re, sn * x.im + cs * ey.im};
        }
      }
    }
    if (!rotated) break;
  }
  for (uint32_t j = 0; j < rr; ++j) {
    double sj = 0.0;
    for (uint32_t i = lane; i < nmin; i += 32) sj += cabs2(Tt[i + (size_t)j * ld]);
    sj = G32::sum(sj);
    if (lane == 0) sig[j] = sqrt(sj);
  }
  __syncwarp();
  if (lane == 0) {
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
  __syncwarp();
  const uint32_t kt = (uint32_t)perm[rr];
  // Un = Q1 [Qr [Z(:, p) s_p; 0]; 0],  Vn = Q2 [P W(:, p); 0]
  for (uint32_t j = 0; j < kt; ++j) {
    const int pj = perm[j];
    const double sj = sig[pj];
    for (uint32_t i = lane; i < n1; i += 32) {
      const Cx z = i < rr ? Z[i + (size_t)pj * ld] : Cx{0.0, 0.0};
      Un[i + (size_t)j * n1] = Cx{z.re * sj, z.im * sj};
    }
    for (uint32_t i = lane; i < n2; i += 32) {
      if (i < nmin) {
        const Cx w = Tt[i + (size_t)pj * ld];
        Vn[(uint32_t)cperm[i] + (size_t)j * n2] = Cx{w.re / sj, w.im / sj};
      } else {
        Vn[i + (size_t)j * n2] = Cx{0.0, 0.0};
      }
    }
  }
  __syncwarp();
  for (int c = (int)rr - 1; c >= 0; --c) {
    const Cx t = qtau[c];
    if (t.re != 0.0 || t.im != 0.0) {
      const Cx* a = R + (size_t)c * ld;
      for (uint32_t j = 0; j < kt; ++j) {
        Cx* b = Un + (size_t)j * n1;
        double sr = 0.0, si = 0.0;
        for (uint32_t i = (uint32_t)c + lane; i < mmin; i += 32) {
          if (i > (uint32_t)c) {
            const Cx z = cmulc(a[i], b[i]);
            sr += z.re;
            si += z.im;
          } else {
            sr += b[i].re;
            si += b[i].im;
          }
        }
        G32::sum2(sr, si);
        const Cx f = cmul(t, Cx{sr, si});
        for (uint32_t i = (uint32_t)c + lane; i < mmin; i += 32) {
          if (i > (uint32_t)c) {
            const Cx z = cmul(f, a[i]);
            b[i].re -= z.re;
            b[i].im -= z.im;
          } else {
            b[i].re -= f.re;
            b[i].im -= f.im;
          }
        }
      }
    }
    __syncwarp();
  }
  zapply_q(g, n1, mmin, U, tau1, kt, Un);
  zapply_q(g, n2, nmin, V, tau2, kt, Vn);
  __syncwarp();
  return kt;
}

// one warp per union (CTA of one warp: consecutive unions on different SMs)
__global__ void __launch_bounds__(32) zmerge_kernel(MergeParams p) {
  const uint32_t ti = blockIdx.x;
  if (ti >= p.ntasks) return;
  G32 g(threadIdx.x & 31);
  const MergeTask t = p.tasks[ti];
  const uint32_t m = t.m, n = t.n, kc = t.k;
  Cx* U = reinterpret_cast<Cx*>(p.ws) + t.ws;
  Cx* V = U + (size_t)m * kc;
  Cx* Un = V + (size_t)n * kc;
  Cx* Vn = Un + (size_t)m * kc;
  Cx* R = Vn + (size_t)n * kc;
  Cx* Tt = R + (size_t)kc * kc;
  double* sig = reinterpret_cast<double*>(Tt + (size_t)kc * kc);
  Cx* tau = Tt + (size_t)kc * kc + kc;
  Cx* Z = tau + 2 * (size_t)kc;
  double* cn = reinterpret_cast<double*>(Z + (size_t)kc * kc);
  Cx* qtau = Z + (size_t)kc * kc + kc;
  int* cperm = reinterpret_cast<int*>(qtau + kc);
  uint32_t kt = 0;
  if (kc > 0) kt = zrecompress_qrcp(g, m, n, kc, U, V, Un, Vn, p.eps, R, Tt, Z, kc, sig, tau, cn, qtau, cperm,
                                    p.zs + t.zs);
  if (g.rank == 0) p.res[ti] = AcaResult{kAcaOk, kc, kt, 0u};
}

__global__ void helm_dense_kernel(PointsSoA P, double k, double h, const DenseTask* __restrict__ tasks,
                                  Cx* __restrict__ arena) {
  const DenseTask t = tasks[blockIdx.x];
  Cx* out = arena + t.off;
  const uint32_t si = blockDim.x % t.n1, sj = blockDim.x / t.n1;
  for (uint32_t i = threadIdx.x % t.n1, j = threadIdx.x / t.n1; j < t.n2;) {
    const Cx v = helm_entry(P, k, h, t.b1 + i, t.b2 + j);
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

struct HTask {
  uint32_t b1, n1, b2, n2, kmax, kcap, leaf, pad;
  uint64_t ws;  // Cx offset of U (then V) in the batch workspace
  uint64_t zs;  // int offset of Z (then S)
};

__global__ void __launch_bounds__(32 * kWarps)
    helm_aca_kernel(PointsSoA P, double k, double h, double eps, const HTask* __restrict__ tasks, uint32_t n,
                    Cx* __restrict__ ws, int* __restrict__ zs, int2* __restrict__ res) {
  const uint32_t t = blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (t >= n) return;
  const HTask T = tasks[t];
  Team<1> g(threadIdx.x & 31, nullptr);
  lowrank::Blk<HelmGen> B;
  B.gen = HelmGen{P, k, h};
  B.b1 = T.b1;
  B.n1 = T.n1;
  B.b2 = T.b2;
  B.n2 = T.n2;
  B.U = ws + T.ws;
  B.V = B.U + (size_t)T.n1 * T.kcap;
  B.Z = zs + T.zs;
  B.S = B.Z + T.n1;
  B.P = nullptr;  // the ranks alone: no recompression
  B.d2 = nullptr;
  B.ld = 0;
  uint32_t kk = 0;
  const int st = lowrank::aca(g, B, 0u, T.kmax, T.kcap, eps, kk);
  if (g.rank == 0) res[t] = make_int2(st, (int)kk);
}

}  // namespace
}  // namespace ahx

using namespace ahx;

extern "C" int ahx_helm_aca_ranks(ahx_hmat* H, double wavenumber, double h, double eps, uint32_t rankmax,
                                  const float* rank_hint, int32_t* ranks) {
  if (!H || !ranks || !(h > 0.0) || !(eps > 0.0) || H->tree.kind != kTreeBbx) {
    set_error("ahx_helm_aca_ranks: invalid argument (bounding-box trees only)");
    return AHX_ERR_ARG;
  }
  const HandleLock lk(H->mu);
  int rc = ensure_device(H);
  if (rc) return rc;
  const auto& Ls = H->tree.leaves;
  const uint32_t nl = (uint32_t)Ls.size();
  std::vector<HTask> tasks;
  for (uint32_t l = 0; l < nl; ++l) {
    const Leaf& L = Ls[l];
    ranks[l] = -1;
    const uint32_t maxk = maxk_of(L.n1, L.n2, rankmax);
    if (!L.adm || !maxk) continue;
    HTask t{};
    t.b1 = L.b1;
    t.n1 = L.n1;
    t.b2 = L.b2;
    t.n2 = L.n2;
    t.kmax = maxk;
    t.kcap = std::min(kcap_limit(maxk), aca_kcap_default());
    if (rank_hint && rank_hint[l] >= 0.f)
      t.kcap = std::min(kcap_limit(maxk), std::max(8u, (uint32_t)std::ceil(rank_hint[l] * 1.25f + 4.f)));
    t.leaf = l;
    tasks.push_back(t);
  }
  H->stat_ws_bytes = H->stat_retries = H->stat_batches = 0;
  const size_t budget = aca_ws_budget();
  const double* pts = H->pts.as<double>();
  const PointsSoA P{pts, pts + H->tree.n, pts + 2 * (size_t)H->tree.n};
  DevBuf ws, zs, dtasks, dres;
  while (!tasks.empty()) {
    std::sort(tasks.begin(), tasks.end(), [](const HTask& a, const HTask& b) {
      return (uint64_t)(a.n1 + a.n2) * a.kcap > (uint64_t)(b.n1 + b.n2) * b.kcap;
    });
    std::vector<HTask> retry;
    size_t i = 0;
    while (i < tasks.size()) {
      uint64_t wsc = 0, zsi = 0;
      size_t j = i;
      for (; j < tasks.size(); ++j) {
        const uint64_t w = (uint64_t)(tasks[j].n1 + tasks[j].n2) * tasks[j].kcap;
        if (j > i && (wsc + w) * sizeof(Cx) + (zsi + tasks[j].n1 + tasks[j].n2) * 4 > budget) break;
        tasks[j].ws = wsc;
        tasks[j].zs = zsi;
        wsc += w;
        zsi += tasks[j].n1 + tasks[j].n2;
      }
      std::vector<HTask> batch(tasks.begin() + i, tasks.begin() + j);
      i = j;
      H->stat_ws_bytes = std::max<uint64_t>(H->stat_ws_bytes, wsc * sizeof(Cx) + zsi * 4);
      H->stat_batches++;
      if ((rc = ws.reserve(std::max<uint64_t>(wsc, 1) * sizeof(Cx)))) return rc;
      if ((rc = zs.reserve(std::max<uint64_t>(zsi, 1) * 4))) return rc;
      if ((rc = upload(dtasks, batch, H->stream))) return rc;
      if ((rc = dres.reserve(batch.size() * sizeof(int2)))) return rc;
      const uint32_t nb = (uint32_t)batch.size();
      helm_aca_kernel<<<(nb + kWarps - 1) / kWarps, 32 * kWarps, 0, H->stream>>>(
          P, wavenumber, h, eps, dtasks.as<HTask>(), nb, ws.as<Cx>(), zs.as<int>(), dres.as<int2>());
      AHX_CUDA(cudaGetLastError());
      std::vector<int2> res(nb);
      AHX_CUDA(cudaMemcpyAsync(res.data(), dres.p, nb * sizeof(int2), cudaMemcpyDeviceToHost, H->stream));
      AHX_CUDA(cudaStreamSynchronize(H->stream));
      for (uint32_t q = 0; q < nb; ++q) {
        const HTask& t = batch[q];
        if (res[q].x == kAcaOverflow && t.kcap < kcap_limit(t.kmax)) {
          HTask u = t;
          u.kcap = std::min(kcap_limit(t.kmax), std::max(t.kcap * 4, 16u));
          retry.push_back(u);
          H->stat_retries++;
        } else {
          ranks[t.leaf] = res[q].x == kAcaOk ? res[q].y : -2;
        }
      }
    }
    tasks.swap(retry);
  }
  return AHX_OK;
}

namespace ahx {

// Append-only growable complex arena of the Helmholtz leaves.
int zarena_append(ahx_hmat* H, uint64_t count, uint64_t& off) {
  ZState& Z = H->z;
  const uint64_t need = (Z.elems + count) * sizeof(Cx);
  if (need > Z.arena.bytes) {
    size_t nb = std::max<size_t>(need, Z.arena.bytes * 2);
    void* np = nullptr;
    cudaError_t e = cudaMalloc(&np, nb);
    if (e != cudaSuccess) {
      cudaGetLastError();
      nb = need;
      e = cudaMalloc(&np, nb);
      if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("device allocation of the complex leaf arena failed");
        return AHX_ERR_NOMEM;
      }
    }
    if (Z.elems) {
      const cudaError_t ce = cudaMemcpyAsync(np, Z.arena.p, Z.elems * sizeof(Cx), cudaMemcpyDeviceToDevice, H->stream);
      if (ce != cudaSuccess) {
        cudaFree(np);
        return cuda_fail(ce, "cudaMemcpyAsync (complex arena)");
      }
    }
    AHX_CUDA(cudaStreamSynchronize(H->stream));
    if (Z.arena.p) cudaFree(Z.arena.p);
    Z.arena.p = np;
    Z.arena.bytes = nb;
  }
  off = Z.elems;
  Z.elems += count;
  return AHX_OK;
}

}  // namespace ahx

extern "C" int ahx_helm_assemble(ahx_hmat* H, double wavenumber, double h, double eps, uint32_t rankmax) {
  if (!H || !(h > 0.0) || !(eps > 0.0) || !std::isfinite(wavenumber)) {
    set_error("ahx_helm_assemble: invalid argument");
    return AHX_ERR_ARG;
  }
  const HandleLock lk(H->mu);
  int rc = ensure_device(H);
  if (rc) return rc;
  ZState& Z = H->z;
  Z.assembled = false;
  Z.drop_table();
  Z.elems = 0;
  Z.k = wavenumber;
  Z.h = h;
  Z.eps = eps;
  const auto& Ls = H->tree.leaves;
  const uint32_t nl = (uint32_t)Ls.size();
  Z.rank.assign(nl, -1);
  Z.aca_rank.assign(nl, -1);
  Z.off.assign(nl, 0);
  H->stat_ws_bytes = H->stat_retries = H->stat_batches = 0;
  std::vector<AcaTask> tasks;
  std::vector<uint32_t> dense;
  const uint32_t kcap0 = aca_kcap_default();
  for (uint32_t l = 0; l < nl; ++l) {
    const Leaf& L = Ls[l];
    const uint32_t maxk = maxk_of(L.n1, L.n2, rankmax);
    if (L.adm && maxk) tasks.push_back(AcaTask{L.b1, L.n1, L.b2, L.n2, L.i0, maxk, std::min(kcap_limit(maxk), kcap0), l});
    else dense.push_back(l);
  }
  uint64_t est = 0;
  for (uint32_t l : dense) est += (uint64_t)Ls[l].n1 * Ls[l].n2;
  for (const AcaTask& t : tasks) est += (uint64_t)(t.n1 + t.n2) * std::min(t.kmax, 16u);
  if (Z.arena.bytes < est * sizeof(Cx)) {
    Z.arena.release();
    if ((rc = Z.arena.reserve(std::max<uint64_t>(est, 1) * sizeof(Cx)))) return rc;
  }
  const double* pts = H->pts.as<double>();
  const PointsSoA P{pts, pts + H->tree.n, pts + 2 * (size_t)H->tree.n};
  AcaParams par{};
  par.pts = P;
  par.k = wavenumber;
  par.h = h;
  par.eps = eps;
  if ((rc = run_aca(H, true, tasks, par, dense))) return rc;
  // dense leaves (inadmissible and failed ACA) in leaf order
  std::sort(dense.begin(), dense.end());
  for (uint32_t l : dense) {
    const Leaf& L = Ls[l];
    uint64_t off = 0;
    if ((rc = zarena_append(H, (uint64_t)L.n1 * L.n2, off))) return rc;
    Z.off[l] = off;
    Z.rank[l] = -1;
    Z.aca_rank[l] = -1;
  }
  const std::vector<DenseTask> dt = dense_tasks(Ls, H->tree.n, dense, Z.off);
  if (!dt.empty()) {
    ScopedBuf ddt;
    if ((rc = upload(ddt, dt, H->stream))) return rc;
    helm_dense_kernel<<<(uint32_t)dt.size(), 256, 0, H->stream>>>(P, wavenumber, h, ddt.as<DenseTask>(), Z.arena.as<Cx>());
    AHX_CUDA(cudaGetLastError());
  }
  AHX_CUDA(cudaStreamSynchronize(H->stream));
  Z.assembled = true;
  return AHX_OK;
}

extern "C" int ahx_helm_ranks(const ahx_hmat* H, int32_t* ranks) {
  if (!H || !ranks) return AHX_ERR_ARG;
  const HandleLock lk(H->mu);
  if (!H->z.assembled) {
    set_error("ahx_helm_ranks: Helmholtz leaves not assembled");
    return AHX_ERR_STATE;
  }
  std::copy(H->z.rank.begin(), H->z.rank.end(), ranks);
  return AHX_OK;
}

namespace {
// dense diagonal block of a symmetric tree: stored full, given out packed (SyM)
bool packed_zleaf(const ahx_hmat* H, uint32_t l) {
  const Leaf& L = H->tree.leaves[l];
  return H->tree.sym && H->z.rank[l] < 0 && L.b1 == L.b2;
}
}  // namespace

extern "C" uint64_t ahx_helm_leaf_size(const ahx_hmat* H, uint32_t l) {
  if (!H) return 0;
  const HandleLock lk(H->mu);
  if (!H->z.assembled || l >= H->tree.leaves.size()) return 0;
  const Leaf& L = H->tree.leaves[l];
  const int32_t r = H->z.rank[l];
  if (packed_zleaf(H, l)) return (uint64_t)L.n1 * (L.n1 + 1) / 2;
  return r < 0 ? (uint64_t)L.n1 * L.n2 : (uint64_t)r * (L.n1 + L.n2);
}

extern "C" int ahx_helm_get_leaf(const ahx_hmat* H, uint32_t l, double* out) {
  if (!H || !out) {
    set_error("ahx_helm_get_leaf: invalid argument");
    return AHX_ERR_ARG;
  }
  const HandleLock lk(H->mu);
  if (l >= H->tree.leaves.size()) {
    set_error("ahx_helm_get_leaf: invalid argument");
    return AHX_ERR_ARG;
  }
  if (!H->z.assembled) {
    set_error("ahx_helm_get_leaf: Helmholtz leaves not assembled");
    return AHX_ERR_STATE;
  }
  const uint64_t cnt = ahx_helm_leaf_size(H, l);
  if (!cnt) return AHX_OK;
  AHX_CUDA(cudaSetDevice(H->device));
  if (packed_zleaf(H, l)) {
    // upper triangle column by column (data[i + j (j + 1) / 2] = A(i, j), i <= j)
    const uint32_t n1 = H->tree.leaves[l].n1;
    std::vector<Cx> full((size_t)n1 * n1);
    AHX_CUDA(cudaMemcpyAsync(full.data(), H->z.arena.as<Cx>() + H->z.off[l], full.size() * sizeof(Cx),
                             cudaMemcpyDeviceToHost, H->stream));
    AHX_CUDA(cudaStreamSynchronize(H->stream));
    Cx* o = reinterpret_cast<Cx*>(out);
    for (uint32_t j = 0; j < n1; ++j)
      for (uint32_t i = 0; i <= j; ++i) o[i + (size_t)j * (j + 1) / 2] = full[i + (size_t)j * n1];
    return AHX_OK;
  }
  AHX_CUDA(cudaMemcpyAsync(out, H->z.arena.as<Cx>() + H->z.off[l], cnt * sizeof(Cx), cudaMemcpyDeviceToHost,
                           H->stream));
  AHX_CUDA(cudaStreamSynchronize(H->stream));
  return AHX_OK;
}

namespace ahx {
cudaError_t launch_zaca(const AcaParams& p, uint32_t grid, cudaStream_t s) {
  return lowrank::launch_aca_kernel(HelmGen{p.pts, p.k, p.h}, p, grid, s);
}
cudaError_t resident_zaca(int device, uint32_t& ctas) {
  return lowrank::resident_aca_kernel<HelmGen>(device, ctas);
}

cudaError_t launch_zmerge(const MergeParams& p, cudaStream_t s) {
  if (p.ntasks == 0) return cudaSuccess;
  zmerge_kernel<<<p.ntasks, 32, 0, s>>>(p);
  return cudaGetLastError();
}
}  // namespace ahx
