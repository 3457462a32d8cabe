// Learned ACA-rank predictor: an 8 -> 64 -> 64 -> 1 MLP (ReLU) with
// hand-written forward, backward and Adam kernels, trained on the GPU.
//
// Parameters (4801 floats): W1[8][64] b1[64] W2[64][64] b2[64] w3[64] b3.
// Inputs are normalised with per-feature mean / std fixed before training;
// the target is log(1 + ACA rank).
//
// A training step is two launches: mlp_grad_kernel takes 16 samples per CTA
// through forward and backward in shared memory and leaves one partial gradient
// per CTA; mlp_adam_kernel sums the partials and updates the parameters.  Every
// sum runs in a fixed order, so a training run is reproducible.  (With one
// thread per parameter walking all samples, the weight gradient alone took 0.3 ms
// of each 1,024-sample step.)
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <numeric>
#include <random>
#include <vector>

#include "ahx_hmat.hpp"

namespace ahx {
namespace {

constexpr int kIn = 8, kHid = 64;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kIn * kHid, kOffW2 = kOffB1 + kHid,
              kOffB2 = kOffW2 + kHid * kHid, kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid;
constexpr int kNParams = kOffB3 + 1;  // 4801

constexpr int kT = 256;        // threads of the sample kernels: 16 column groups x 16 samples
constexpr int kTS = 16;        // samples per pass of a CTA
// row stride of W2 and of the samples' rows in shared memory: 16-byte loads along
// a row, and of 16 consecutive rows at one column, hit every bank once per eighth
constexpr int kLd = kHid + 4;
constexpr int kPart = (kNParams + 3) / 4 * 4;  // row stride of the partial gradients
constexpr uint32_t kMaxParts = 512;  // CTAs (partial gradients) of one gradient

struct Shared {
  alignas(16) float w2[kHid * kLd];
  alignas(16) float w1[kIn * kHid];
  alignas(16) float h1[kTS][kLd], g2[kTS][kLd], g1[kTS][kLd], h2[kTS][kLd];
  alignas(16) float b1[kHid], b2[kHid], w3[kHid];
  float x[kTS][kIn], mean[kIn], std[kIn], out[kTS], dout[kTS], b3;
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// z += a w
__device__ __forceinline__ void fma4(float (&z)[4], float a, const float4& w) {
  z[0] = fmaf(a, w.x, z[0]);
  z[1] = fmaf(a, w.y, z[1]);
  z[2] = fmaf(a, w.z, z[2]);
  z[3] = fmaf(a, w.w, z[3]);
}

__device__ __forceinline__ void load_params(Shared& S, const float* __restrict__ p, const float* __restrict__ norm) {
  static_assert(kOffW2 % 4 == 0 && kOffB1 % 4 == 0 && kOffB2 % 4 == 0 && kOffW3 % 4 == 0, "16-byte loads");
  const int t = threadIdx.x;
  const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
  for (int i = 0; i < kHid * kHid / 4 / kT; ++i) {
    const int e = t + i * kT;
    *reinterpret_cast<float4*>(&S.w2[(e / (kHid / 4)) * kLd + 4 * (e % (kHid / 4))]) = q[kOffW2 / 4 + e];
  }
  if (t < kIn * kHid / 4) *reinterpret_cast<float4*>(&S.w1[4 * t]) = q[kOffW1 / 4 + t];
  else if (t < 128 + 16) *reinterpret_cast<float4*>(&S.b1[4 * (t - 128)]) = q[kOffB1 / 4 + t - 128];
  else if (t < 144 + 16) *reinterpret_cast<float4*>(&S.b2[4 * (t - 144)]) = q[kOffB2 / 4 + t - 144];
  else if (t < 160 + 16) *reinterpret_cast<float4*>(&S.w3[4 * (t - 160)]) = q[kOffW3 / 4 + t - 160];
  else if (t < 176 + kIn) S.mean[t - 176] = norm[t - 176];
  else if (t < 184 + kIn) S.std[t - 184] = norm[kIn + t - 184];
  else if (t == 192) S.b3 = p[kOffB3];
}

// Forward of samples s0 .. s0 + ns - 1 (ns <= 16; the rows of the others are
// zero).  Thread (tx, ty): columns 4 tx .. + 3 of sample ty, each summed over its
// inputs in order.  Leaves h1, h2 (after ReLU) and out.
__device__ __forceinline__ void forward(Shared& S, const float* __restrict__ X, const uint32_t* __restrict__ idx,
                                        uint32_t s0, uint32_t ns) {
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  __syncthreads();  // parameters loaded; the last pass's rows are no longer read
  if (t < kTS * kIn) {
    const int f = t % kIn, q = t / kIn;
    const uint32_t s = s0 + q;
    S.x[q][f] = (uint32_t)q < ns ? (X[(size_t)(idx ? idx[s] : s) * kIn + f] - S.mean[f]) / S.std[f] : 0.f;
  }
  __syncthreads();
  float4 b = ld4(&S.b1[4 * tx]);
  float z[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int f = 0; f < kIn; ++f) fma4(z, S.x[ty][f], ld4(&S.w1[f * kHid + 4 * tx]));
#pragma unroll
  for (int q = 0; q < 4; ++q) z[q] = fmaxf(z[q], 0.f);
  st4(&S.h1[ty][4 * tx], z);
  __syncwarp();  // a sample's 16 threads are half a warp
  b = ld4(&S.b2[4 * tx]);
  z[0] = b.x, z[1] = b.y, z[2] = b.z, z[3] = b.w;
#pragma unroll 8
  for (int i = 0; i < kHid; i += 4) {
    const float4 h = ld4(&S.h1[ty][i]);
    const float* w = &S.w2[i * kLd + 4 * tx];
    fma4(z, h.x, ld4(w));
    fma4(z, h.y, ld4(w + kLd));
    fma4(z, h.z, ld4(w + 2 * kLd));
    fma4(z, h.w, ld4(w + 3 * kLd));
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) z[q] = fmaxf(z[q], 0.f);
  st4(&S.h2[ty][4 * tx], z);
  const float4 w = ld4(&S.w3[4 * tx]);
  float y = fmaf(z[3], w.w, fmaf(z[2], w.z, fmaf(z[1], w.y, z[0] * w.x)));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
  if (tx == 0) S.out[ty] = y + S.b3;
  __syncwarp();
}

// Predictions, and with Y the squared error: err[block] = its sum over the block's samples.
__global__ void __launch_bounds__(kT) mlp_fwd_kernel(const float* __restrict__ X, uint32_t n,
                                                     const float* __restrict__ params, const float* __restrict__ norm,
                                                     const float* __restrict__ Y, float* __restrict__ out,
                                                     float* __restrict__ err) {
  __shared__ Shared S;
  load_params(S, params, norm);
  const int t = threadIdx.x;
  float e = 0.f;
  for (uint32_t s0 = blockIdx.x * kTS; s0 < n; s0 += gridDim.x * kTS) {
    const uint32_t ns = min((uint32_t)kTS, n - s0);
    forward(S, X, nullptr, s0, ns);
    __syncthreads();
    if ((uint32_t)t < ns) {
      const float y = S.out[t];
      if (out) out[s0 + t] = y;
      if (Y) {
        const float d = y - Y[s0 + t];
        e = fmaf(d, d, e);
      }
    }
  }
  if (err && t < 32) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (t == 0) err[blockIdx.x] = e;
  }
}

// sum[0] = err[0] + .. + err[n - 1] (one warp, fixed order)
__global__ void mlp_sum_kernel(const float* __restrict__ err, uint32_t n, float* __restrict__ sum) {
  float e = 0.f;
  for (uint32_t i = threadIdx.x; i < n; i += 32) e += err[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (threadIdx.x == 0) *sum = e;
}

// Partial gradient of the mean squared error: CTA b takes passes of 16 samples
// b, b + gridDim.x, .. and writes part[b][param].  Thread (tx, ty) owns rows 4 ty
// .. + 3 x columns 4 tx .. + 3 of dW2, summed over the samples in registers.
__global__ void __launch_bounds__(kT) mlp_grad_kernel(const float* __restrict__ X, const float* __restrict__ Y,
                                                      const uint32_t* __restrict__ idx, uint32_t n, float inv_n,
                                                      const float* __restrict__ params,
                                                      const float* __restrict__ norm, float* __restrict__ part,
                                                      float* __restrict__ err) {
  __shared__ Shared S;
  load_params(S, params, norm);
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  float w2[4][4] = {}, w1[2] = {}, vec = 0.f, b3 = 0.f, e = 0.f;
  for (uint32_t s0 = blockIdx.x * kTS; s0 < n; s0 += gridDim.x * kTS) {
    const uint32_t ns = min((uint32_t)kTS, n - s0);
    forward(S, X, idx, s0, ns);
    // dout = 2 (out - y) / n, dZ2, dZ1 (zero for the samples past n)
    float d = 0.f;
    if ((uint32_t)ty < ns) {
      const uint32_t s = s0 + ty;
      const float r = S.out[ty] - Y[idx ? idx[s] : s];
      d = 2.f * r * inv_n;
      if (tx == 0) e = fmaf(r, r, e);
    }
    if (tx == 0) S.dout[ty] = d;
    {
      const float4 h = ld4(&S.h2[ty][4 * tx]), w = ld4(&S.w3[4 * tx]);
      const float g[4] = {h.x > 0.f ? d * w.x : 0.f, h.y > 0.f ? d * w.y : 0.f, h.z > 0.f ? d * w.z : 0.f,
                          h.w > 0.f ? d * w.w : 0.f};
      st4(&S.g2[ty][4 * tx], g);
    }
    __syncwarp();
    // dZ1 rows tx + 16 q
    float g[4] = {};
#pragma unroll 8
    for (int o = 0; o < kHid; o += 4) {
      const float4 v = ld4(&S.g2[ty][o]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 w = ld4(&S.w2[(tx + 16 * q) * kLd + o]);
        g[q] = fmaf(w.x, v.x, g[q]);
        g[q] = fmaf(w.y, v.y, g[q]);
        g[q] = fmaf(w.z, v.z, g[q]);
        g[q] = fmaf(w.w, v.w, g[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = tx + 16 * q;
      S.g1[ty][i] = S.h1[ty][i] > 0.f ? g[q] : 0.f;
    }
    __syncthreads();
    // sums over the pass's samples, in order
#pragma unroll 4
    for (int s = 0; s < kTS; ++s) {
      const float4 h = ld4(&S.h1[s][4 * ty]), v = ld4(&S.g2[s][4 * tx]);
      fma4(w2[0], h.x, v);
      fma4(w2[1], h.y, v);
      fma4(w2[2], h.z, v);
      fma4(w2[3], h.w, v);
    }
    const int o = t % kHid, f = t / kHid;  // W1 rows f, f + 4; b1, b2, w3: f = 0, 1, 2
#pragma unroll 4
    for (int s = 0; s < kTS; ++s) {
      const float v = S.g1[s][o];
      w1[0] = fmaf(S.x[s][f], v, w1[0]);
      w1[1] = fmaf(S.x[s][f + 4], v, w1[1]);
      if (f == 0) vec += v;
      else if (f == 1) vec += S.g2[s][o];
      else if (f == 2) vec = fmaf(S.h2[s][o], S.dout[s], vec);
      else if (o == 0) b3 += S.dout[s];
    }
  }
  float* p = part + (size_t)blockIdx.x * kPart;
#pragma unroll
  for (int r = 0; r < 4; ++r) st4(&p[kOffW2 + (4 * ty + r) * kHid + 4 * tx], w2[r]);
  const int o = t % kHid, f = t / kHid;
  p[kOffW1 + f * kHid + o] = w1[0];
  p[kOffW1 + (f + 4) * kHid + o] = w1[1];
  if (f == 0) p[kOffB1 + o] = vec;
  else if (f == 1) p[kOffB2 + o] = vec;
  else if (f == 2) p[kOffW3 + o] = vec;
  else if (o == 0) p[kOffB3] = b3;
  if (err) {  // (a kernel argument: the same for all threads)
    __syncthreads();
    if (tx == 0) S.out[ty] = e;
    __syncthreads();
    if (t == 0) {
      float sum = 0.f;
      for (int s = 0; s < kTS; ++s) sum += S.out[s];
      err[blockIdx.x] = sum;
    }
  }
}

// Sums the partial gradients; with m the Adam update of the parameters (Kingma and
// Ba), else the gradient itself to grad.  A thread adds every eighth partial of
// four parameters, the eight sums are added in order.
constexpr int kAdamSlices = 8, kAdamQuads = 16;  // per CTA: 128 threads, 64 parameters
__global__ void __launch_bounds__(kAdamSlices* kAdamQuads)
    mlp_adam_kernel(const float* __restrict__ part, uint32_t parts, float* __restrict__ grad, float* __restrict__ p,
                    float* __restrict__ m, float* __restrict__ v, float lr, float b1t, float b2t) {
  __shared__ float4 sum[kAdamSlices][kAdamQuads];
  const int quad = threadIdx.x % kAdamQuads, sl = threadIdx.x / kAdamQuads;
  const int q4 = blockIdx.x * kAdamQuads + quad;
  float s[4] = {};
  if (q4 < kPart / 4) {
#pragma unroll 8
    for (uint32_t b = sl; b < parts; b += kAdamSlices)
      fma4(s, 1.f, __ldg(reinterpret_cast<const float4*>(part + (size_t)b * kPart) + q4));
  }
  sum[sl][quad] = make_float4(s[0], s[1], s[2], s[3]);
  __syncthreads();
  const int i = blockIdx.x * kAdamQuads * 4 + threadIdx.x;
  if (threadIdx.x >= kAdamQuads * 4 || i >= kNParams) return;
  float g = 0.f;
#pragma unroll
  for (int k = 0; k < kAdamSlices; ++k) g += reinterpret_cast<const float*>(&sum[k][0])[threadIdx.x];
  if (!m) {
    grad[i] = g;
    return;
  }
  const float b1 = 0.9f, b2 = 0.999f;
  m[i] = b1 * m[i] + (1.f - b1) * g;
  v[i] = b2 * v[i] + (1.f - b2) * g * g;
  const float mh = m[i] / (1.f - b1t), vh = v[i] / (1.f - b2t);
  p[i] -= lr * mh / (sqrtf(vh) + 1e-8f);
}
constexpr unsigned kAdamGrid = (kPart / 4 + kAdamQuads - 1) / kAdamQuads;

}  // namespace
}  // namespace ahx

using namespace ahx;

struct ahx_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  ahx::DevBuf state;  // params, m, v (kPart floats each), norm
  float* params() const { return state.as<float>(); }
  float* m() const { return params() + kPart; }
  float* v() const { return params() + 2 * kPart; }
  float* norm() const { return params() + 3 * kPart; }
  ahx::DevBuf part, out, X, Y, err;  // work buffers (kept between calls)
  uint64_t step = 0;
};

namespace {

uint32_t parts_of(uint32_t n) { return std::min<uint32_t>((n + kTS - 1) / kTS, kMaxParts); }

// CTAs of a forward over n samples: passes of 16, at most a few per CTA
unsigned fwd_grid(uint32_t n) { return std::min<uint32_t>((n + kTS - 1) / kTS, 152u * 4); }

// partial gradients of the samples idx[0..n) of (X, Y); parts_of(n) of them
int mlp_grad(ahx_mlp* M, const float* X, const float* Y, const uint32_t* idx, uint32_t n, float* err) {
  int rc = M->part.reserve((size_t)parts_of(n) * kPart * sizeof(float));
  if (rc) return rc;
  mlp_grad_kernel<<<parts_of(n), kT, 0, M->stream>>>(X, Y, idx, n, 1.f / (float)n, M->params(),
                                                     M->norm(), M->part.as<float>(), err);
  AHX_CUDA(cudaGetLastError());
  return AHX_OK;
}

}  // namespace

extern "C" {

uint32_t ahx_mlp_nparams(void) { return (uint32_t)kNParams; }

int ahx_mlp_create(int device, uint64_t seed, ahx_mlp** out) {
  if (!out) return AHX_ERR_ARG;
  *out = nullptr;
  AHX_CUDA(cudaSetDevice(device));
  ahx_mlp* M = new (std::nothrow) ahx_mlp;
  if (!M) return AHX_ERR_NOMEM;
  M->device = device;
  cudaError_t e = cudaStreamCreateWithFlags(&M->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete M;
    return cuda_fail(e, "cudaStreamCreate");
  }
  // He initialisation from a fixed-seed host generator (reproducible)
  std::vector<float> p(3 * kPart + 2 * kIn, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<double> nd(0.0, 1.0);
  for (int i = 0; i < kIn * kHid; ++i) p[kOffW1 + i] = (float)(nd(rng) * std::sqrt(2.0 / kIn));
  for (int i = 0; i < kHid * kHid; ++i) p[kOffW2 + i] = (float)(nd(rng) * std::sqrt(2.0 / kHid));
  for (int i = 0; i < kHid; ++i) p[kOffW3 + i] = (float)(nd(rng) * std::sqrt(1.0 / kHid));
  for (int f = 0; f < kIn; ++f) p[3 * kPart + kIn + f] = 1.f;
  int rc = M->state.reserve(p.size() * 4);
  if (rc == AHX_OK && (e = cudaMemcpy(M->state.p, p.data(), p.size() * 4, cudaMemcpyHostToDevice)) != cudaSuccess)
    rc = cuda_fail(e, "cudaMemcpy");
  if (rc) {
    ahx_mlp_destroy(M);
    return rc;
  }
  *out = M;
  return AHX_OK;
}

int ahx_mlp_destroy(ahx_mlp* M) {
  if (!M) return AHX_OK;
  cudaSetDevice(M->device);
  if (M->stream) cudaStreamSynchronize(M->stream);
  for (DevBuf* b : {&M->state, &M->part, &M->out, &M->X, &M->Y, &M->err}) b->release();
  if (M->stream) cudaStreamDestroy(M->stream);
  delete M;
  return AHX_OK;
}

int ahx_mlp_get_params(const ahx_mlp* M, float* out) {
  if (!M || !out) return AHX_ERR_ARG;
  AHX_CUDA(cudaSetDevice(M->device));
  AHX_CUDA(cudaMemcpy(out, M->params(), kNParams * 4, cudaMemcpyDeviceToHost));
  return AHX_OK;
}

int ahx_mlp_set_params(ahx_mlp* M, const float* in) {
  if (!M || !in) return AHX_ERR_ARG;
  AHX_CUDA(cudaSetDevice(M->device));
  AHX_CUDA(cudaMemcpy(M->params(), in, kNParams * 4, cudaMemcpyHostToDevice));
  return AHX_OK;
}

// feature normalisation: mean[8], std[8]
int ahx_mlp_set_norm(ahx_mlp* M, const float* mean, const float* stdev) {
  if (!M || !mean || !stdev) return AHX_ERR_ARG;
  float nm[2 * kIn];
  for (int f = 0; f < kIn; ++f) {
    nm[f] = mean[f];
    nm[kIn + f] = stdev[f] > 0.f ? stdev[f] : 1.f;
  }
  AHX_CUDA(cudaSetDevice(M->device));
  AHX_CUDA(cudaMemcpy(M->norm(), nm, sizeof(nm), cudaMemcpyHostToDevice));
  return AHX_OK;
}

// mean[8] and std[8] of the columns of X (host, n x 8), for ahx_mlp_set_norm
int ahx_mlp_moments(const float* X, uint32_t n, float* mean, float* stdev) {
  if (!X || !mean || !stdev || n == 0) return AHX_ERR_ARG;
  column_moments(X, n, mean, stdev);
  return AHX_OK;
}

// Gradient of the mean squared error over all n samples (host arrays), for checking.
int ahx_mlp_gradients(ahx_mlp* M, const float* X, const float* Y, uint32_t n, float* grad,
                      float* loss) {
  if (!M || !X || !Y || !grad || n == 0) return AHX_ERR_ARG;
  AHX_CUDA(cudaSetDevice(M->device));
  int rc;
  if ((rc = M->X.reserve((size_t)n * kIn * 4)) || (rc = M->Y.reserve((size_t)n * 4))) return rc;
  AHX_CUDA(cudaMemcpyAsync(M->X.p, X, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, M->stream));
  AHX_CUDA(cudaMemcpyAsync(M->Y.p, Y, (size_t)n * 4, cudaMemcpyHostToDevice, M->stream));
  // gradient, then the sum of the squared errors
  const uint32_t parts = parts_of(n);
  if ((rc = M->out.reserve((size_t)(kNParams + 1) * 4)) || (rc = M->err.reserve((size_t)parts * 4))) return rc;
  if ((rc = mlp_grad(M, M->X.as<float>(), M->Y.as<float>(), nullptr, n, M->err.as<float>()))) return rc;
  float* out = M->out.as<float>();
  mlp_adam_kernel<<<kAdamGrid, kAdamSlices * kAdamQuads, 0, M->stream>>>(M->part.as<float>(), parts, out, nullptr, nullptr,
                                                                 nullptr, 0.f, 0.f, 0.f);
  mlp_sum_kernel<<<1, 32, 0, M->stream>>>(M->err.as<float>(), parts, out + kNParams);
  AHX_CUDA(cudaGetLastError());
  float se = 0.f;
  AHX_CUDA(cudaMemcpyAsync(grad, out, kNParams * 4, cudaMemcpyDeviceToHost, M->stream));
  AHX_CUDA(cudaMemcpyAsync(&se, out + kNParams, 4, cudaMemcpyDeviceToHost, M->stream));
  AHX_CUDA(cudaStreamSynchronize(M->stream));
  if (loss) *loss = se / (float)n;
  return AHX_OK;
}

// Adam on mini-batches of (X, Y) (host arrays, n samples), `epochs` passes in a
// fixed-seed shuffled order; loss[e] = training MSE after epoch e (may be NULL).
int ahx_mlp_train(ahx_mlp* M, const float* X, const float* Y, uint32_t n, uint32_t epochs,
                  uint32_t batch, float lr, uint64_t seed, float* loss) {
  if (!M || !X || !Y || n == 0 || batch == 0) return AHX_ERR_ARG;
  AHX_CUDA(cudaSetDevice(M->device));
  int rc;
  if ((rc = M->X.reserve((size_t)n * kIn * 4)) || (rc = M->Y.reserve((size_t)n * 4))) return rc;
  const unsigned fg = fwd_grid(n);
  if ((rc = M->part.reserve((size_t)parts_of(std::min(batch, n)) * kPart * sizeof(float)))) return rc;
  if ((rc = M->err.reserve((size_t)(fg + epochs) * 4))) return rc;
  float* const dloss = M->err.as<float>() + fg;  // squared error after each epoch
  AHX_CUDA(cudaMemcpyAsync(M->X.p, X, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, M->stream));
  AHX_CUDA(cudaMemcpyAsync(M->Y.p, Y, (size_t)n * 4, cudaMemcpyHostToDevice, M->stream));
  std::vector<uint32_t> order(n);
  std::iota(order.begin(), order.end(), 0u);
  std::mt19937_64 rng(seed);
  // two order buffers: the host shuffles and hands over the next epoch's order
  // while the GPU runs the present one
  ScopedBuf dorder[2];
  std::vector<uint32_t> staged[2];
  for (int q = 0; q < 2; ++q) {
    if ((rc = dorder[q].reserve((size_t)n * 4))) return rc;
    staged[q].resize(n);
  }
  struct Events {
    cudaEvent_t e[2] = {nullptr, nullptr};
    ~Events() {
      for (auto x : e)
        if (x) cudaEventDestroy(x);
    }
  } done;
  for (auto& x : done.e) AHX_CUDA(cudaEventCreateWithFlags(&x, cudaEventDisableTiming));
  // copies from `staged` may still be read until the epoch that uses them is over:
  // whatever happens, the stream is idle before the vectors go
  struct Idle {
    cudaStream_t s;
    ~Idle() { cudaStreamSynchronize(s); }
  } idle{M->stream};
  for (uint32_t e = 0; e < epochs; ++e) {
    const int q = (int)(e & 1);
    std::shuffle(order.begin(), order.end(), rng);
    if (e >= 2) AHX_CUDA(cudaEventSynchronize(done.e[q]));
    std::copy(order.begin(), order.end(), staged[q].begin());
    AHX_CUDA(cudaMemcpyAsync(dorder[q].p, staged[q].data(), (size_t)n * 4, cudaMemcpyHostToDevice, M->stream));
    for (uint32_t b0 = 0; b0 < n; b0 += batch) {
      const uint32_t nb = std::min(batch, n - b0);
      if ((rc = mlp_grad(M, M->X.as<float>(), M->Y.as<float>(), dorder[q].as<uint32_t>() + b0, nb, nullptr))) return rc;
      ++M->step;
      const float b1t = (float)std::pow(0.9, (double)M->step), b2t = (float)std::pow(0.999, (double)M->step);
      mlp_adam_kernel<<<kAdamGrid, kAdamSlices * kAdamQuads, 0, M->stream>>>(M->part.as<float>(), parts_of(nb), nullptr,
                                                                  M->params(), M->m(),
                                                                  M->v(), lr, b1t, b2t);
    }
    if (loss) {
      mlp_fwd_kernel<<<fg, kT, 0, M->stream>>>(M->X.as<float>(), n, M->params(), M->norm(),
                                               M->Y.as<float>(), nullptr, M->err.as<float>());
      mlp_sum_kernel<<<1, 32, 0, M->stream>>>(M->err.as<float>(), fg, dloss + e);
    }
    AHX_CUDA(cudaEventRecord(done.e[q], M->stream));
  }
  AHX_CUDA(cudaGetLastError());
  if (loss && epochs) {
    AHX_CUDA(cudaMemcpyAsync(loss, dloss, (size_t)epochs * 4, cudaMemcpyDeviceToHost, M->stream));
    AHX_CUDA(cudaStreamSynchronize(M->stream));
    for (uint32_t e = 0; e < epochs; ++e) loss[e] /= (float)n;
  }
  AHX_CUDA(cudaStreamSynchronize(M->stream));
  return AHX_OK;
}

int ahx_mlp_predict(ahx_mlp* M, const float* X, uint32_t n, float* out) {
  if (!M || !X || !out) return AHX_ERR_ARG;
  if (n == 0) return AHX_OK;
  AHX_CUDA(cudaSetDevice(M->device));
  int rc;
  if ((rc = M->X.reserve((size_t)n * kIn * 4)) || (rc = M->out.reserve((size_t)n * 4))) return rc;
  AHX_CUDA(cudaMemcpyAsync(M->X.p, X, (size_t)n * kIn * 4, cudaMemcpyHostToDevice, M->stream));
  mlp_fwd_kernel<<<fwd_grid(n), kT, 0, M->stream>>>(M->X.as<float>(), n, M->params(), M->norm(),
                                                   nullptr, M->out.as<float>(), nullptr);
  AHX_CUDA(cudaGetLastError());
  AHX_CUDA(cudaMemcpyAsync(out, M->out.p, (size_t)n * 4, cudaMemcpyDeviceToHost, M->stream));
  AHX_CUDA(cudaStreamSynchronize(M->stream));
  return AHX_OK;
}

}  // extern "C"
