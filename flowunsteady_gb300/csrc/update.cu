// update.cu — the O(N) FP64 kernels of a time step: what happens to the particles
// between two pair passes (post_kernel, with the functions of update_dev.cuh, in one
// launch: six launches of 4 to 11 µs a stage of a small field before), relaxation and
// the diagnostics.
#include "internal.h"
#include "update.h"
#include "update_dev.cuh"
#include "vpm_device.cuh"

namespace vpm {

template <int KERNEL>
__global__ void __launch_bounds__(kPostThreads) post_kernel(const PostArgs p) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < p.n) post_particle<KERNEL>(p, i);
}

// Backscatter clipping on its own (vpm.clipping_backscatter): C_d = 0 where
// C_d Γ·E_str < 0.
__global__ void sfs_clip_kernel(int64_t nv, const uint8_t* __restrict__ stat, int64_t ld,
                                const double* __restrict__ G, const double* __restrict__ E,
                                double* __restrict__ C) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nv || (stat && stat[i])) return;
  const double ge = G[i] * E[i] + G[ld + i] * E[ld + i] + G[2 * ld + i] * E[2 * ld + i];
  if (C[i] * ge < 0.0) C[i] = 0.0;
}

// Pedrizzetti relaxation: Γ <- (1-r)Γ + r|Γ| ω/|ω|, ω = ∇×u from J.
__global__ void relax_kernel(int64_t nv, const uint8_t* __restrict__ stat, int64_t ld,
                             const double* __restrict__ J, double* G, double r) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= nv || (stat && stat[i])) return;
  const double w0 = J[7 * ld + i] - J[5 * ld + i];
  const double w1 = J[2 * ld + i] - J[6 * ld + i];
  const double w2 = J[3 * ld + i] - J[1 * ld + i];
  const double nw = sqrt(w0 * w0 + w1 * w1 + w2 * w2);
  if (nw == 0.0) return;
  const double g0 = G[i], g1 = G[ld + i], g2 = G[2 * ld + i];
  const double ng = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
  G[i] = (1.0 - r) * g0 + r * ng * w0 / nw;
  G[ld + i] = (1.0 - r) * g1 + r * ng * w1 / nw;
  G[2 * ld + i] = (1.0 - r) * g2 + r * ng * w2 / nw;
}

__global__ void zero_kernel(double* p, int64_t n) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) p[i] = 0.0;
}

// ------------------------------------------------------------ reductions --
// Deterministic two-level FP64 reductions: kRedBlocks blocks each reduce a
// fixed, strided share of the particles in a fixed tree order into a partial
// row; one block then reduces the rows in order.
constexpr int kRedThreads = 256;

struct DiagAcc {
  double v[kDiagSlots];
};

__device__ inline void diag_combine(DiagAcc& a, const DiagAcc& b) {
#pragma unroll
  for (int k = 0; k < kDiagSlots; ++k) {
    if (k == DS_CMIN) a.v[k] = fmin(a.v[k], b.v[k]);
    else if (k == DS_CMAX) a.v[k] = fmax(a.v[k], b.v[k]);
    else a.v[k] += b.v[k];
  }
}

__device__ inline void diag_identity(DiagAcc& a) {
#pragma unroll
  for (int k = 0; k < kDiagSlots; ++k) a.v[k] = 0.0;
  a.v[DS_CMIN] = INFINITY;
  a.v[DS_CMAX] = -INFINITY;
}

__device__ inline void block_reduce(DiagAcc& acc, DiagAcc* sh) {
  const int t = threadIdx.x;
  sh[t] = acc;
  __syncthreads();
  for (int s = kRedThreads / 2; s > 0; s >>= 1) {
    if (t < s) {
      DiagAcc o = sh[t + s];
      diag_combine(sh[t], o);
    }
    __syncthreads();
  }
  acc = sh[0];
}

// raw: ζ sums (rows 0..2 Ω without self) or null (no enstrophy).
// C_d statistics cover the free particles: [0, nf) without flags, or every
// particle whose static flag is zero (stat non-null).
__global__ void __launch_bounds__(kRedThreads) diag_partial_kernel(
    int64_t n, int64_t nf, const uint8_t* __restrict__ stat, int64_t ld,
    const double* __restrict__ X, const double* __restrict__ G, const double* __restrict__ S,
    const double* __restrict__ C, const double* __restrict__ raw, double zeta0,
    double* partial) {
  __shared__ DiagAcc sh[kRedThreads];
  DiagAcc acc;
  diag_identity(acc);
  for (int64_t i = int64_t(blockIdx.x) * kRedThreads + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * kRedThreads) {
    const double x0 = X[i], x1 = X[ld + i], x2 = X[2 * ld + i];
    const double g0 = G[i], g1 = G[ld + i], g2 = G[2 * ld + i];
    const double sg = S[i];
    if (raw) {
      const double self = zeta0 / (sg * sg * sg);
      acc.v[DS_ENS] += 0.5 * (g0 * (raw[i] + self * g0) + g1 * (raw[ld + i] + self * g1) +
                              g2 * (raw[2 * ld + i] + self * g2));
    }
    acc.v[DS_IX] += 0.5 * (x1 * g2 - x2 * g1);
    acc.v[DS_IY] += 0.5 * (x2 * g0 - x0 * g2);
    acc.v[DS_IZ] += 0.5 * (x0 * g1 - x1 * g0);
    acc.v[DS_GX] += g0;
    acc.v[DS_GY] += g1;
    acc.v[DS_GZ] += g2;
    acc.v[DS_SIG] += sg;
    const bool fin = isfinite(x0) && isfinite(x1) && isfinite(x2) && isfinite(g0) &&
                     isfinite(g1) && isfinite(g2) && isfinite(sg);
    acc.v[DS_NONFIN] += fin ? 0.0 : 1.0;
    if (C && (stat ? !stat[i] : i < nf)) {
      const double c = C[i];
      if (c == 0.0) {
        acc.v[DS_CZERO] += 1.0;
      } else {
        const double c2 = c * c;
        acc.v[DS_CCNT] += 1.0;
        acc.v[DS_CSUM] += c;
        acc.v[DS_CSUM2] += c2;
        acc.v[DS_CSUM3] += c2 * c;
        acc.v[DS_CSUM4] += c2 * c2;
        acc.v[DS_CMIN] = fmin(acc.v[DS_CMIN], c);
        acc.v[DS_CMAX] = fmax(acc.v[DS_CMAX], c);
      }
    }
  }
  block_reduce(acc, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < kDiagSlots; ++k) partial[int64_t(blockIdx.x) * kDiagSlots + k] = acc.v[k];
}

__global__ void __launch_bounds__(kRedThreads) diag_final_kernel(int nblocks,
                                                                 const double* __restrict__ partial,
                                                                 double* out) {
  __shared__ DiagAcc sh[kRedThreads];
  DiagAcc acc;
  diag_identity(acc);
  for (int b = threadIdx.x; b < nblocks; b += kRedThreads) {
    DiagAcc o;
    for (int k = 0; k < kDiagSlots; ++k) o.v[k] = partial[int64_t(b) * kDiagSlots + k];
    diag_combine(acc, o);
  }
  block_reduce(acc, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < kDiagSlots; ++k) out[k] = acc.v[k];
}

// Σ|Γ| x and Σ|Γ| over [i0, i1) -> out[4] (same two-level structure).
__global__ void __launch_bounds__(kRedThreads) centroid_partial_kernel(
    int64_t i0, int64_t i1, int64_t ld, const double* __restrict__ X,
    const double* __restrict__ G, double* partial) {
  __shared__ DiagAcc sh[kRedThreads];
  DiagAcc acc;
  diag_identity(acc);
  acc.v[DS_CMIN] = 0.0;
  acc.v[DS_CMAX] = 0.0;
  for (int64_t i = i0 + int64_t(blockIdx.x) * kRedThreads + threadIdx.x; i < i1;
       i += int64_t(gridDim.x) * kRedThreads) {
    const double g0 = G[i], g1 = G[ld + i], g2 = G[2 * ld + i];
    const double w = sqrt(g0 * g0 + g1 * g1 + g2 * g2);
    acc.v[0] += w * X[i];
    acc.v[1] += w * X[ld + i];
    acc.v[2] += w * X[2 * ld + i];
    acc.v[3] += w;
  }
  block_reduce(acc, sh);
  if (threadIdx.x == 0)
    for (int k = 0; k < kDiagSlots; ++k) partial[int64_t(blockIdx.x) * kDiagSlots + k] = acc.v[k];
}

// ---------------------------------------------------------------- launchers --
static inline int grid_for(int64_t n, int bs) { return int((n + bs - 1) / bs); }

cudaError_t launch_post(int kernel, const PostArgs& p, cudaStream_t st) {
  if (p.n <= 0 || p.flags == 0) return cudaSuccess;
  const int grid = grid_for(p.n, kPostThreads);
  if (kernel == VPM_KERNEL_WINCKELMANS)
    post_kernel<VPM_KERNEL_WINCKELMANS><<<grid, kPostThreads, 0, st>>>(p);
  else
    post_kernel<VPM_KERNEL_GAUSSIANERF><<<grid, kPostThreads, 0, st>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_sfs_clip(int64_t nv, const uint8_t* stat, int64_t ld, const double* G,
                            const double* E, double* C, cudaStream_t st) {
  if (nv <= 0) return cudaSuccess;
  sfs_clip_kernel<<<grid_for(nv, 256), 256, 0, st>>>(nv, stat, ld, G, E, C);
  return cudaGetLastError();
}

cudaError_t launch_relax(int64_t nv, const uint8_t* stat, int64_t ld, const double* J, double* G,
                         double r, cudaStream_t st) {
  if (nv <= 0) return cudaSuccess;
  relax_kernel<<<grid_for(nv, 256), 256, 0, st>>>(nv, stat, ld, J, G, r);
  return cudaGetLastError();
}

cudaError_t launch_zero(double* p, int64_t n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  zero_kernel<<<grid_for(n, 256), 256, 0, st>>>(p, n);
  return cudaGetLastError();
}

cudaError_t launch_diagnostics(int64_t n, int64_t nf, const uint8_t* stat, int64_t ld,
                               const double* X, const double* G, const double* S, const double* C,
                               const double* raw, double zeta0, double* partial, double* out,
                               cudaStream_t st) {
  diag_partial_kernel<<<kRedBlocks, kRedThreads, 0, st>>>(n, nf, stat, ld, X, G, S, C, raw, zeta0,
                                                          partial);
  diag_final_kernel<<<1, kRedThreads, 0, st>>>(kRedBlocks, partial, out);
  return cudaGetLastError();
}

cudaError_t launch_centroid(int64_t i0, int64_t i1, int64_t ld, const double* X, const double* G,
                            double* partial, double* out, cudaStream_t st) {
  centroid_partial_kernel<<<kRedBlocks, kRedThreads, 0, st>>>(i0, i1, ld, X, G, partial);
  diag_final_kernel<<<1, kRedThreads, 0, st>>>(kRedBlocks, partial, out);
  return cudaGetLastError();
}

}  // namespace vpm
