// ffv.cu — free-vortex force terms of bound particles (FLOWUnsteady's
// _Ffv_direct, src/FLOWUnsteady_processing_force.jl:879-929) on the GPU.
//
// For every bound particle b and every free particle f with r = |x_f - x_b| > 0
// (kernel evaluated with the bound core σ_b, q = g(r/σ_b)/r³, Δx = x_f - x_b):
//   M[0:3] = Σ_f U_b(x_f) × Γ_f,  U_b(x_f) = -q/(4π) (Δx × Γ_b)
//   M[3:6] = Σ_f q/(4π) Δx × (Γ_b × Γ_f)
// With (Δx × Γ_b) × Γ_f = Γ_b (Δx·Γ_f) - Δx (Γ_b·Γ_f) and
// Δx × (Γ_b × Γ_f) = Γ_b (Δx·Γ_f) - Γ_f (Δx·Γ_b), everything follows from the nine
// sums T = Σ_f q Δx ⊗ Γ_f, formed with 3 products and 9 FMAs a pair:
//   M[0:3] = -(Γ_b tr T - T Γ_b)/(4π),   M[3:6] = (Γ_b tr T - Tᵀ Γ_b)/(4π).
// FP64 throughout (a force evaluation over bound particles).  Bound by the FP64
// pipe (about two operations per SM and cycle): 27 to 30 operations a pair.  Bound
// particles are scattered over the rotor, so that nearly every warp holds pairs
// inside and outside the core at every source; with erf, exp and the series in a
// branch each, a pair took 200 operations.  421 bound and 30,011 free particles:
// 4.10 -> 0.93 ms, and the sum of the chunks 145 -> 21 µs.
// One thread per bound particle; free particles are staged in shared-memory tiles;
// the free range is split into chunks summed afterwards in fixed order.
#include <cuda_runtime.h>

#include "capi_internal.h"
#include "pair_f64.cuh"

namespace vpm {

constexpr int kFfvBlock = 128;
constexpr int kFfvNval = 9;

// M of bound particle b from T.
__device__ __forceinline__ void ffv_finish(const double* T, const double* __restrict__ gb, int64_t ldb,
                                           int64_t b, double* M, int64_t ldm) {
  const double g[3] = {gb[b], gb[ldb + b], gb[2 * ldb + b]};
  const double s = T[0] + T[4] + T[8], w = kInv4Pi;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double tg = T[3 * i] * g[0] + T[3 * i + 1] * g[1] + T[3 * i + 2] * g[2];
    const double gt = T[i] * g[0] + T[3 + i] * g[1] + T[6 + i] * g[2];
    M[i * ldm + b] = -w * (g[i] * s - tg);
    M[(3 + i) * ldm + b] = w * (g[i] * s - gt);
  }
}

template <int KERNEL>
__global__ void __launch_bounds__(kFfvBlock) ffv_kernel(int64_t nb, const double* __restrict__ xb,
                                                        const double* __restrict__ gb,
                                                        const double* __restrict__ sb, int64_t ldb,
                                                        int64_t nf, const double* __restrict__ xf,
                                                        const double* __restrict__ gf, int64_t ldf,
                                                        int64_t chunk, int n_tb, double* part,
                                                        double* M, int64_t ldm, int n_chunk) {
  __shared__ double sx[kFfvBlock][3], sg[kFfvBlock][3];
  extern __shared__ __align__(16) double ffv_tab[];   // Gaussian-erf: the core table
  constexpr bool GAUSS = KERNEL == VPM_KERNEL_GAUSSIANERF;
  if constexpr (GAUSS) stage_table(ffv_tab, d_core_table.v, kCoreRows * kCoreCoef);
  const int tid = threadIdx.x;
  const int tb = blockIdx.x % n_tb, c = blockIdx.x / n_tb;
  const int64_t b = int64_t(tb) * kFfvBlock + tid;
  const bool valid = b < nb;
  double bx = 0, by = 0, bz = 0, sig = 1.0;
  if (valid) {
    bx = xb[b]; by = xb[ldb + b]; bz = xb[2 * ldb + b];
    sig = sb[b];
  }
  double ka, kb, kc, u0, u1, u2;   // constants of the bound core σ_b
  uj_consts_f64<KERNEL, false>(sig, ka, kb, kc, u0, u1, u2);
  double T[kFfvNval];
#pragma unroll
  for (int k = 0; k < kFfvNval; ++k) T[k] = 0.0;
  const int64_t f0 = int64_t(c) * chunk, f1 = min(f0 + chunk, nf);
  const bool live = int64_t(tb) * kFfvBlock + (tid & ~31) < nb;   // the warp has bound particles
  for (int64_t tile0 = f0; tile0 < f1; tile0 += kFfvBlock) {
    __syncthreads();
    const int64_t j = tile0 + tid;
    if (j < f1) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        sx[tid][d] = xf[d * ldf + j];
        sg[tid][d] = gf[d * ldf + j];
      }
    }
    __syncthreads();
    const int cnt = live ? int(min(int64_t(kFfvBlock), f1 - tile0)) : 0;
    for (int js = 0; js < cnt; ++js) {
      const double dx = sx[js][0] - bx, dy = sx[js][1] - by, dz = sx[js][2] - bz;
      double q;   // 0 at r = 0
      if constexpr (GAUSS) {
        const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        const double u = r2 * ka;
        if (core_is_near(u)) {
          q = core_f1(u, ffv_tab) * (is_zero_f64(r2) ? 0.0 : kb);
        } else {
          const double ri = rsqrt(r2);
          q = ri * ri * ri;
        }
      } else {
        const double rs = rsqrt(fma(dx, dx, fma(dy, dy, fma(dz, dz, ka))));
        const double rs2 = rs * rs, rs3 = rs2 * rs;
        q = coincident_f64(dx, dy, dz) ? 0.0 : fma(kb, rs3 * rs2, rs3);
      }
      const double qx = q * dx, qy = q * dy, qz = q * dz;
      const double fx = sg[js][0], fy = sg[js][1], fz = sg[js][2];
      T[0] = fma(qx, fx, T[0]); T[1] = fma(qx, fy, T[1]); T[2] = fma(qx, fz, T[2]);
      T[3] = fma(qy, fx, T[3]); T[4] = fma(qy, fy, T[4]); T[5] = fma(qy, fz, T[5]);
      T[6] = fma(qz, fx, T[6]); T[7] = fma(qz, fy, T[7]); T[8] = fma(qz, fz, T[8]);
    }
  }
  if (!valid) return;
  if (n_chunk > 1) {
#pragma unroll
    for (int k = 0; k < kFfvNval; ++k) part[(int64_t(c) * kFfvNval + k) * nb + b] = T[k];
    return;
  }
  ffv_finish(T, gb, ldb, b, M, ldm);
}

// Sum of the chunks: kFfvRed bound particles (x) times the nine sums (y) times
// kFfvSegs runs of chunks (z) per block, each run in chunk order, then the runs in
// order.  (32 particles and three runs a block left 14 blocks to sum 469 chunks: 45 µs.)
constexpr int kFfvRed = 8, kFfvSegs = 14;
__global__ void __launch_bounds__(kFfvRed * kFfvNval * kFfvSegs) ffv_reduce_kernel(
    int64_t nb, const double* __restrict__ gb, int64_t ldb, const double* __restrict__ part,
    int n_chunk, double* M, int64_t ldm) {
  __shared__ double sv[kFfvSegs][kFfvNval][kFfvRed];
  const int tx = threadIdx.x, k = threadIdx.y, z = threadIdx.z;
  const int64_t b = int64_t(blockIdx.x) * kFfvRed + tx;
  if (b < nb) {
    const int c0 = int(int64_t(n_chunk) * z / kFfvSegs), c1 = int(int64_t(n_chunk) * (z + 1) / kFfvSegs);
    const double* p = part + int64_t(k) * nb + b;
    const int64_t step = int64_t(kFfvNval) * nb;
    double v = 0.0;
#pragma unroll 8
    for (int c = c0; c < c1; ++c) v += p[c * step];
    sv[z][k][tx] = v;
  }
  __syncthreads();
  if (k == 0 && z == 0 && b < nb) {
    double T[kFfvNval];
#pragma unroll
    for (int i = 0; i < kFfvNval; ++i) {
      T[i] = sv[0][i][tx];
      for (int q = 1; q < kFfvSegs; ++q) T[i] += sv[q][i][tx];
    }
    ffv_finish(T, gb, ldb, b, M, ldm);
  }
}

// Scratch (elements) an FFV launch of nb bound and nf free particles needs.
// Chunks of 64 or more free particles for about 16 CTAs per SM: every CTA costs the
// same, so what the count decides is how even the SMs end (421 bound, 30,011 free:
// 472 CTAs of 256 left a quarter of the last round idle, 1,876 of 64 a twentieth).
size_t ffv_plan(int64_t nb, int64_t nf, int num_sms, int64_t* chunk, int* n_chunk) {
  const int64_t n_tb = ceil_div(std::max<int64_t>(nb, 1), kFfvBlock);
  *chunk = std::max<int64_t>(64, round_up(ceil_div(nf * n_tb, 16 * std::max(num_sms, 1)), 32));
  *n_chunk = int(std::max<int64_t>(1, ceil_div(nf, *chunk)));
  return *n_chunk > 1 ? size_t(*n_chunk) * kFfvNval * size_t(nb) : 0;
}

template <int KERNEL>
cudaError_t ffv_start(int grid, int64_t nb, const double* xb, const double* gb, const double* sb,
                      int64_t ldb, int64_t nf, const double* xf, const double* gf, int64_t ldf,
                      int64_t chunk, int n_tb, double* part, double* M, int64_t ldm, int n_chunk,
                      cudaStream_t st) {
  const size_t smem = KERNEL == VPM_KERNEL_GAUSSIANERF ? sizeof(CoreTable) : 0;
  static PerContext done;
  const cudaError_t e = allow_smem(done, ffv_kernel<KERNEL>, smem);
  if (e != cudaSuccess) return e;
  ffv_kernel<KERNEL><<<grid, kFfvBlock, smem, st>>>(nb, xb, gb, sb, ldb, nf, xf, gf, ldf, chunk,
                                                    n_tb, part, M, ldm, n_chunk);
  return cudaGetLastError();
}

cudaError_t launch_ffv(int kernel, int64_t nb, const double* xb, const double* gb,
                       const double* sb, int64_t ldb, int64_t nf, const double* xf,
                       const double* gf, int64_t ldf, double* part, double* M, int64_t ldm,
                       int num_sms, cudaStream_t st) {
  if (nb <= 0) return cudaSuccess;
  int64_t chunk = 0;
  int n_chunk = 1;
  ffv_plan(nb, nf, num_sms, &chunk, &n_chunk);
  const int n_tb = int(ceil_div(nb, kFfvBlock));
  const int grid = n_tb * n_chunk;
  auto start = kernel == VPM_KERNEL_WINCKELMANS ? ffv_start<VPM_KERNEL_WINCKELMANS>
                                                : ffv_start<VPM_KERNEL_GAUSSIANERF>;
  const cudaError_t e = start(grid, nb, xb, gb, sb, ldb, nf, xf, gf, ldf, chunk, n_tb, part, M, ldm,
                              n_chunk, st);
  if (e != cudaSuccess || n_chunk <= 1) return e;
  ffv_reduce_kernel<<<int(ceil_div(nb, kFfvRed)), dim3(kFfvRed, kFfvNval, kFfvSegs), 0, st>>>(
      nb, gb, ldb, part, n_chunk, M, ldm);
  return cudaGetLastError();
}

}  // namespace vpm
