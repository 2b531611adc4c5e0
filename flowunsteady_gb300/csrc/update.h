// update.h — O(N) kernels of a time step (launchers in update.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace vpm {

// Device status word bits (OR-ed by kernels, read by the host after a call).
enum : int { STATUS_NONFINITE = 1, STATUS_TIMEOUT = 2 };

struct SfsParams {
  double alpha, rlxf, minC, maxC, zeta0;
  double inv_zeta0;   // 1/ζ(0) (FP64 divides are scarce on the FP64 pipe)
  int transposed;
  int force_positive;
  int analytic;   // Jt, Et hold 1: DJ, DE (analytic α-derivatives), 2: the differences
};

struct UpdateParams {
  double a, b, dt;          // low-storage RK coefficients of the stage, time step
  double uinf0, uinf1, uinf2;
  double zs;                // (f+g)/(1+3f)
  double ze;                // f/(1+3f)
  double zeta0;             // ζ(0) of the kernel
  double inv_zeta0;         // 1/ζ(0)
  double nu;                // core spreading viscosity (0 = off)
  int transposed;
  int sfs;                  // E_str / C_d terms on
  int clip_backscatter;
};

// Diagnostic reduction slots.
enum {
  DS_ENS = 0, DS_IX, DS_IY, DS_IZ, DS_GX, DS_GY, DS_GZ, DS_SIG, DS_NONFIN,
  DS_CCNT, DS_CSUM, DS_CSUM2, DS_CZERO, DS_CMIN, DS_CMAX, DS_CSUM3, DS_CSUM4, kDiagSlots
};
constexpr int kRedBlocks = 304;   // 2 x 152 SMs

// What happens to the particles between two pair passes (update_dev.cuh), in this
// order.  Js and Eo: the J that the stretching and E_str take, and where E_str goes
// (J and E, or at the test-filter level Jt and Et).
enum : int {
  POST_STRETCH = 1,      // rows V 0..2 = S(Js, Γ)
  POST_STRETCH_D = 2,    // rows V 3..5 = S(Jt, Γ)
  POST_ZETA_REC = 4,     // packed ζ records at rec_scale (with w_q if POST_STRETCH_D)
  POST_ESTR = 8,         // Eo from raw and Js
  POST_ESTR_D = 16,      // Et from raw, Js and Jt
  POST_CONSTANT = 32,    // C_d = cd
  POST_DYNAMIC = 64,     // C_d from J, Jt, E, Et
  POST_UPDATE = 128,     // the Runge-Kutta stage
  POST_UJ_REC = 256      // packed U/J records at rec_scale
};
struct PostArgs {
  int flags = 0, transposed = 0;
  int64_t n = 0, nv = 0, ld = 0;    // C_d and the update visit [0, nv) where stat is 0
  const uint8_t* stat = nullptr;
  double *X = nullptr, *G = nullptr, *S = nullptr, *C = nullptr, *Q = nullptr, *V = nullptr;
  const double *U = nullptr, *J = nullptr, *Jt = nullptr, *E = nullptr, *raw = nullptr;
  const double* Js = nullptr;
  double *Eo = nullptr, *Et = nullptr;
  double cd = 0.0;
  SfsParams sfs;
  UpdateParams up;
  float4* rec = nullptr;
  double rec_scale = 1.0;
  int* status = nullptr;
};
constexpr int kPostThreads = 128;
cudaError_t launch_post(int kernel, const PostArgs& p, cudaStream_t st);
// The per-particle kernels below visit particles [0, nv) and skip those whose
// static flag stat[i] is nonzero (stat may be null: no static particles in range).
cudaError_t launch_sfs_clip(int64_t nv, const uint8_t* stat, int64_t ld, const double* G,
                            const double* E, double* C, cudaStream_t st);
cudaError_t launch_relax(int64_t nv, const uint8_t* stat, int64_t ld, const double* J, double* G,
                         double r, cudaStream_t st);
cudaError_t launch_zero(double* p, int64_t n, cudaStream_t st);
// partial: kRedBlocks*kDiagSlots doubles; out: kDiagSlots doubles (device).
cudaError_t launch_diagnostics(int64_t n, int64_t nf, const uint8_t* stat, int64_t ld,
                               const double* X, const double* G, const double* S, const double* C,
                               const double* raw, double zeta0, double* partial, double* out,
                               cudaStream_t st);
cudaError_t launch_centroid(int64_t i0, int64_t i1, int64_t ld, const double* X, const double* G,
                            double* partial, double* out, cudaStream_t st);

}  // namespace vpm
