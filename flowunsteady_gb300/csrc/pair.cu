// pair.cu — instantiates the U/∇U and ζ pair passes (the kernel template is in
// pair_kernel.cuh) and dispatches every pass; the α-derivative passes are
// compiled in pair_d.cu.
#include "pair_kernel.cuh"

namespace vpm {

bool pair_shape_supported(int precision, Shape s) {
  if (precision == VPM_PREC_FP64) return s.block == 128 && s.tpt == 1;
  return (s.block == 128 && (s.tpt == 2 || s.tpt == 4)) || (s.block == 256 && s.tpt == 2);
}

int pair_ctas_per_sm(int pass, int kernel, int precision, Shape s) {
  if (pass == PASS_UJ) return ctas_per_sm<PASS_UJ>(kernel, precision, s);
  if (pass == PASS_ZETA) return ctas_per_sm<PASS_ZETA>(kernel, precision, s);
  return pair_ctas_per_sm_d(pass, kernel, precision, s);
}

int pair_max_active_clusters(int pass, int kernel, int precision, Shape s, int cluster) {
  if (pass == PASS_UJ) return max_active_clusters<PASS_UJ>(kernel, precision, s, cluster);
  if (pass == PASS_ZETA) return max_active_clusters<PASS_ZETA>(kernel, precision, s, cluster);
  return pair_max_active_clusters_d(pass, kernel, precision, s, cluster);
}

cudaError_t launch_pair(int pass, int kernel, int precision, Shape s, const PairArgs& a, int grid,
                        cudaStream_t st) {
  if (pass == PASS_UJ) return launch<PASS_UJ>(kernel, precision, s, a, grid, st);
  if (pass == PASS_ZETA) return launch<PASS_ZETA>(kernel, precision, s, a, grid, st);
  return launch_pair_d(pass, kernel, precision, s, a, grid, st);
}

template <int KERNEL>
__global__ void __launch_bounds__(kPostThreads) pack_sources_kernel(
    int64_t n, const double* __restrict__ X, const double* __restrict__ G,
    const double* __restrict__ S, int64_t ld, double scale, float4* __restrict__ rec) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) uj_record_at<KERNEL>(i, ld, X, G, S, scale, rec);
}

template <int KERNEL, bool D>
__global__ void __launch_bounds__(kPostThreads) pack_zeta_sources_kernel(
    int64_t n, const double* __restrict__ X, const double* __restrict__ G,
    const double* __restrict__ S, const double* __restrict__ V, const double* __restrict__ W,
    int64_t ld, double scale, float4* __restrict__ rec) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) zeta_record_at<KERNEL>(i, ld, D, X, G, S, V, W, scale, rec);
}

cudaError_t launch_pack_zeta_sources(int kernel, bool d, int64_t n, const double* X,
                                     const double* G, const double* S, const double* V,
                                     const double* W, int64_t ld, double scale, float4* rec,
                                     cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int grid = int((n + kPostThreads - 1) / kPostThreads);
  auto go = [&](auto kern) { kern<<<grid, kPostThreads, 0, st>>>(n, X, G, S, V, W, ld, scale, rec); };
  if (kernel == VPM_KERNEL_WINCKELMANS) {
    if (d) go(pack_zeta_sources_kernel<VPM_KERNEL_WINCKELMANS, true>);
    else go(pack_zeta_sources_kernel<VPM_KERNEL_WINCKELMANS, false>);
  } else {
    if (d) go(pack_zeta_sources_kernel<VPM_KERNEL_GAUSSIANERF, true>);
    else go(pack_zeta_sources_kernel<VPM_KERNEL_GAUSSIANERF, false>);
  }
  return cudaGetLastError();
}

cudaError_t launch_pack_sources(int kernel, int64_t n, const double* X, const double* G,
                                const double* S, int64_t ld, double scale, float4* rec,
                                cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int grid = int((n + kPostThreads - 1) / kPostThreads);
  if (kernel == VPM_KERNEL_WINCKELMANS)
    pack_sources_kernel<VPM_KERNEL_WINCKELMANS><<<grid, kPostThreads, 0, st>>>(n, X, G, S, ld, scale, rec);
  else
    pack_sources_kernel<VPM_KERNEL_GAUSSIANERF><<<grid, kPostThreads, 0, st>>>(n, X, G, S, ld, scale, rec);
  return cudaGetLastError();
}

cudaError_t launch_reduce(int pass, int kernel, int precision, const double* part, int64_t ldp,
                          const int64_t* foff, const int32_t* fchunks, int nfields,
                          int scalar_chunks, int segs, int64_t t_begin, int64_t t_end, double* u,
                          double* j, double* dj, int64_t ldo, const PostArgs* post,
                          cudaStream_t st) {
  if (pass == PASS_UJ)
    return reduce<PASS_UJ>(kernel, precision, part, ldp, foff, fchunks, nfields, scalar_chunks, segs, t_begin,
                           t_end, u, j, dj, ldo, post, st);
  if (pass == PASS_ZETA)
    return reduce<PASS_ZETA>(kernel, precision, part, ldp, foff, fchunks, nfields, scalar_chunks, segs, t_begin,
                             t_end, u, j, dj, ldo, post, st);
  return launch_reduce_d(pass, kernel, precision, part, ldp, foff, fchunks, nfields, scalar_chunks, segs, t_begin,
                         t_end, u, j, dj, ldo, post, st);
}

}  // namespace vpm
