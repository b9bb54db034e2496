// tsu_dual.cu -- the dual gap-affine align_kernel instantiations
// (align_kernel<..., kModelDual>), in their own translation unit so they
// compile beside the one-piece kernels of tsu_engine.cu.
#include "tsu_launch.cuh"

namespace tsu {

cudaError_t align_occupancy_dual(bool cigar, int mode, int gw, int threads, size_t smem, int optin, int* occ, int flag) {
  return launch_detail::occupancy<kModelDual>(cigar, mode, gw, threads, smem, optin, occ, flag);
}

void launch_align_dual(bool cigar, int mode, int gw, int blocks, int threads, size_t smem, cudaStream_t st,
                       const AlignArgs& a, int flag) {
  launch_detail::launch<kModelDual>(cigar, mode, gw, blocks, threads, smem, st, a, flag);
}

cudaError_t probe_occupancy_dual(bool wide, bool deep, int threads, size_t smem, int optin, int* occ) {
  return launch_detail::probe_occupancy<kModelDual>(wide, deep, threads, smem, optin, occ);
}

void launch_probe_dual(bool wide, int blocks, int threads, size_t smem, cudaStream_t st, const ProbeArgs& a) {
  launch_detail::probe<kModelDual>(wide, blocks, threads, smem, st, a);
}

void launch_wide_dual(bool cigar, int blocks, int cluster, size_t smem, cudaStream_t st, const AlignArgs& a) {
  launch_detail::wide<kModelDual>(cigar, blocks, cluster, smem, st, a);
}

}  // namespace tsu
