// tsu_linear.cu -- the gap-linear align_kernel instantiations
// (align_kernel<..., kModelLinear>), in their own translation unit so they
// compile beside the gap-affine kernels of tsu_engine.cu (edit and indel
// distance are gap-linear penalties).
#include "tsu_launch.cuh"

namespace tsu {

cudaError_t align_occupancy_linear(bool cigar, int mode, int gw, int threads, size_t smem, int optin, int* occ, int flag) {
  return launch_detail::occupancy<kModelLinear>(cigar, mode, gw, threads, smem, optin, occ, flag);
}

void launch_align_linear(bool cigar, int mode, int gw, int blocks, int threads, size_t smem, cudaStream_t st,
                         const AlignArgs& a, int flag) {
  launch_detail::launch<kModelLinear>(cigar, mode, gw, blocks, threads, smem, st, a, flag);
}

cudaError_t probe_occupancy_linear(bool wide, bool deep, int threads, size_t smem, int optin, int* occ) {
  return launch_detail::probe_occupancy<kModelLinear>(wide, deep, threads, smem, optin, occ);
}

void launch_probe_linear(bool wide, int blocks, int threads, size_t smem, cudaStream_t st, const ProbeArgs& a) {
  launch_detail::probe<kModelLinear>(wide, blocks, threads, smem, st, a);
}

void launch_wide_linear(bool cigar, int blocks, int cluster, size_t smem, cudaStream_t st, const AlignArgs& a) {
  launch_detail::wide<kModelLinear>(cigar, blocks, cluster, smem, st, a);
}

}  // namespace tsu
