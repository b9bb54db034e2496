// tsu_launch.cuh -- occupancy queries and launches of the align_kernel
// instantiations: CIGAR or score only, shared or global wavefront ring,
// 1/2/4/8/16/32 warps per pair, penalty model (gap-affine, dual gap-affine,
// gap-linear).  Each model's kernels are instantiated in a translation unit
// of their own (tsu_engine.cu, tsu_dual.cu, tsu_linear.cu), compiled in
// parallel.  Each kernel's dynamic
// shared memory limit is set to the device maximum once per device (always
// the same value, so contexts planning on several host threads cannot lower
// it under another's launch).
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "tsu_align.cuh"

namespace tsu {

// The dual gap-affine kernels (tsu_dual.cu) and the gap-linear ones
// (tsu_linear.cu).
// flag: 0, or a variant: kLowMemFlag (CIGARs; cigar is then ignored),
// kBoundFlag (shared ring, pairs with score bounds), kDeepFlag (shared ring,
// with or without kBoundFlag), kSingleFlag (shared ring, one diagonal per
// thread).
cudaError_t align_occupancy_dual(bool cigar, int mode, int gw, int threads, size_t smem, int optin, int* occ,
                                 int flag);
void launch_align_dual(bool cigar, int mode, int gw, int blocks, int threads, size_t smem, cudaStream_t st,
                       const AlignArgs& a, int flag);
cudaError_t align_occupancy_linear(bool cigar, int mode, int gw, int threads, size_t smem, int optin, int* occ,
                                   int flag);
void launch_align_linear(bool cigar, int mode, int gw, int blocks, int threads, size_t smem, cudaStream_t st,
                         const AlignArgs& a, int flag);

// The bound probe of each model (probe_kernel).
// wide: of pairs of any length (wide_probe_kernel).
cudaError_t probe_occupancy_dual(bool wide, bool deep, int threads, size_t smem, int optin, int* occ);
void launch_probe_dual(bool wide, int blocks, int threads, size_t smem, cudaStream_t st, const ProbeArgs& a);
cudaError_t probe_occupancy_linear(bool wide, bool deep, int threads, size_t smem, int optin, int* occ);
void launch_probe_linear(bool wide, int blocks, int threads, size_t smem, cudaStream_t st, const ProbeArgs& a);
// The wide kernel of each model (wide_kernel; one block of kWideThreads per
// pair, or `cluster` of them; a.wide_cell bytes per ring cell).
void launch_wide_dual(bool cigar, int blocks, int cluster, size_t smem, cudaStream_t st, const AlignArgs& a);
void launch_wide_linear(bool cigar, int blocks, int cluster, size_t smem, cudaStream_t st, const AlignArgs& a);

namespace launch_detail {

template <int kModel>
cudaError_t probe_occupancy(bool wide, bool deep, int threads, size_t smem, int optin, int* occ) {
  const void* const f = wide   ? (const void*)wide_probe_kernel<kModel>
                        : deep ? (const void*)probe_kernel<kModel | kDeepFlag>
                               : (const void*)probe_kernel<kModel>;
  const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, f, threads, smem);
}

template <int kModel>
void probe(bool wide, int blocks, int threads, size_t smem, cudaStream_t st, const ProbeArgs& a) {
  if (wide)
    wide_probe_kernel<kModel><<<blocks, threads, smem, st>>>(a);
  else if (a.pen.rm > 64)
    probe_kernel<kModel | kDeepFlag><<<blocks, threads, smem, st>>>(a);
  else
    probe_kernel<kModel><<<blocks, threads, smem, st>>>(a);
}

template <bool kCigar, int kModel, typename ST>
void wide_one(int blocks, int cluster, size_t smem, cudaStream_t st, const AlignArgs& a) {
  if (cluster <= 1) {
    wide_kernel<kCigar, kModel, ST><<<blocks, kWideThreads, smem, st>>>(a);
    return;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(kWideThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, wide_kernel<kCigar, kModel, ST, true>, a);
}

// blocks: of all clusters together
template <int kModel>
void wide(bool cigar, int blocks, int cluster, size_t smem, cudaStream_t st, const AlignArgs& a) {
  if (a.wide_cell == 2)
    cigar ? wide_one<true, kModel, uint16_t>(blocks, cluster, smem, st, a)
          : wide_one<false, kModel, uint16_t>(blocks, cluster, smem, st, a);
  else
    cigar ? wide_one<true, kModel, uint32_t>(blocks, cluster, smem, st, a)
          : wide_one<false, kModel, uint32_t>(blocks, cluster, smem, st, a);
}

template <bool kCigar, int kMode, int GW, int kModel>
cudaError_t occ_one(int threads, size_t smem, int optin, int* occ) {
  static std::atomic<uint64_t> limit_set{0};  // bit d: set on device d
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const uint64_t bit = dev < 64 ? (1ull << dev) : 0;
  if (!bit || !(limit_set.load() & bit)) {
    e = cudaFuncSetAttribute(align_kernel<kCigar, kMode, GW, kModel>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin);
    if (e != cudaSuccess) return e;
    limit_set.fetch_or(bit);
  }
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, align_kernel<kCigar, kMode, GW, kModel>, threads, smem);
}

template <bool kCigar, int kMode, int kModel>
cudaError_t occ_gw(int gw, int threads, size_t smem, int optin, int* occ) {
  switch (gw) {
    case 1: return occ_one<kCigar, kMode, 1, kModel>(threads, smem, optin, occ);
    case 2: return occ_one<kCigar, kMode, 2, kModel>(threads, smem, optin, occ);
    case 4: return occ_one<kCigar, kMode, 4, kModel>(threads, smem, optin, occ);
    case 8: return occ_one<kCigar, kMode, 8, kModel>(threads, smem, optin, occ);
    case 16: return occ_one<kCigar, kMode, 16, kModel>(threads, smem, optin, occ);
    case 32:
      if constexpr (!(kModel & kBoundFlag)) return occ_one<kCigar, kMode, 32, kModel>(threads, smem, optin, occ);
      return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
  }
}

// f(flag as a compile-time constant) for the shared ring's variants.
template <class F>
auto with_flag(int flag, F&& f) {
  switch (flag) {
    case kBoundFlag: return f(std::integral_constant<int, kBoundFlag>{});
    case kBoundFlag | kDeepFlag: return f(std::integral_constant<int, kBoundFlag | kDeepFlag>{});
    case kDeepFlag: return f(std::integral_constant<int, kDeepFlag>{});
    case kSingleFlag: return f(std::integral_constant<int, kSingleFlag>{});
    default: return f(std::integral_constant<int, 0>{});
  }
}

template <int kModel>
cudaError_t occupancy(bool cigar, int mode, int gw, int threads, size_t smem, int optin, int* occ, int flag) {
  if (flag == kLowMemFlag)
    return mode == kModeShared ? occ_gw<true, kModeShared, kModel | kLowMemFlag>(gw, threads, smem, optin, occ)
                               : occ_gw<true, kModeGlobal, kModel | kLowMemFlag>(gw, threads, smem, optin, occ);
  if (mode == kModeGlobal)
    return cigar ? occ_gw<true, kModeGlobal, kModel>(gw, threads, smem, optin, occ)
                 : occ_gw<false, kModeGlobal, kModel>(gw, threads, smem, optin, occ);
  return with_flag(flag, [&](auto f) {
    constexpr int kM = kModel | decltype(f)::value;
    return cigar ? occ_gw<true, kModeShared, kM>(gw, threads, smem, optin, occ)
                 : occ_gw<false, kModeShared, kM>(gw, threads, smem, optin, occ);
  });
}

template <bool kCigar, int kMode, int kModel>
void launch_gw(int gw, int blocks, int threads, size_t smem, cudaStream_t st, const AlignArgs& a) {
  switch (gw) {
    case 1: align_kernel<kCigar, kMode, 1, kModel><<<blocks, threads, smem, st>>>(a); break;
    case 2: align_kernel<kCigar, kMode, 2, kModel><<<blocks, threads, smem, st>>>(a); break;
    case 4: align_kernel<kCigar, kMode, 4, kModel><<<blocks, threads, smem, st>>>(a); break;
    case 8: align_kernel<kCigar, kMode, 8, kModel><<<blocks, threads, smem, st>>>(a); break;
    case 16: align_kernel<kCigar, kMode, 16, kModel><<<blocks, threads, smem, st>>>(a); break;
    case 32:
      if constexpr (!(kModel & kBoundFlag)) align_kernel<kCigar, kMode, 32, kModel><<<blocks, threads, smem, st>>>(a);
      break;
    default: break;
  }
}

template <int kModel>
void launch(bool cigar, int mode, int gw, int blocks, int threads, size_t smem, cudaStream_t st, const AlignArgs& a,
            int flag) {
  if (flag == kLowMemFlag) {
    if (mode == kModeShared)
      launch_gw<true, kModeShared, kModel | kLowMemFlag>(gw, blocks, threads, smem, st, a);
    else
      launch_gw<true, kModeGlobal, kModel | kLowMemFlag>(gw, blocks, threads, smem, st, a);
  } else if (mode == kModeGlobal) {
    if (cigar)
      launch_gw<true, kModeGlobal, kModel>(gw, blocks, threads, smem, st, a);
    else
      launch_gw<false, kModeGlobal, kModel>(gw, blocks, threads, smem, st, a);
  } else {
    with_flag(flag, [&](auto f) {
      constexpr int kM = kModel | decltype(f)::value;
      if (cigar)
        launch_gw<true, kModeShared, kM>(gw, blocks, threads, smem, st, a);
      else
        launch_gw<false, kModeShared, kM>(gw, blocks, threads, smem, st, a);
    });
  }
}

}  // namespace launch_detail
}  // namespace tsu
