// tsu_extend.cuh -- the extend step: longest common prefix along a diagonal.
//
// Replaces the reference's count_chars (wfa_gpu.cu:724-752: a 32-byte
// window reduced through shared memory with 5 barriers, then a byte-serial
// tail on lane 0, wfa_gpu.cu:266-281).  Here each lane extends its own
// diagonal: 16 bases of pattern and text are cut out of the 2-bit words with
// one funnel shift each, XORed, and the first set bit gives the first
// mismatch.  Reads stay inside the sequence plus its padding word because
// the window start is always < the sequence length.
#pragma once

#include "tsu_common.cuh"

namespace tsu {

// Sequence word sources: shared memory (staged copy) or global memory.
struct SharedSeq {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator[](int i) const { return p[i]; }
};
struct GlobalSeq {
  const uint32_t* __restrict__ p;
  __device__ __forceinline__ uint32_t operator[](int i) const { return __ldg(p + i); }
};
// Global-ring groups: the pair's words staged in shared memory, or (pairs
// too long to stage) the packed words in global memory, through one generic
// pointer.
struct AnySeq {
  const uint32_t* p;
  __device__ __forceinline__ uint32_t operator[](int i) const { return p[i]; }
};

template <class S>
__device__ __forceinline__ uint32_t win16(const S& w, int pos) {
  const int i = pos >> 4;
  return __funnelshift_r(w[i], w[i + 1], (pos & 15) << 1);
}

// LCP of pattern[v..] and text[h..], at most rem characters.
template <class S>
__device__ __forceinline__ int lcp16(const S& pw, int v, const S& tw, int h, int rem) {
  int l = 0;
  while (l < rem) {
    const uint32_t d = win16(pw, v + l) ^ win16(tw, h + l);
    if (d) {
      l += (__ffs(d) - 1) >> 1;
      break;
    }
    l += 16;
  }
  return l < rem ? l : rem;
}

// Byte path for pairs with bytes outside ACGT: LCP of p[v..] and t[h..], at
// most rem characters, 8 per step; reads only the rem bytes compared.  (The
// windows were once built as 64-bit words of bytes guarded by the sequences'
// lengths.  Compiled into the two-piece CIGAR kernels of 2 to 16 warps, that
// form took the second window for different when it held the last 3 bases of
// both sequences, one mismatch too many, and otherwise changed from run to
// run; the same source was right in every other kernel and on the CPU.)
__device__ __forceinline__ int lcp8(const uint8_t* __restrict__ p, int v, const uint8_t* __restrict__ t, int h, int rem) {
  int l = 0;
  while (l < rem) {
    const int c = rem - l;
    int first = 8;  // the first of 8 that differ
#pragma unroll
    for (int i = 7; i >= 0; --i)
      if (i < c && p[v + l + i] != t[h + l + i]) first = i;
    if (first < 8) return l + first;
    l += 8;
  }
  return rem;
}

}  // namespace tsu
