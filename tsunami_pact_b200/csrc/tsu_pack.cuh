// tsu_pack.cuh -- ASCII -> 2-bit packing (the reference compares raw bytes,
// wfa_gpu.cu:735; here every A/C/G/T-only sequence is packed 32 bases per
// 64-bit word so the extend step compares 16 bases per 32-bit funnel shift).
#pragma once

#include <algorithm>

#include "tsu_common.cuh"

namespace tsu {

// Four ASCII bases (byte i: base i) -> 8 bits (bits 2 i, 2 i + 1); *bad is
// nonzero when one of them is not A, C, G or T.  The 2-bit code of a base is
// (c >> 1) & 3 (A=0, C=1, T=2, G=3), a bijection on "ACGT"; the letter of a
// code b is 0x41 + 2 b, and 15 more for b = 2.  The product moves code i from
// bit 8 i to bit 24 + 2 i; what it adds elsewhere stays below bit 24 or
// leaves the word.
__device__ __forceinline__ uint32_t pack4(uint32_t c, uint32_t* bad) {
  const uint32_t x = (c >> 1) & 0x03030303u;
  const uint32_t two = (x >> 1) & ~x & 0x01010101u;
  *bad |= c ^ (0x41414141u + 2u * x + 15u * two);
  return (x * 0x01041040u) >> 24;
}

// kLanes lanes per sequence, 16 bases (one 32-bit word) per lane: four aligned
// words and the one after them shifted to the sequence's alignment, so a warp
// reads 512 bytes with five load instructions; the first and the last word of
// a sequence, whose aligned words reach outside it, are read by bytes (all 16
// in flight at once).  What bounds it is DRAM for long sequences, and the chain
// of loads per sequence (offsets, bytes) for short ones, several of which share
// a warp (launch_pack).  Measured on one B200, 400,000 sequences of 1 kbp: a
// byte per lane and three ballots per 32 bases took 1.65 ms (0.24 TB/s), this
// 0.25 with a warp each and 0.15 with 4 lanes each.  kRev packs each sequence reversed (base p of the packed form is byte
// len - 1 - p), for the reverse passes of the bidirectional mode.
template <bool kRev = false, int kLanes = 32>
static __global__ void pack_kernel(SeqView sv, PackView pk) {
  constexpr int kSeqs = 32 / kLanes;  // sequences per warp
  const int lane = threadIdx.x & 31, gl = lane % kLanes;
  const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * kSeqs;
  const int64_t nseq = 2 * sv.n;
  for (int64_t j0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kSeqs; j0 < nseq; j0 += step) {
    const int64_t j = j0 + lane / kLanes;
    uint32_t bad = 0;
    if (j < nseq) {
      const bool is_pat = j < sv.n;
      const int64_t i = is_pat ? j : j - sv.n;
      const uint8_t* src = is_pat ? sv.pat + sv.pat_off[i] : sv.txt + sv.txt_off[i];
      const int len = is_pat ? sv.pat_len[i] : sv.txt_len[i];
      uint32_t* dst = reinterpret_cast<uint32_t*>(pk.words + pk.woff[j]);
      const int nw = 2 * (int)packed_words(len);  // the data words, then zero padding
      for (int w = gl; w < nw; w += kLanes) {
        const int p = 16 * w;
        uint32_t word = 0;
        const int from = kRev ? len - 16 - p : p;  // first of the 16 bytes, in memory order
        if (from >= 3 && from + 19 <= len) {
          const uintptr_t a = reinterpret_cast<uintptr_t>(src + from);
          const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~(uintptr_t)3);
          const uint32_t sh = (uint32_t)(a & 3) * 8;
          uint32_t v[5];
#pragma unroll
          for (int t = 0; t < 5; ++t) v[t] = t < 4 || sh ? __ldg(q + t) : 0u;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            uint32_t c = __funnelshift_r(v[t], v[t + 1], sh);
            if (kRev) c = (c >> 24) | ((c >> 8) & 0xff00u) | ((c << 8) & 0xff0000u) | (c << 24);
            word |= pack4(c, &bad) << (kRev ? 24 - 8 * t : 8 * t);
          }
        } else if (p < len) {
          uint32_t c[16];
#pragma unroll
          for (int t = 0; t < 16; ++t) c[t] = p + t < len ? src[kRev ? len - 1 - p - t : p + t] : 0x41u;
#pragma unroll
          for (int t = 0; t < 4; ++t)
            word |= pack4(c[4 * t] | (c[4 * t + 1] << 8) | (c[4 * t + 2] << 16) | (c[4 * t + 3] << 24), &bad) << (8 * t);
        }
        dst[w] = word;
      }
    }
    const uint32_t any = __ballot_sync(0xffffffffu, bad != 0) >> (lane - gl);
    if (gl == 0 && j < nseq) pk.nonacgt[j] = (kLanes == 32 ? any : any & ((1u << (kLanes & 31)) - 1)) ? 1 : 0;
  }
}

// Lanes per sequence: as few as still give every thread of the GPU a sequence's
// word to pack (2,048 threads per SM), since a sequence costs its group the same
// chain of loads however many lanes it has; but no more than 32 words a lane, so
// that one long sequence does not hold up the others of its warp.  Measured on
// one B200 at 4, 8, 16 and 32 lanes, us (before: one warp each, 32-bit words /
// a byte per lane): 2,000,000 x 36 bp 124, 214, 406, 717 (1,258 / 731);
// 800,000 x 150 bp 94, 139, 177, 306 (514 / 600); 400,000 x 1 kbp 146, 155, 182,
// 247 (385 / 1,654).
inline int pack_lanes(int64_t nseq, int32_t maxlen, int sms) {
  int lanes = 4;
  while (lanes < 32 && (nseq * lanes < (int64_t)sms * 2048 || maxlen > 512 * lanes)) lanes *= 2;
  return lanes;
}

#ifndef TSU_WARP_EMU
// The pack kernel over sequences of at most maxlen bases.
template <bool kRev>
inline void launch_pack(int32_t maxlen, int sms, cudaStream_t st, const SeqView& sv, const PackView& pk) {
  const int lanes = pack_lanes(2 * sv.n, maxlen, sms);
  const int blocks = (int)std::min<int64_t>((2 * sv.n * lanes + 255) / 256, (int64_t)sms * 16);
  switch (lanes) {
    case 4: pack_kernel<kRev, 4><<<blocks, 256, 0, st>>>(sv, pk); break;
    case 8: pack_kernel<kRev, 8><<<blocks, 256, 0, st>>>(sv, pk); break;
    case 16: pack_kernel<kRev, 16><<<blocks, 256, 0, st>>>(sv, pk); break;
    default: pack_kernel<kRev><<<blocks, 256, 0, st>>>(sv, pk); break;
  }
}
#endif

// words per sequence: packed_words (data words, padding, even count)
static __global__ void word_count_kernel(int64_t n, const int32_t* __restrict__ pat_len, const int32_t* __restrict__ txt_len,
                                  int64_t* __restrict__ words) {
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < 2 * n; j += (int64_t)gridDim.x * blockDim.x) {
    const int len = j < n ? pat_len[j] : txt_len[j - n];
    words[j] = packed_words(len);
  }
}

}  // namespace tsu
