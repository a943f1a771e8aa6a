// conv_first_words.h -- pieces of an image row that may start and end anywhere, by aligned 32-bit loads, for the row
// kernel of the first layer.  `end` is the address behind the tensor: no load goes past it (near it, single halfs or bytes
// are read).  A tensor starts on a 16-byte boundary, so the part of a word before a row's start lies inside it.
// Mem does the loads: word(address), half(address), byte(address).
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define AIG_ROW_FN __device__ __forceinline__
#else
#define AIG_ROW_FN inline
#endif

// the 32 bits that start `bits` (0, 8, 16 or 24) above bit 0 of the pair (hi, lo)
AIG_ROW_FN uint32_t row_shift(uint32_t lo, uint32_t hi, int bits) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, bits);
#else
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> bits);
#endif
}

// Eight halves from `src` on in each of three planes (`plane` bytes apart), `n` (at least one) of them in the row, zero
// beyond.  One test for the three: with one per plane between the loads, 19 frames of 107x189 took 99.6 us instead of 96.3.
template <class Mem>
AIG_ROW_FN void row_halfs8x3(uintptr_t src, size_t plane, int n, uintptr_t end, const Mem& mem, uint32_t (&out)[3][4]) {
  const bool inside = src + 2 * plane + 20 <= end;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const uintptr_t at = src + c * plane, w = at & ~(uintptr_t)3;
    const int odd = (int)(at >> 1) & 1;
    uint32_t v[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const bool needed = 2 * k - odd < n && (k < 4 || odd);
      v[k] = !needed ? 0u : inside || w + 4 * k + 4 <= end ? mem.word(w + 4 * k) : mem.half(w + 4 * k);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      out[c][k] = odd ? row_shift(v[k], v[k + 1], 16) : v[k];
      if (2 * k >= n) out[c][k] = 0u;
      else if (2 * k + 1 >= n) out[c][k] &= 0xFFFFu;
    }
  }
}

// four bytes likewise
template <class Mem>
AIG_ROW_FN void row_bytes4x3(uintptr_t src, size_t plane, int n, uintptr_t end, const Mem& mem, uint32_t (&out)[3]) {
  if (src + 2 * plane + 8 <= end) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const uintptr_t at = src + c * plane, w = at & ~(uintptr_t)3;
      const int off = (int)(at & 3);
      const uint32_t v = row_shift(mem.word(w), off + n > 4 ? mem.word(w + 4) : 0u, off * 8);
      out[c] = n < 4 ? v & ((1u << (8 * n)) - 1u) : v;
    }
  } else {
    for (int c = 0; c < 3; ++c) {
      out[c] = 0u;
      for (int k = 0; k < 4 && k < n; ++k) out[c] |= mem.byte(src + c * plane + k) << (8 * k);
    }
  }
}
