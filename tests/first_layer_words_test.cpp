// first_layer_words_test.cpp -- the row pieces of conv_first_words.h over every start, length and distance to the end of a
// tensor: the values, and that no load leaves the tensor.  Built and run by test_first_layer_words_cpu.py.
#include <stdio.h>
#include <string.h>

#include "conv_first_words.h"

namespace {

struct Checked {   // loads that must lie in [base, base + bytes), aligned
  const unsigned char* base;
  size_t bytes;
  mutable int bad = 0;
  template <class T>
  uint32_t get(uintptr_t a) const {
    const size_t at = a - reinterpret_cast<uintptr_t>(base);
    if (a < reinterpret_cast<uintptr_t>(base) || at + sizeof(T) > bytes || a % sizeof(T) != 0) {
      ++bad;
      return 0xA5A5A5A5u;
    }
    T v;
    memcpy(&v, base + at, sizeof(T));
    return v;
  }
  uint32_t word(uintptr_t a) const { return get<uint32_t>(a); }
  uint32_t half(uintptr_t a) const { return get<uint16_t>(a); }
  uint32_t byte(uintptr_t a) const { return get<uint8_t>(a); }
};

}  // namespace

int main() {
  alignas(16) unsigned char mem[3 * 2 * 40];
  for (int i = 0; i < (int)sizeof(mem); ++i) mem[i] = (unsigned char)(37 * i + 11 + i / 64);
  const uintptr_t base = reinterpret_cast<uintptr_t>(mem);
  int failed = 0;
  // planes of `total` elements, the last one's end the tensor's end
  for (int total = 1; total <= 40; ++total)
    for (int src = 0; src < total; ++src)
      for (int n = 1; n <= total - src; ++n) {
        Checked b{mem, (size_t)3 * total}, h{mem, (size_t)6 * total};
        uint32_t bytes[3], halves[3][4], want_b[3] = {0, 0, 0}, want_h[3][4] = {};
        for (int c = 0; c < 3; ++c) {
          for (int k = 0; k < 4 && k < n; ++k) want_b[c] |= (uint32_t)mem[c * total + src + k] << (8 * k);
          for (int k = 0; k < 8 && k < n; ++k) {
            const unsigned char* at = mem + 2 * (c * total + src + k);
            want_h[c][k / 2] |= (uint32_t)(at[0] | at[1] << 8) << (16 * (k % 2));
          }
        }
        row_bytes4x3(base + src, (size_t)total, n, base + 3 * total, b, bytes);
        row_halfs8x3(base + 2 * src, (size_t)2 * total, n, base + 6 * total, h, halves);
        if (b.bad || memcmp(bytes, want_b, sizeof(bytes)) != 0) failed += printf("FAILED: bytes: %d of %d, %d in the row, %d loads outside\n", src, total, n, b.bad) > 0;
        if (h.bad || memcmp(halves, want_h, sizeof(halves)) != 0) failed += printf("FAILED: halves: %d of %d, %d in the row, %d loads outside\n", src, total, n, h.bad) > 0;
      }
  if (failed == 0) printf("all as expected\n");
  return failed ? 1 : 0;
}
