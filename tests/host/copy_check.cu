// The pieces of a mapped copy (CopySplit) cover every byte once, for every
// alignment of the two addresses: the words its two word loops copy (widths 16
// and 4), and the single bytes from words * width on.
#include <cstdio>

#include "../../mpsft_gb300/csrc/common.cuh"

int main() {
  long checked = 0, bad = 0;
  for (uintptr_t src = 0; src < 16; ++src) {
    for (uintptr_t dst = 0; dst < 16; ++dst) {
      for (size_t bytes = 0; bytes <= 100; ++bytes) {
        const mpsft::CopyWords cw = mpsft::CopySplit(src | dst, bytes);
        const bool loop = cw.width == 16 || cw.width == 4;
        const size_t by_words = loop ? cw.words * cw.width : 0;
        const size_t first_single = cw.words * cw.width;
        const bool aligned = !loop || ((src | dst) % cw.width) == 0;
        if (by_words != first_single || first_single > bytes || !aligned) ++bad;
        ++checked;
      }
    }
  }
  std::printf("copy checked %ld mismatches %ld\n", checked, bad);
  return bad != 0;
}
