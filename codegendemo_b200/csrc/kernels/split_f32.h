// Arguments of the kernel that splits the operands of an fp32 product (kcg_f32split.cu), and where the parts lie in a
// launch's workspace. Plain C++, shared by the kernel and the launcher.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace kcg {

struct SplitF32Args {
  const float *A, *B;  // M x K and K x N, rows of lda and ldb values; all multiples of four
  int64_t lda, ldb;
  int M, N, K;
  uint8_t *parts_a, *parts_b;
  float *scale_a, *scale_b;      // [64 values of K][scale_lda rows], [64 values of K][scale_ldb x 64 columns]
  float* columns;                // what a column of the product is multiplied by at the end
  int scale_lda, scale_ldb;
  unsigned int* words;           // words[0] becomes 1 where a value does not split
};

// Byte offsets of the five arrays behind `base`, and the end. Rows and columns of the exponents are padded to whole tiles:
// the product reads those of rows and columns past the edge (and multiplies zeros by them).
struct SplitF32Layout {
  size_t parts_a, parts_b, scale_a, scale_b, columns, end;
  int scale_lda, scale_ldb;
};
inline SplitF32Layout split_f32_layout(size_t base, int M, int N, int K) {
  auto up = [](size_t v) { return (v + 1023) / 1024 * 1024; };
  const size_t kb = (static_cast<size_t>(K) + 63) / 64;
  SplitF32Layout l;
  l.scale_lda = (M + 255) / 256 * 256;
  l.scale_ldb = (N + 255) / 256 * 4;
  l.parts_a = up(base);
  l.parts_b = up(l.parts_a + (static_cast<size_t>(M) + 127) / 128 * kb * 32768);
  l.scale_a = up(l.parts_b + (static_cast<size_t>(N) + 63) / 64 * kb * 16384);
  l.scale_b = up(l.scale_a + kb * l.scale_lda * 4);
  l.columns = up(l.scale_b + kb * l.scale_ldb * 4);
  l.end = up(l.columns + static_cast<size_t>(l.scale_ldb) * 64 * 4);
  return l;
}

}  // namespace kcg
