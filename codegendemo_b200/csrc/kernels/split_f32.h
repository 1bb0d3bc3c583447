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
  unsigned int* words;           // H2_WORDS
  uint8_t *far_a, *far_b;        // far parts, a slot a chunk
  float *far_scale_a, *far_scale_b;  // [slot][128 rows], [slot] and behind them a zero
  int far_slots_a, far_slots_b;
};

// Byte offsets of the arrays behind `base`, and the end. Rows and columns of the exponents are padded to whole tiles:
// the product reads those of rows and columns past the edge (and multiplies zeros by them).
// Far parts may be had for a sixteenth of the chunks (products of less than 16 chunks have none): their memory, and at most 40 %
// more chunks for a tile to multiply when they are spread over A and B, where 3xTF32 takes 2.2 times as long.
struct SplitF32Layout {
  size_t parts_a, parts_b, far_a, far_b, scale_a, scale_b, columns, far_scale_a, far_scale_b, end;
  int scale_lda, scale_ldb, far_slots_a, far_slots_b;
};
inline SplitF32Layout split_f32_layout(size_t base, int M, int N, int K) {
  auto up = [](size_t v) { return (v + 1023) / 1024 * 1024; };
  const size_t kb = (static_cast<size_t>(K) + 63) / 64;
  SplitF32Layout l;
  l.scale_lda = (M + 255) / 256 * 256;
  l.scale_ldb = (N + 255) / 256 * 4;
  l.parts_a = up(base);
  const size_t chunks_a = (static_cast<size_t>(M) + 127) / 128 * kb, chunks_b = (static_cast<size_t>(N) + 63) / 64 * kb;
  l.far_slots_a = static_cast<int>(chunks_a / 16);
  l.far_slots_b = static_cast<int>(chunks_b / 16);
  l.parts_b = up(l.parts_a + chunks_a * 32768);
  l.far_a = up(l.parts_b + chunks_b * 16384);
  l.far_b = up(l.far_a + static_cast<size_t>(l.far_slots_a) * 32768);
  l.scale_a = up(l.far_b + static_cast<size_t>(l.far_slots_b) * 16384);
  l.scale_b = up(l.scale_a + kb * l.scale_lda * 4);
  l.columns = up(l.scale_b + kb * l.scale_ldb * 4);
  l.far_scale_a = up(l.columns + static_cast<size_t>(l.scale_ldb) * 64 * 4);
  l.far_scale_b = up(l.far_scale_a + static_cast<size_t>(l.far_slots_a) * 128 * 4);
  l.end = up(l.far_scale_b + (static_cast<size_t>(l.far_slots_b) + 1) * 4);
  return l;
}

}  // namespace kcg
