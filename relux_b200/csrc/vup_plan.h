// How the up-projection of a latent call deals the pieces of its rows to CTAs (mla_vup_pieces_kernel).  Plain C++: no CUDA, so that it can be
// checked on its own.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace relux {

constexpr int kVupMaxCols = 240;                  // columns of a CTA: two of the 512 tensor-memory columns each, in whole blocks
constexpr int kVupRing = 96 << 10, kVupMaxStages = 8;

// First column of a row of the call: the pieces of row (sequence i, query token q) are [first[i] S + q n_i, + n_i), n_i = first[i + 1] - first[i].
inline int vup_col(const std::vector<int32_t>& first, int S, int row) {
  const int i = row / S, q = row - i * S;
  return q == 0 ? first[i] * S : first[i] * S + q * (first[i + 1] - first[i]);
}

struct VupShape {
  int groups, rows_each;                          // rows of a group of CTAs, one for each head (the last group may have fewer)
  int most;                                       // columns that a group may find
  int blocks, n_block, n_kb, n_stages;            // a stage: n_kb times 64 latent columns of n_block columns, [n_kb][hi | lo][n_block][64]
  int tmem_cols;
  bool fits() const { return most <= kVupMaxCols && tmem_cols <= 512; }
};

// Rows (n_seqs x S) are dealt to groups of CTAs: one where the heads fill the GPU (`fit` groups do), more where they do not and there are more than 40
// columns (52 where only two groups fit), of about 32 columns each, or where a group would have more columns than it has room for.  (One group -> two of
// 24 to 32: 32 heads, 16 x 300 tokens 17.9 -> 16.5 us, 10 x 600 18.0 -> 16.8, 50 x 600 26.9 -> 25.3, 64 heads, 30 x 800 26.4 -> 25.6; not at 48 columns
// of 64 heads, 12 x 900 21.4 -> 22.1, nor at 36 of 32, 12 x 300 15.6 -> 17.2.)  A group's columns are one block where a stage of it, 64 latent columns,
// fits the ring four times, and equal blocks otherwise.
// `first`: the plan's pieces at the host's lengths.  With `workers` the launch may find other lengths, on which the builder cuts at most workers - 1
// sequences once more each (build_stream): what a group then has at most is its rows, and every cut once for each of its rows of the sequence.
inline VupShape vup_shape(const std::vector<int32_t>& first, int rows, int S, int fit, int halves, int dC, int workers) {
  VupShape k;
  const int all = vup_col(first, S, rows);
  // (a row at a time fewer, from as many groups as the columns need at least: all numbers of groups in turn were quadratic in the rows)
  int groups = std::max({1, std::min({fit, (all + (fit > 2 ? 23 : 11)) / 32, rows}), workers > 0 ? 1 : std::min(rows, (all + kVupMaxCols - 1) / kVupMaxCols)});
  for (;; groups = (rows + k.rows_each - 2) / (k.rows_each - 1)) {
    k.rows_each = (rows + groups - 1) / groups;
    k.most = 0;
    for (int r = 0; r < rows && (k.most <= kVupMaxCols || k.rows_each == 1); r += k.rows_each) {
      const int end = std::min(rows, r + k.rows_each), n = end - r;
      const int now = vup_col(first, S, end) - vup_col(first, S, r), later = workers > 0 ? n + std::min(S, n) * (workers - 1) : now;
      k.most = std::max(k.most, k.rows_each > 1 ? later : std::max(now, std::min(later, kVupMaxCols)));   // one row: the kernel reports what is more
    }
    if (k.most <= kVupMaxCols || k.rows_each == 1) break;
  }
  k.groups = (rows + k.rows_each - 1) / k.rows_each;
  const int widest = kVupRing / 4 / (halves * 128);
  k.blocks = std::max(1, (k.most + widest - 1) / widest);
  const int unit = (k.blocks > 1 ? 32 : 16) / halves;   // N is a multiple of 16, and a block begins at a multiple of 32 tensor-memory columns
  k.n_block = std::max(unit, ((k.most + k.blocks - 1) / k.blocks + unit - 1) / unit * unit);
  const int blk_bytes = halves * k.n_block * 128;
  k.n_kb = 4;
  while (k.n_kb > 1 && k.n_kb * blk_bytes > kVupRing / (k.n_kb > 2 ? 2 : 3)) k.n_kb /= 2;
  k.n_stages = std::min({kVupMaxStages, kVupRing / (k.n_kb * blk_bytes), (dC / 64 + k.n_kb - 1) / k.n_kb * k.blocks});
  k.tmem_cols = 32;
  while (k.tmem_cols < k.blocks * halves * k.n_block) k.tmem_cols *= 2;
  return k;
}

}  // namespace relux
