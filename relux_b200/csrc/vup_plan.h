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
  int planned, most;                              // columns that a group has at the host's lengths, and may find
  int blocks, n_block, n_kb, n_stages;            // a stage: n_kb times 64 latent columns of n_block columns, [n_kb][hi | lo][n_block][64]
  int tmem_cols;
  bool fits() const { return most <= kVupMaxCols && tmem_cols <= 512; }
};

// Rows (n_seqs x S) are dealt to groups of CTAs: one where the heads fill the GPU (`fit` groups do), more, of about 32 columns each, where they do not, or where
// a group would have more columns than it has room for.  The second group comes with 41 columns, or with 53 where no third one would fit.  Steps with one group
// and with two, us, by columns: 32 heads 33 20.7 / 20.8, 36 17.9 / 17.8, 39 25.0 / 25.2, 42 17.7 / 17.5, 45 19.4 / 18.0, 48 19.7 / 17.7, 51 19.2 / 18.1, 54 23.5 /
// 22.0, 57 20.9 / 18.5, 60 18.0 / 16.8; 64 heads 41 27.4 / 26.3, 45 24.4 / 24.6, 49 28.9 / 28.9, 53 22.1 / 22.3, 57 22.5 / 22.5, 61 22.3 / 22.4, 65 24.5 / 23.6, 69
// 34.1 / 33.6.  A group's columns are one block where a stage of it, 64 latent columns, fits the ring four times, and equal blocks otherwise.
// `first`: the plan's pieces at the host's lengths.  With `workers` the launch may find other lengths, on which the builder cuts at most workers - 1
// sequences once more each (build_stream): what a group then has at most is its rows, and every cut once for each of its rows of the sequence.  With
// kVupAnyChunks it may find any chunks, as many as were planned in all (build_worklist_kernel): one group may have them all.
constexpr int kVupAnyChunks = -1;
inline VupShape vup_shape(const std::vector<int32_t>& first, int rows, int S, int fit, int halves, int dC, int workers) {
  VupShape k;
  const int all = vup_col(first, S, rows);
  // (a row at a time fewer, from as many groups as the columns need at least: all numbers of groups in turn were quadratic in the rows)
  const int second = fit > 2 ? 41 : 53;
  int groups = std::max({1, std::min({fit, (all + 64 - second) / 32, rows}), workers > 0 ? 1 : std::min(rows, (all + kVupMaxCols - 1) / kVupMaxCols)});
  if (workers == kVupAnyChunks && all > kVupMaxCols) groups = rows;
  for (;; groups = (rows + k.rows_each - 2) / (k.rows_each - 1)) {
    k.rows_each = (rows + groups - 1) / groups;
    k.planned = k.most = 0;
    for (int r = 0; r < rows && (k.most <= kVupMaxCols || k.rows_each == 1); r += k.rows_each) {
      const int end = std::min(rows, r + k.rows_each), n = end - r;
      const int now = vup_col(first, S, end) - vup_col(first, S, r);
      const int later = workers > 0 ? n + std::min(S, n) * (workers - 1) : workers == kVupAnyChunks ? all : now;
      k.planned = std::max(k.planned, now);
      k.most = std::max(k.most, k.rows_each > 1 ? later : std::max(now, std::min(later, kVupMaxCols)));   // one row: the kernel reports what is more
    }
    if (k.most <= kVupMaxCols || k.rows_each == 1) break;
  }
  k.groups = (rows + k.rows_each - 1) / k.rows_each;
  // As wide as the host's lengths need, and as many as others may; as wide as those need where that would be more tensor memory than there is.
  const int widest = kVupRing / 4 / (halves * 128);
  for (int wide : {k.planned, k.most}) {
    const int n = std::max(1, (wide + widest - 1) / widest), unit = (k.most > wide || n > 1 ? 32 : 16) / halves;
    // N is a multiple of 16, and a block begins at a multiple of 32 tensor-memory columns
    k.n_block = std::max(unit, ((wide + n - 1) / n + unit - 1) / unit * unit);
    k.blocks = std::max(1, (k.most + k.n_block - 1) / k.n_block);
    if (k.blocks * k.n_block * halves <= 512) break;
  }
  const int blk_bytes = halves * k.n_block * 128;
  k.n_kb = 4;
  while (k.n_kb > 1 && k.n_kb * blk_bytes > kVupRing / (k.n_kb > 2 ? 2 : 3)) k.n_kb /= 2;
  k.n_stages = std::min({kVupMaxStages, kVupRing / (k.n_kb * blk_bytes), (dC / 64 + k.n_kb - 1) / k.n_kb * k.blocks});
  k.tmem_cols = 32;
  while (k.tmem_cols < k.blocks * halves * k.n_block) k.tmem_cols *= 2;
  return k;
}

}  // namespace relux
