// Device parts of the fused MLA decode-step preparation (one launch instead of three): the append of the step's new
// rows, and the stream partition the persistent decode kernel walks.  They run as extra blocks of the query-absorb grid
// (mla_proj.cu); the stand-alone kernels in append.cu and splitkv.cu do the same work for the unfused calls.
#pragma once

#include "common.cuh"
#include "splitkv.h"

namespace relux {

struct PrepAppend {
  const int32_t* table;
  int32_t table_stride;
  int32_t* len;                // this layer's [max_seqs]
  const int32_t* seq_ids;
  const int32_t* row_off;      // nullptr = rows_each new rows per sequence
  int32_t rows_each;
  int32_t num_pages, page_tokens, max_pages_per_seq, n_seqs;
  int32_t* status;
  uint32_t* done;              // zero between launches; counts the blocks that have finished with the lengths
  uint16_t* layer_base;
  const void* ckv;
  const void* kr;
  int32_t f32, dC, dHR, blocked;
};

struct PrepPlan {
  int32_t listed;              // nothing to build
  int32_t extra, G, workers, by_item, start_units;
  int32_t room;                // items that `items` and the partial results have room for
  StreamItem* items;
  int32_t* chunk_off;
  int32_t* worker_first;
};

// 8 consecutive source elements -> one uint4 of bf16 bits (float32 sources rounded with the reference's rule).
__device__ __forceinline__ uint4 prep_load8(const void* src, size_t elem_off, bool f32) {
  if (f32) {
    const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(src) + elem_off);
    const float4 a = load_chained(s), b = load_chained(s + 1);
    return make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
  return load_chained(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(src) + elem_off));
}

// Every block that reads the lengths arrives here once it is done with them; the last one to arrive advances all
// lengths by the rows appended (MLACache.Append: total += newLen, mla_cache.go:178) and re-arms the counter.
__device__ __forceinline__ void prep_arrive_and_advance(const PrepAppend& g, uint32_t expected) {
  __shared__ bool s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(g.done, 1u) == expected - 1;
  }
  __syncthreads();
  if (!s_last) return;
  for (int i = threadIdx.x; i < g.n_seqs; i += blockDim.x) {
    const int seq = g.seq_ids ? g.seq_ids[i] : i;
    g.len[seq] = load_chained(g.len + seq) + (g.row_off ? g.row_off[i + 1] - g.row_off[i] : g.rows_each);
  }
  if (threadIdx.x == 0) *g.done = 0u;
}

// All new rows of sequence i, by a warp (MLA row = [dC | dHR] fused; 16-byte stores).  A row's values do not wait for the length and the page that
// say where they go.  `advance`: the length is this warp's to advance.
__device__ __forceinline__ void prep_append_seq(const PrepAppend& g, int i, bool advance) {
  const int seq = g.seq_ids ? g.seq_ids[i] : i;
  const int r0 = g.row_off ? g.row_off[i] : i * g.rows_each;
  const int nrows = g.row_off ? g.row_off[i + 1] - r0 : g.rows_each;
  const int lane = threadIdx.x & 31;
  const int base_len = load_chained(g.len + seq);
  const int row_elems = g.dC + g.dHR, vec_per_row = row_elems / 8, vc = g.dC / 8;
  auto source = [&](int r, int v) {
    return (v < vc) ? prep_load8(g.ckv, (size_t)(r0 + r) * g.dC + (size_t)v * 8, g.f32 != 0)
                    : prep_load8(g.kr, (size_t)(r0 + r) * g.dHR + (size_t)(v - vc) * 8, g.f32 != 0);
  };
  constexpr int kHeld = 3;   // vectors of a row that a lane asks for ahead: a row of 512 + 64 columns
  for (int r = 0; r < nrows; r++) {
    uint4 held[kHeld];
#pragma unroll
    for (int k = 0; k < kHeld; k++)
      if (lane + 32 * k < vec_per_row) held[k] = source(r, lane + 32 * k);
    const int pos = base_len + r;
    const int slot = pos / g.page_tokens;
    int32_t pg;
    if (slot >= g.max_pages_per_seq || !page_of(g.table, g.table_stride, seq, slot, g.num_pages, g.status, &pg)) {
      if (slot >= g.max_pages_per_seq) set_status(g.status, RELUX_ERR_OVERFLOW);
      continue;
    }
    uint16_t* page = g.layer_base + (size_t)pg * g.page_tokens * row_elems;
    auto put = [&](int v, const uint4& w) {
      *reinterpret_cast<uint4*>(page + mla_page_off(g.blocked != 0, g.page_tokens, row_elems, pos % g.page_tokens, v * 8)) = w;
    };
#pragma unroll
    for (int k = 0; k < kHeld; k++)
      if (lane + 32 * k < vec_per_row) put(lane + 32 * k, held[k]);
    for (int v = lane + 32 * kHeld; v < vec_per_row; v += 32) put(v, source(r, v));
  }
  if (advance && lane == 0) g.len[seq] = base_len + nrows;
  fence_chained_writes();
}

// Exclusive prefix sum over a block of kWarps warps; *total receives the block's sum.
template <int kWarps>
__device__ __forceinline__ int prep_block_excl_scan(int v, int32_t* s_warp, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();   // s_warp may still be read from the previous call
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int base = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    if (w < warp) base += s_warp[w];
    sum += s_warp[w];
  }
  *total = sum;
  return base + incl - v;
}

// The stream partition, by a block: sequence i, of the pool's `seq`, has tokens_of(i, seq) tokens and occupies `units` units of the stream from `at`
// on, where SeqCut cuts it; items are numbered in stream order, so the items of a sequence and the items of a worker are both contiguous.
// The plan was made for the lengths that the host knows.  Where the device's are others (SplitPlan::loose) and have outgrown its workers or its room,
// the sequences are cut into equal ranges for as many workers instead, n_seqs + workers - 1 items at most.  That serves all lengths; if it did not, the
// plan would be empty and the status would say so: nothing is written past its room.
template <int kWarps, typename Tokens>
__device__ __forceinline__ void build_stream(const PrepPlan& pl, int n_seqs, const int32_t* seq_ids, int page_tokens, int32_t* status, Tokens tokens_of) {
  __shared__ int32_t s_warp[kWarps];
  int by_item = pl.by_item, G = pl.G, start_units = pl.start_units;
#pragma unroll 1
  for (int pass = 0;; pass++) {
    int unit_base = 0, item_base = 0;
    for (int i0 = 0; i0 < n_seqs; i0 += blockDim.x) {
      const int i = i0 + threadIdx.x;
      int seq = 0, pages = 0, tokens = 0;
      if (i < n_seqs) {
        seq = seq_ids ? seq_ids[i] : i;
        tokens = tokens_of(i, seq);
        pages = (tokens + page_tokens - 1) / page_tokens;
      }
      int tot_units, tot_items;
      const int at = unit_base + prep_block_excl_scan<kWarps>(SeqCut(by_item, G, start_units, 0, pages).units, s_warp, &tot_units);
      const SeqCut cut(by_item, G, start_units, at, pages);
      const int c0 = item_base + prep_block_excl_scan<kWarps>(cut.n, s_warp, &tot_items);
      if (i < n_seqs) {
        pl.chunk_off[i] = c0;
        for (int c = 0; c < cut.n && c0 + c < pl.room; c++) {
          StreamItem w;
          w.seq_index = i;
          w.seq = seq;
          w.page_begin = cut.begin(c);
          w.page_end = cut.end(c);
          w.tokens = tokens;
          w.first = c0;
          w.n = cut.n;
          w.pad = 0;
          pl.items[c0 + c] = w;
          const int worker = by_item ? c0 + c : cut.first + c;
          if (worker < pl.workers && (by_item || cut.leads(c, at))) pl.worker_first[worker] = c0 + c;
        }
      }
      unit_base += tot_units;
      item_base += tot_items;
    }
    const int used = by_item ? item_base : (unit_base + G - 1) / G;
    if (used <= pl.workers && item_base <= pl.room) {
      if (threadIdx.x == 0) pl.chunk_off[n_seqs] = item_base;
      for (int w = used + threadIdx.x; w <= pl.workers; w += blockDim.x) pl.worker_first[w] = item_base;   // no work
      return;
    }
    __syncthreads();
    if (pass == 1) {
      if (threadIdx.x == 0) set_status(status, RELUX_ERR_UNSUPPORTED);
      for (int w = threadIdx.x; w <= pl.workers; w += blockDim.x) pl.worker_first[w] = 0;
      for (int i = threadIdx.x; i <= n_seqs; i += blockDim.x) pl.chunk_off[i] = 0;
      return;
    }
    int units = 0;
    for (int i0 = 0; i0 < n_seqs; i0 += blockDim.x) {
      const int i = i0 + threadIdx.x;
      int pages = 0, tot;
      if (i < n_seqs) pages = (tokens_of(i, seq_ids ? seq_ids[i] : i) + page_tokens - 1) / page_tokens;
      prep_block_excl_scan<kWarps>(SeqCut(0, 1, kStartUnits, 0, pages).units, s_warp, &tot);
      units += tot;
    }
    by_item = 0;
    start_units = kStartUnits;
    G = range_units(units, pl.workers);
  }
}

// The same over the lengths AFTER this step's append (the append of the same launch has not advanced them yet: every sequence counts its cached rows +
// its new rows + extra).
template <int kWarps>
__device__ __forceinline__ void prep_build_stream(const PrepAppend& g, const PrepPlan& pl) {
  build_stream<kWarps>(pl, g.n_seqs, g.seq_ids, g.page_tokens, g.status, [&](int i, int seq) {
    return load_chained(g.len + seq) + (g.row_off ? g.row_off[i + 1] - g.row_off[i] : g.rows_each) + pl.extra;
  });
}

}  // namespace relux
