// Split-KV work list shared by the FAST attention kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "stream_plan.h"

namespace relux {

struct WorkItem {
  int32_t seq_index;   // position of the sequence inside this call (row block of q / out)
  int32_t seq;         // pool sequence id (page-table row)
  int32_t page_begin;  // first logical page of the chunk
  int32_t page_end;    // one past the last logical page
};

// Item of a stream plan (plan_stream): like WorkItem plus the sequence's token count, so that a persistent kernel
// needs a single load per item.
struct __align__(16) StreamItem {
  int32_t seq_index;
  int32_t seq;
  int32_t page_begin;
  int32_t page_end;
  int32_t tokens;      // cached length of the sequence + the call's extra tokens
  int32_t first, n;    // the sequence's first item and how many it has
  int32_t pad;
};

// A stream plan as kernel arguments, for calls of a few items: the decode kernel then knows its work, and asks for cached rows, before the
// launch in front of it is complete.
constexpr int kListedItems = 160, kListedWorkers = 80;
struct ListedItem {
  int32_t seq, tokens;
  uint16_t page_begin, page_end, seq_index, first, n, pad;   // as in StreamItem
};
struct ListedPlan {
  int32_t listed;        // 0: the plan is in device memory
  int32_t new_rows;      // the call's launches before the decode kernel write the last new_rows of a sequence's tokens, at most
  uint16_t worker_first[kListedWorkers + 2];
  ListedItem items[kListedItems];
};

struct SplitPlan {
  int chunk_pages = 0;                 // of a stream plan: pages of a piece, or units of a range
  int num_items = 0;
  bool loose = false;           // made for the host's lengths, but the launches find the device's, which may be others: in a graph, and once a
                                // graph has changed them (Pool::graph_lengths)
  int room_items = 0;           // partials are given room for as many (num_items, where that is more): StreamShape::room
  WorkItem* items = nullptr;    // device
  int32_t* chunk_off = nullptr; // device [n_seqs + 1]
  std::vector<int32_t> first;   // the same on the host: sequence i has items [first[i], first[i + 1])
  // stream plans only (plan_stream): worker w owns items [worker_first[w], worker_first[w + 1])
  int num_workers = 0;
  // every worker has one item, chunk_pages pages of a sequence; or ranges of chunk_pages units, a sequence's pages (an even number of
  // units) behind `start_units` units of fixed cost (plan_stream)
  bool by_item = false;
  int start_units = 0;
  StreamItem* stream_items = nullptr;  // device [num_items]
  int32_t* worker_first = nullptr;     // device [num_workers + 1]
};

// A row of a latent call's partial results: float32, the bf16 value of the row's whole attention or two bf16 halves a column (write_partial,
// mla_decode_sm100.cu).
enum PartialForm { kPartialFloat32 = 0, kPartialOne = 1, kPartialHalves = 2 };

struct Pool;
struct SeqBatch;
// `max_row_items`: more chunks than that no sequence is cut into (0: any number).
int32_t plan_splitkv(Pool* p, const SeqBatch& sb, int layer, int extra, int ctas_per_item, int min_chunk_pages, int chunk_multiple,
                     int max_chunk_pages, int max_row_items, SplitPlan* plan);
// Stream partition for persistent kernels: the sequences of the call, laid end to end, are cut into at most `workers` equal ranges;
// one item = the part of one sequence inside one range, so a worker meets an item boundary only where a sequence ends inside its
// range.  Where that is cheaper they are cut sequence by sequence instead, one item a worker (cheapest_plan).  With the tuning knob
// CHUNK_PAGES: ranges of that many pages, rounded up to `page_multiple`.
// The host half: counts and buffers.  The lists are built by the fused decode step's preparation (mla_proj.cu), or by
// launch_build_stream behind a preparation that only absorbs.
// `list`: where the plan fits there, it is written there and not built on the device.
int32_t plan_stream(Pool* p, const SeqBatch& sb, int layer, int extra, int workers, int page_multiple, SplitPlan* plan, ListedPlan* list);
int32_t launch_build_stream(Pool* p, const SeqBatch& sb, int layer, int extra, const SplitPlan& plan, bool chained);
int32_t launch_build_worklist_raw(cudaStream_t st, const int32_t* len, const int32_t* seq_ids, int n_seqs, int extra, int page_tokens,
                                  int chunk_pages, WorkItem* items, int32_t* chunk_off, int room, int32_t* status);
int32_t launch_merge_raw(cudaStream_t st, const float* part_o, const float* part_ml, const int32_t* chunk_off, int n_seqs, int rows,
                         int width, float* out);
int32_t launch_merge(Pool* p, const SplitPlan& plan, int n_seqs, int rows, int width, float* out);
// Same, for a launch that covers `rows` of the `out_rows` output rows of every sequence, starting at row out_row0.
int32_t launch_merge_rows(Pool* p, const SplitPlan& plan, int n_seqs, int rows, int width, float* out, int out_rows, int out_row0,
                          int slices = 1, long long part_group_rows = 0);

}  // namespace relux
