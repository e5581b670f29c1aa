// Host-side structures of librelux_cuda: device handle, paged pool, per-call staging.
#pragma once

#include <cuda_runtime.h>
#include <cuda.h>

#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "common.cuh"
#include "host_ring.h"
#include "relux_cuda.h"

namespace relux {

constexpr uint32_t kDeviceMagic = 0x52444556u;  // "RDEV"
constexpr uint32_t kPoolMagic = 0x52504F4Cu;    // "RPOL"

void set_error(const char* fmt, ...);
int32_t cuda_fail(cudaError_t e, const char* what);

#define RELUX_CUDA_TRY(expr)                                  \
  do {                                                        \
    cudaError_t e__ = (expr);                                 \
    if (e__ != cudaSuccess) return ::relux::cuda_fail(e__, #expr); \
  } while (0)

constexpr int64_t kResidentBytes = (int64_t)63 << 20;   // half of L2: what a launch may count on finding there again

struct Device {
  uint32_t magic = kDeviceMagic;
  int index = 0;
  int sm_count = 0;
  size_t total_mem = 0;
  char name[256] = {0};
  cudaStream_t stream = nullptr;
  // copy streams of pipelined calls (RELUX_CALL_PIPELINED): host -> device inputs, device -> host outputs
  cudaStream_t h2d_stream = nullptr, d2h_stream = nullptr;
  cudaEvent_t ev_copy_join = nullptr;
  bool copies_in_flight = false;
  std::mutex mu;
  int64_t launches = 0;
  std::vector<std::pair<const void*, size_t>> smem_allowed;   // what allow_smem knows of the kernels' limits, under mu
  void* flush_buf = nullptr;
  size_t flush_bytes = 0;
  // Page-locked memory for results of host calls, written by the kernel that makes them: the call waits for the stream and
  // copies on, so nothing is left in it when `mu` is given up.  A device-to-host copy behind the kernel cost 5-9 us at 16 KB and
  // 15 us at 512 KB; at 1 MB and more the driver's own copy is as fast or faster.
  static constexpr size_t kHostOutBytes = 512 << 10;
  void* host_out = nullptr;
  // Page-locked memory for the new rows of an append or a GQA step that arrive in pageable memory, read by the kernel that caches them: a
  // copy costs the host 2-3 us and the stream a trip to the copy engine and back (one token through the cache object, 700 cached:
  // 44.2 -> 40.6 us; a step of one sequence 35.3 -> 33.0).  Queries are still copied: every CTA that works on a stream reads them, and
  // over PCIe that cost more (44.2 -> 46.8); so are a latent step's rows.  Calls take their places one behind another; the stream is waited for where they start again,
  // and a call that waits for it anyway starts again at its end.  Used under `mu`.
  static constexpr size_t kHostInBytes = 1 << 20, kHostInMax = 32 << 10;
  char* host_in = nullptr;
  HostRing host_in_ring{kHostInBytes};
};

// A device buffer that grows on demand (never shrinks) for inputs that arrive in host memory
// and for kernel scratch.  Growth synchronises the stream before the old block is freed.
struct GrowBuf {
  void* p = nullptr;
  size_t cap = 0;
};

// Tuning knobs of a pool.  Defaults come from the environment ONCE, when the pool is created (RELUX_MLA_GENERIC,
// RELUX_MLA_WORKERS, RELUX_CHUNK_PAGES, RELUX_GEMM_GENERIC, RELUX_GEMM_SPLIT, RELUX_GQA_PROMPT_PARTIAL_MB,
// RELUX_SEL_CLUSTER, RELUX_SEL_LOOKAHEAD, RELUX_SEL_BATCHED, RELUX_GQA_PROMPT_SLICES); relux_pool_tune changes them
// afterwards.  No launch path reads the environment.
struct Tuning {
  int32_t v[RELUX_TUNE_COUNT];
  int32_t get(int knob) const { return v[knob]; }
};

// Two device buffers used in turn by pipelined calls.  `copied`: the copy into (inputs) or out of (outputs) the slot is done; `reader`: the
// PipeCalls number of the call whose kernels read an input's slot last.
struct PipeSlots {
  static constexpr int kSlots = 2;
  GrowBuf buf[kSlots];
  cudaEvent_t copied[kSlots] = {};
  uint64_t reader[kSlots] = {};
  bool used[kSlots] = {};   // of an output
  uint64_t next = 0;
};

// The ends of pipelined calls on the compute stream, numbered from 1: one event a call serves all of its buffers.  An event that a later call has
// recorded again says more than is asked for.
struct PipeCalls {
  static constexpr int kEvents = 4;
  cudaEvent_t done[kEvents] = {};
  uint64_t last = 0;      // calls recorded
  uint64_t copies = 0;    // the input copies are behind this one
  cudaEvent_t of(uint64_t call) const { return done[call % kEvents]; }
};

// Times of the last kCalls calls.  A call is timed by stamps its kernel writes (one launch: time_stamp_next), or by an
// event pair around several launches (time_events_begin / _end).
struct TimeRing {
  static constexpr int kCalls = 8192, kSlots = kCalls + 1;   // a call clears the slot of the one after it
  TimeSlot* slots = nullptr;                                 // device [kSlots], zero-filled
  cudaEvent_t ev[kCalls][2] = {};
  uint8_t stamped[kCalls] = {};
  uint64_t calls = 0;
};

struct Pool {
  uint32_t magic = kPoolMagic;
  Device* dev = nullptr;
  relux_pool_params prm{};
  Tuning tune{};
  int row_elems_a = 0;  // MLA: dC + dHR (one fused row); GQA: head_dim
  size_t page_elems = 0;    // elements per page per tensor (MLA: P*(dC+dHR); GQA: Hkv*P*D for K, same for V)
  size_t layer_elems = 0;   // elements per layer (GQA: K then V)
  uint16_t* storage = nullptr;  // bf16 bits
  void* meta = nullptr;         // one device block: table, lengths, status, ids, row offsets, time slots of the attention calls
  int32_t* d_table = nullptr;   // [max_seqs][max_pages_per_seq]
  int32_t* d_len = nullptr;     // [num_layers][max_seqs]
  int32_t* d_status = nullptr;   // [0] status word, [1] block counter of the append kernels
  std::vector<int32_t> h_table, h_len;
  bool graph_lengths = false;   // a call that changes lengths was captured: launches of the graph change the device's alone, h_len may be older
  std::vector<int32_t> seq_pages;  // pages reserved per sequence (capacity), 0 = slot not live
  std::vector<uint8_t> seq_owned;  // 1 = table rows were filled by relux_seq_alloc
  bool caller_tables = false;      // relux_pool_set_tables filled the tables: the free list stays unused until a reset
  std::vector<int32_t> free_pages;
  std::vector<uint32_t> seq_stamp;  // duplicate-id detection of stage_batch: call number that last named the sequence
  uint32_t stamp = 0;
  // reference-compat pools (RELUX_POOL_FLAG_REFERENCE_COMPAT): what the quirk-faithful attention mode needs
  bool compat = false;
  float* shadow_f32 = nullptr;   // MLA: float32 copy of every appended row, [layer][page][token][dC + dHR] (the reference's cache
                                 // is float32, mla_cache.go:46-52)
  std::vector<std::vector<int32_t>> chunks;   // GQA: per (layer, sequence) the first row of every Append call (kvcache.go:407-438
                                              // writes chunk-linear; mha.go:299-312 reads head-major)
  GrowBuf chunk_tab;             // device staging of the chunk starts of one call's sequences
  // per-call staging of small host arrays (seq ids, row offsets)
  int32_t* d_seq_ids = nullptr;  // [max_seqs]
  int32_t* d_row_off = nullptr;  // [max_seqs + 1]
  // Pinned staging for per-call id / row-offset / length arrays: a ring of slots, each guarded by its own event, so
  // that a call waits for a copy issued kStageSlots calls ago (long finished) instead of for the previous step's kernels.
  static constexpr int kStageSlots = 8;
  int32_t* h_stage = nullptr;    // pinned [kStageSlots][4 * (max_seqs + 1)]
  cudaEvent_t stage_ev[kStageSlots] = {};
  bool stage_busy[kStageSlots] = {};
  uint32_t stage_next = 0;
  size_t stage_slot_ints() const { return 4 * ((size_t)prm.max_seqs + 1); }
  // staging of activations that arrive in host memory, and outputs that leave to it
  GrowBuf in_a, in_b, out_buf, q_conv;
  GrowBuf expand_buf;  // expanded keys / values of an MLA prompt (+ the sequences' first rows)
  GrowBuf step_rows;   // host-resident new rows of a fused decode step (the attention call uses in_a / in_b for the queries)
  PipeCalls pipe_calls;
  PipeSlots pipe_in_a, pipe_in_b, pipe_app_a, pipe_app_b, pipe_out;   // the same for pipelined calls
  // attention scratch
  GrowBuf q_abs;     // MLA absorbed queries, bf16 [n][S][H][dC+dHR]
  GrowBuf part_o;    // split-KV partial accumulators, f32
  GrowBuf part_ml;   // split-KV partial (max, sum), f32 pairs
  GrowBuf stream_done;   // GQA stream kernel: finished pieces per (sequence, kv head), zero between launches
  int32_t* sel_host = nullptr;   // page-locked result words of the selection kernels
  size_t sel_words = 0;
  GrowBuf seq_list;      // GQA stream kernel: the sequences of a call too long for kernel arguments
  GrowBuf work;      // int32 work list + per-sequence chunk offsets
  GrowBuf o_lat;     // MLA merged latent output, f32/bf16
  // TMA descriptors over the pool storage (built at create when the shape allows it)
  CUtensorMap tmap_mla{};   // 2-D [rows][dC+dHR], box 64 x 64, 128-byte swizzle
  CUtensorMap tmap_mla_2{}, tmap_mla_3{};   // the same in boxes of two and of three neighbouring blocks of a page
  CUtensorMap tmap_gqa{};   // 2-D [rows][D],      box 64 x 64, 128-byte swizzle
  bool has_tmap = false;
  bool mla_blocked = false;   // MLA pages stored as 64-column blocks (see mla_page_off)
  // layer-level step (layer_step.cu): RoPE tables [cos | sin][positions][dHR / 2] and the step's scratch block
  GrowBuf rope_tab, layer_buf;
  int rope_dim = 0, rope_positions = 0;
  float rope_base = 0.f;
  // device times of the dominant kernel of the last kTimeRing attention calls, and of the input-projection GEMM of the
  // layer steps, for a caller to read after the fact without a synchronisation between the calls
  TimeRing attn_times, proj_times;
  uint64_t attn_calls = 0;   // MLA decode calls, timed or not (RELUX_TUNE_KERNEL_TIMING_STRIDE)
};

inline Device* as_device(relux_device_t h) {
  Device* d = (Device*)h;
  return (d && d->magic == kDeviceMagic) ? d : nullptr;
}
inline Pool* as_pool(relux_pool_t h) {
  Pool* p = (Pool*)h;
  return (p && p->magic == kPoolMagic && p->dev && p->dev->magic == kDeviceMagic) ? p : nullptr;
}

int32_t grow(Device* dev, GrowBuf& b, size_t bytes);
// Pipelined staging: copies a host input into the next slot on the copy stream; with `last` the compute stream waits for it, and for the copies
// before it.  pipe_end is called once the kernels that read a call's slots have been queued, then pipe_release for each of the slots.
int32_t pipe_stage_in(Pool* p, PipeSlots& ps, const void* src, size_t bytes, bool last, const void** dptr, int* slot);
int32_t pipe_end(Pool* p);
inline void pipe_release(Pool* p, PipeSlots& ps, int slot) {
  if (slot >= 0) ps.reader[slot] = p->pipe_calls.last;
}
// Next staging slot (waits for the copy that last used it); call stage_release after the copies are enqueued.
int32_t stage_acquire(Pool* p, int32_t** slot, int* slot_index);
int32_t stage_release(Pool* p, int slot_index);

// Resolved view of one call's sequences on the device.
struct SeqBatch {
  int32_t n_seqs = 0;
  const int32_t* d_seq_ids = nullptr;  // nullptr = identity
  const int32_t* d_row_off = nullptr;  // nullptr = rows_each rows per sequence
  int32_t rows_each = 1;
  int32_t total_rows = 0;
  int32_t max_rows = 0;
  std::vector<int32_t> seq;  // host copy of ids
  std::vector<int32_t> rows; // host copy of rows per sequence
};
int32_t stage_batch(Pool* p, int32_t n_seqs, const int32_t* seq_ids, const int32_t* n_rows, int32_t uniform_rows,
                    SeqBatch* out, bool upload = true);

// kernels (defined in the .cu files of this directory)
int32_t launch_mla_append(Pool* p, const SeqBatch& sb, int layer, const void* ckv, const void* kr, int dtype, int advance);
int32_t launch_gqa_append(Pool* p, const SeqBatch& sb, int layer, const void* k, const void* v, int dtype, int layout,
                          int advance);
int32_t launch_set_len(Pool* p, const SeqBatch& sb, int layer0, int layers, const int32_t* new_len);   // new_len: host
int32_t launch_gather_rows(Pool* p, int layer, int seq, int tok0, int n, uint16_t* d_a, uint16_t* d_b);
int32_t launch_attn_reference_gqa(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const float* d_q, float* d_out);
int32_t launch_attn_reference_mla(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const float* d_q, const float* d_qr,
                                  float* d_out);
int32_t launch_gqa_decode_fast(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const void* d_q, void* d_out);
// The new rows of a GQA decode or verify step that its attention launch appends itself (gqa_stream.cu).
struct GqaAppend {
  const void* k;
  const void* v;
  int dtype, layout, advance;
  const int32_t* rows;   // host: new rows per sequence
};
bool gqa_stream_eligible(const Pool* p, const relux_attn_args& a);
bool gqa_append_fusable(const Pool* p, const relux_attn_args& a, int max_new_rows, bool advance);
int32_t launch_gqa_stream(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const void* d_q, void* d_out, bool out_bf16,
                          const GqaAppend* app);
// True when this call is a multi-token call that the tcgen05 prefill kernel serves (it takes bf16 queries).
bool mla_expand_eligible(const Pool* p, int num_heads, int head_dim);
int64_t mla_expand_rows(const Pool* p, const SeqBatch& sb, int layer, int extra);
int32_t launch_mla_expand_sm100(Pool* p, const SeqBatch& sb, int layer, int extra, int H, const uint16_t* w_uk, const uint16_t* w_uv,
                                int64_t Ttot, uint16_t* kx, uint16_t* vx, int32_t* seq_base);
bool mla_prefill_eligible(const Pool* p, const SeqBatch& sb, const relux_attn_args& a);
bool gqa_prompt_wants_bf16(const Pool* p, const relux_attn_args& a);
// The new rows of a decode step handed to the attention call, for the fused preparation (one launch for absorb + append +
// stream partition); the host lengths already include them.
struct StepAppend {
  const void* ckv;
  const void* kr;
  int dtype;
  const int32_t* d_row_off;   // device row offsets of the append batch (nullptr = rows_each rows per sequence)
  int32_t rows_each = 1, max_rows = 1;   // new rows of a sequence: of each (where there are no offsets), at most
  bool weights_ready = false; // a launch before this one in the call has waited for everything older (launch_mla_prep)
};
int32_t launch_mla_decode_fast(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const void* d_q, const void* d_qr,
                               void* d_out, bool out_bf16 = false, const StepAppend* step = nullptr);
// True when that path's last kernel can write its result as bf16 itself.
bool mla_writes_bf16(const Pool* p, const SeqBatch& sb, const relux_attn_args& a);
// True when launch_mla_decode_fast can take the step's append into its preparation launch.
bool mla_step_fusable(Pool* p, const relux_attn_args& a);

int32_t do_mla_layer(Pool* p, const relux_mla_layer_args* a);
int32_t do_gqa_layer(Pool* p, const relux_gqa_layer_args* a);
int32_t do_spec_accept(Pool* p, const relux_spec_accept_args* a);
int32_t do_sample(Pool* p, const relux_sample_args* a);
int32_t do_matmul(Pool* p, const relux_matmul_args* a);
int32_t do_import_mla(Pool* p, const relux_mla_import_args* a);
int32_t do_selftest_wait(Pool* p, int32_t polls);
// After a fused call that counted sb's rows and failed: the lengths before it, on the host and, whatever the call had queued
// by then, on the device.  The error text of the call stays.
void take_rows_back(Pool* p, const SeqBatch& sb, int layer);
int32_t seq_set_len(Pool* p, int32_t layer, int32_t n_seqs, const int32_t* seq_ids, const int32_t* new_len);
// Chunk bookkeeping of reference-compat pools (no-ops otherwise): an append of n rows at old_len, a length change.
void note_append(Pool* p, int layer, int seq, int old_len, int n);
void note_set_len(Pool* p, int layer, int seq, int old_len, int new_len);
// Host pointers handed over as device memory must be 16-byte aligned: the kernels read them with vector loads.
int32_t check_dev_align(const void* ptr, const char* what);

// Whether what the call launches now is recorded in a graph: it then runs with the device's lengths of later moments, not with the host's.
bool stream_captured(const Device* dev);
// Of a call that changes lengths of a latent pool.
inline void note_lengths_change(Pool* p) {
  if (p->prm.kind == RELUX_POOL_MLA && !p->graph_lengths && stream_captured(p->dev)) p->graph_lengths = true;
}

// Tensor maps (runtime.cu).  bf16 elements, 128-byte swizzle, no out-of-bounds fill value (zeros); false when the driver
// entry point is missing or refuses the map.
//   2-D: [rows][cols], cols contiguous, box = box_cols x box_rows.
//   3-D: [outer][mid][cols], cols contiguous and mid rows adjacent, box = box_cols x box_mid x box_outer.
bool make_tmap_2d(CUtensorMap* m, void* base, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);
//   view: any of up to five dims, innermost first, strides of dims 1 .. in elements.
bool make_tmap_view(CUtensorMap* m, void* base, int rank, const uint64_t* dims, const uint64_t* stride_elems, const uint32_t* box);
//   4-D, float32, for stores: dims and box innermost first, box[0] = 16 or 32 columns (swizzled by the row length).
bool make_tmap_4d_f32(CUtensorMap* m, void* base, const uint64_t (&dims)[4], const uint32_t (&box)[4]);
bool make_tmap_3d(CUtensorMap* m, void* base, uint64_t outer, uint64_t mid, uint64_t cols, uint32_t box_cols, uint32_t box_mid,
                  uint32_t box_outer);

TimeStamp time_stamp_next(Pool* p, TimeRing& r);
void time_stamp_done(TimeRing& r, const TimeStamp& ts);
int32_t time_events_begin(Pool* p, TimeRing& r);
int32_t time_events_end(Pool* p, TimeRing& r);

// Dynamic shared memory above 48 KB has to be allowed once per kernel and context, not per launch.
int32_t allow_smem(Device* dev, const void* kernel, size_t bytes);
template <typename... KArgs>
inline int32_t allow_smem(Device* dev, void (*kernel)(KArgs...), size_t bytes) { return allow_smem(dev, (const void*)kernel, bytes); }

inline void count_launch(Device* d, int n = 1) { d->launches += n; }

// Launches `kern`; with `chained` the launch carries the programmatic stream-serialization attribute, so the grid may be
// scheduled as soon as every block of the kernel before it in the stream has called chain_release() (common.cuh) or ended,
// whatever that kernel itself still waits for.  What keeps the stream's order of results:
//   1. Every such kernel calls chain_wait() in the threads that write, and in those that read what a launch of the chain
//      writes, before they do.  A kernel is complete only when all its threads are, so "the launch before me is complete" holds
//      back to the first launch of the chain.
//   2. What a launch of the chain writes is read by load_chained() or by plain loads of pointers that are not
//      const __restrict__, and by TMA only where the writer has called fence_chained_writes().
//   3. Before its wait a kernel may read what was complete before the HEAD of its chain began.  A head is a plain launch, a launch
//      behind a copy or an event, or one whose blocks all wait before they release: cast_bf16_kernel, and mla_prep_kernel
//      without weights_ready.  Those who read early, and why they may:
//        - page tables, everywhere: the host calls that change them wait for the stream and for their copy;
//        - skinny_gemm_sm100_kernel, the weights: the first launch of a layer step or matmul is cast_bf16_kernel, the
//          second GEMM of a layer follows it, a plain absorb launch, or a cast of its own;
//        - mla_prep_kernel with weights_ready, W_UK: only behind the projections of the same call (do_mla_layer);
//        - build_stream_kernel, the lengths (and it writes the plan, which the launches of older calls read): behind an mla_prep_kernel that is
//          a head, or a plain absorb launch;
//        - mla_decode_sm100_kernel, tiles without new rows, where it has the plan as arguments: the call's head is before it;
//        - mla_vup_pieces_kernel, W_UV: the preparation or the plain absorb launch of the same call is before it.  (It also reads part_ml there,
//          whatever it holds, and makes no use of it: mla_proj.cu.)
//      A new early read names its head here; a new launch in front of one of these keeps a head between.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(bool chained, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                  Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace relux
