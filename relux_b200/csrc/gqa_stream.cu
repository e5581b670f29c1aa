// GQA decode / verify step over the paged bf16 K/V pool in ONE launch (RELUX_ATTN_FAST, up to 32 query rows per kv head):
// the append of the step's new rows, split-KV attention, and the merge of the splits.
//
// Bound: HBM bandwidth.  Every cached token costs Hkv * D * 2 (K, V) * 2 B = 4096 B at Hkv = 8, D = 128, against about
// 16 flop/B of work; short steps are bound by launches and by the latency of a page's round trip instead.
//
// One CTA per SM walks an equal share of the call's work, in UNITS of a page's time: sequence by sequence, kv head by kv head,
// all (sequence, kv head) streams -- a stream is its pages and a few units of fixed cost (kStreamUnits) -- are laid end to end and
// cut into gridDim.x ranges that differ by at most one unit; a range may hold fixed units only.  A PIECE is the part of one
// stream's pages inside one range.  The producer warp runs ahead over piece boundaries, so the 128 KB ring
// of pages stays full while a piece is finished.  (One CTA per fixed chunk, the layout before: three waves with a
// prologue and an epilogue each, 54.6 us for 244 MB at 32 sequences of about 1900 tokens.)
//   * Eight consumer warps.  A page takes four warps 0.65 us (a chain of dependent MMAs and shuffles) and arrives every
//     0.74 us at full bandwidth, so four alone cannot make up for a pause: up to 16 query rows, two groups of four take
//     alternate pages; above, each group takes 16 of the rows.
//   * Three finisher warps fetch the next piece's queries and combine, write and merge the piece before while the
//     consumers go on: with the consumers doing it, a piece cost them 2 us (its own output) to 5 us (a partial, with its
//     fence and counter), and the worker with the shortest sequences finished 12 us after the others.
//   * A piece that covers its whole stream writes the normalised output directly.  Otherwise it leaves a float32 partial,
//     and the last piece of the stream to finish (counters per stream, re-armed by that piece) merges all of them, in
//     range order whoever is last: a separate merge launch cost 5-20 us.
//   * The host knows every length, so the sequences travel as kernel arguments (up to 256; longer batches through a staged
//     copy): no work-list launch, no read of the device lengths.
//   * New rows: the CTA that loads a page of a kv head writes the step's new rows of that page and head (rounded with the
//     reference's rule) at its start, ordered before its own TMA loads by a proxy fence and a barrier the
//     producer meets at the first such page; (advance) the worker of a sequence's last page and first head stores the new
//     length.
// All mbarrier waits are bounded; a wait that runs out records RELUX_ERR_TIMEOUT and the CTA finishes with neutral data.
#include <algorithm>
#include <vector>

#include "common.cuh"
#include "gqa_parts.cuh"
#include "internal.h"
#include "umma.cuh"

namespace relux {

namespace {

constexpr int kInlineSmall = 32, kInlineLarge = 256;   // sequences carried as kernel arguments (0.5 KB / 4 KB)

struct GqaSeq {
  int32_t seq;     // pool sequence
  int32_t len0;    // cached rows before this call's new rows
  int32_t unit0;   // first unit of the sequence in the call's list (one kv head counted)
  int32_t row0;    // first new row of the sequence
};

struct GqaStreamCommon {
  const GqaSeq* seqs;      // device copy, or nullptr: the inline array
  const int32_t* table;
  int32_t table_stride, num_pages, n_seqs, range, range_more, Hkv, H, g, S, R, extra, causal;
  int32_t krow0, vrow0;    // first TMA row of this layer's K block / V block
  // A page is read once.  The pages of a call of more than half of L2 are loaded to be evicted first, so that they push out each other
  // and not what the next launches read, nor, in turn after turn, all of themselves: 32 sequences of 100 to 3000 tokens 45.0 -> 43.2 us,
  // 100 of 22 to 700 (64 heads) 42.0 -> 36.5, 16 x 2000 29.2 -> 26.6, a layer of 24 x 2048 66.8 -> 65.9.  Smaller ones may stay in L2 from
  // step to step, which 32 x <= 1000 with 4 kv heads, 34 MB, did less so (16.0 -> 16.65).
  int32_t streams;
  float scale_log2;
  const void* q;
  int32_t q_bf16, out_bf16;
  void* out;               // [n][S][H][128]
  float* part_o;           // [2 * workers][R][128]
  float* part_ml;          // [2 * workers][R][2]
  uint32_t* done;          // [n_seqs * Hkv][kFinishers], zero between launches
  // the step's new rows (k_new == nullptr: none)
  const void* k_new;
  const void* v_new;
  int32_t new_f32, head_major, advance;
  uint16_t* k_base;
  uint16_t* v_base;
  int32_t* len;            // this layer's device lengths
  int32_t* status;
  TimeStamp time;
};
template <int N>
struct GqaStreamParams {
  GqaStreamCommon c;
  GqaSeq seqs[N + 1];
};

// A stream (sequence, kv head) is its pages and kStreamUnits units of fixed cost: what a piece costs its consumers and finishers
// beyond its pages (queries, states, the rows' sums), 2-3 us against 0.74 us a page.  Measured with 0, 1, 4 and 6 units: 32
// sequences of 100 to 3000 tokens 47, 45.4, 44.8, 44.8 us; 100 of 22 to 700 tokens -, 45.3, 36.3, 36.3; 64 of 50 to 1500 -, 46.9,
// 44.2, 44.5.  (Too few, and the workers with the shortest streams finish last.)
constexpr int kStreamUnits = 4;
struct Piece {
  int32_t i, kvh, us, pb, pe, pages;   // sequence of the call, kv head, first unit of the stream, logical pages [pb, pe) of `pages`
};

// RS: rows of one warp's state in shared memory (8 or 16: all of MT = 1, a warp's half for MT = 2).  Up to 8 rows there is room
// for two pieces' states, so the consumers go on while the finishers read: streams of a page or two are as fast as the
// finishers then, not as both in turn.  The number
// of stages is even, so that with alternating pages a stage belongs to one group of warps for good: a group that waited
// on a stage it had skipped for a lap would take that lap's phase for its own (mbarrier phases are told apart by parity).
// Four stages, 128 KB in flight per SM: with six, the SMs' shares of the bandwidth drift apart (28 to 41 us for equal
// ranges, against 33 to 38 us), and the range that got least is what the step waits for.
constexpr int kQBufs = 3, kConsumers = 8, kFinishers = 3, kThreads = 32 * (kConsumers + kFinishers + 1);   // 12 warps: 168 registers a thread
template <int MT, int RS>
struct StreamSmem {
  static constexpr int kStages = 4;
  static_assert(kStages % 2 == 0, "see above");
  static constexpr int kQBytes = 16 * MT * kGqaQStride * 2;
  static constexpr int kQ = kStages * kGqaStageBytes;                       // kQBufs buffers, pieces in turn
  static constexpr int kState = kQ + kQBufs * kQBytes;                           // [kStateBufs][8 warps][RS][kGqaStateStride] f32
  static constexpr int kStateBufs = RS == 8 ? 2 : 1;
  static constexpr int kStateFloats = kConsumers * RS * kGqaStateStride;
  static constexpr int kBar = kState + kStateBufs * kStateFloats * 4;
  static constexpr int kTotal = 1024 + kBar + (2 * kStages + kQBufs + 6) * 8 + 16;
  static_assert(kTotal <= 232448, "more shared memory than a CTA may use");
};

__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

template <int MT, int RS, int N>
__global__ void __launch_bounds__(kThreads, 1) gqa_stream_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ GqaStreamParams<N> prm) {
  using SM = StreamSmem<MT, RS>;
  constexpr int kStages = SM::kStages;
  const GqaStreamCommon& c = prm.c;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* mb = (float*)(smem + SM::kState);
  uint64_t* full = (uint64_t*)(smem + SM::kBar);
  uint64_t* empty = full + kStages;
  uint64_t* q_full = empty + kStages;          // [kQBufs]: the queries of piece n are in buffer n % kQBufs
  constexpr int kStateBufs = SM::kStateBufs;
  uint64_t* state_full = q_full + kQBufs;      // [2]: the consumers' states of piece n are in buffer n % kStateBufs
  uint64_t* state_empty = state_full + 2;      // [2]: and have been read
  uint64_t* rows_done = state_empty + 2;       // the new rows of this CTA's pieces are in their pages
  uint64_t* merge_go = rows_done + 1;          // the finishers know which rows are to be merged here
  uint32_t* merge_flags = (uint32_t*)(merge_go + 1);   // [kFinishers], and the warps that are done with the merge
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  auto seq_of = [&](int i) -> GqaSeq { return c.seqs ? c.seqs[i] : prm.seqs[i]; };
  auto unit0_of = [&](int i) -> int { return c.seqs ? c.seqs[i].unit0 : prm.seqs[i].unit0; };
  // ranges: c.range units per worker, one more for the first c.range_more of them
  auto range_begin = [&](int w) -> int { return w * c.range + min(w, c.range_more); };
  auto worker_of = [&](int u) -> int {
    const int big = c.range_more * (c.range + 1);
    return u < big ? (int)((unsigned)u / (unsigned)(c.range + 1)) : c.range_more + (int)((unsigned)(u - big) / (unsigned)c.range);
  };
  const int u_begin = range_begin(blockIdx.x), u_end = range_begin(blockIdx.x + 1);
  // Every role walks this CTA's pieces: for (p = first_piece(); p.us < u_end; p = next_piece(p)).
  auto next_piece = [&](const Piece& q) -> Piece {
    Piece p = q;
    p.us += p.pages + kStreamUnits;
    if (++p.kvh == c.Hkv) {
      p.kvh = 0;
      p.i++;
      if (p.us < u_end) p.pages = unit0_of(p.i + 1) - unit0_of(p.i) - kStreamUnits;
    }
    p.pb = 0;
    p.pe = min(p.pages, u_end - p.us);
    return p;
  };
  auto first_piece = [&]() -> Piece {
    int lo = 0, hi = c.n_seqs;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (unit0_of(mid) * c.Hkv <= u_begin) lo = mid;
      else hi = mid;
    }
    Piece p;
    p.i = lo;
    const int n0 = unit0_of(lo), len = unit0_of(lo + 1) - n0;
    p.kvh = (u_begin - n0 * c.Hkv) / len;
    p.us = n0 * c.Hkv + p.kvh * len;
    p.pages = len - kStreamUnits;
    p.pb = u_begin - p.us;
    p.pe = min(p.pages, u_end - p.us);
    return p.pb < p.pages ? p : next_piece(p);   // a range may begin in the fixed-cost units of a stream
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], MT == 1 ? 4 : 8);   // the warps that read the page
    }
    for (int b = 0; b < kQBufs; b++) mbar_init(&q_full[b], kFinishers);
    for (int b = 0; b < kStateBufs; b++) {
      mbar_init(&state_full[b], kConsumers);
      mbar_init(&state_empty[b], kFinishers);
    }
    mbar_init(rows_done, kConsumers + kFinishers);
    mbar_init(merge_go, kFinishers);
    merge_flags[kFinishers] = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap);
  }
  for (int e = threadIdx.x; e < kQBufs * SM::kQBytes / 4; e += kThreads) reinterpret_cast<uint32_t*>(smem + SM::kQ)[e] = 0u;   // rows >= R stay zero
  __syncthreads();
  chain_release();
  if (c.seqs) chain_wait();   // the list is a copy that was queued just before this launch
  Piece p = first_piece();

  if (warp == kConsumers + kFinishers) {
    // ---------------- producer: TMA loads, new lengths ----------------
    const bool el = elect_one();
    const uint64_t evict_first = c.streams ? make_evict_first_policy() : 0;
    auto window = [&](const Piece& p, int seq, int first) -> int32_t {   // lane l holds the page id of logical page first + l
      int32_t pg = __ldg(c.table + (size_t)seq * c.table_stride + min(first + lane, p.pages - 1));
      if (pg < 0 || pg >= c.num_pages) {   // reported, and replaced by page 0 so that no load leaves the pool
        set_status(c.status, RELUX_ERR_BAD_PAGE);
        pg = 0;
      }
      return pg;
    };
    GqaSeq sq = seq_of(min(p.i, c.n_seqs - 1));
    int32_t win = p.us < u_end ? window(p, sq.seq, p.pb) : 0;   // the page table is written by host calls that wait for their copy
    chain_wait();
    int g = 0;
    bool ok = true, rows_ready = false;
    while (p.us < u_end && ok) {
      const int n_new = c.k_new ? (c.seqs ? c.seqs[p.i + 1].row0 : prm.seqs[p.i + 1].row0) - sq.row0 : 0;
      const int new_end = sq.len0 + n_new;
      int wfirst = p.pb;
      for (int page = p.pb; page < p.pe; page++, g++) {
        if (page - wfirst == 32) {
          wfirst = page;
          win = window(p, sq.seq, wfirst);
        }
        const int32_t pg = __shfl_sync(0xffffffffu, win, page - wfirst);
        const int st = g % kStages, k = g / kStages;
        if (k > 0 && !mbar_wait(&empty[st], (k - 1) & 1)) {
          set_status(c.status, RELUX_ERR_TIMEOUT);
          ok = false;
          break;
        }
        if (!rows_ready && page >= sq.len0 / kGqaPageTok && n_new > 0) {   // the first page that holds new rows
          rows_ready = true;
          if (!mbar_wait(rows_done, 0)) {
            set_status(c.status, RELUX_ERR_TIMEOUT);
            ok = false;
            break;
          }
        }
        if (el) {
          uint8_t* sb = smem + st * kGqaStageBytes;
          const int32_t krow = c.krow0 + (pg * c.Hkv + p.kvh) * kGqaPageTok;
          const int32_t vrow = c.vrow0 + (pg * c.Hkv + p.kvh) * kGqaPageTok;
          mbar_expect_tx(&full[st], kGqaStageBytes);
          if (c.streams) {
            tma_load_2d_hint(sb, &tmap, 0, krow, &full[st], evict_first);
            tma_load_2d_hint(sb + 8192, &tmap, 64, krow, &full[st], evict_first);
            tma_load_2d_hint(sb + 16384, &tmap, 0, vrow, &full[st], evict_first);
            tma_load_2d_hint(sb + 24576, &tmap, 64, vrow, &full[st], evict_first);
          } else {
            tma_load_2d(sb, &tmap, 0, krow, &full[st]);
            tma_load_2d(sb + 8192, &tmap, 64, krow, &full[st]);
            tma_load_2d(sb + 16384, &tmap, 0, vrow, &full[st]);
            tma_load_2d(sb + 24576, &tmap, 64, vrow, &full[st]);
          }
        }
        __syncwarp();
      }
      if (c.advance && p.kvh == 0 && p.pe == p.pages && lane == 0) c.len[sq.seq] = new_end;
      p = next_piece(p);
      if (p.us < u_end) {
        sq = seq_of(p.i);
        win = window(p, sq.seq, 0);
      }
    }
    return;
  }

  auto timed_wait = [&](uint64_t* bar, int parity) -> bool {
    if (mbar_wait(bar, parity)) return true;
    set_status(c.status, RELUX_ERR_TIMEOUT);
    return false;
  };

  auto store_out = [&](const Piece& q, int r, float4 o) {
    const int s = r / c.g, hq = r - s * c.g;
    const size_t off = (((size_t)q.i * c.S + s) * c.H + (size_t)q.kvh * c.g + hq) * kGqaD + lane * 4;
    if (c.out_bf16) *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(c.out) + off) = make_uint2(pack_bf16x2(o.x, o.y), pack_bf16x2(o.z, o.w));
    else *reinterpret_cast<float4*>(reinterpret_cast<float*>(c.out) + off) = o;
  };
  // All new rows of this CTA's pieces, a piece per warp in turn: 16 lanes write a K row, 16 the V row, 16 bytes each.  By every
  // warp that would wait for the first page now: the loads of a stream's last page wait for all of them, and three warps took
  // 5 us over the pieces of a range of short streams.  (Written by the producer when it reached their page, every short stream
  // cost it two memory latencies.)
  auto write_new_rows = [&]() {
    if (!c.k_new) return;
    int k = 0;
    for (Piece q = p; q.us < u_end; q = next_piece(q), k++) {
      if (k % (kConsumers + kFinishers) != warp) continue;
      const GqaSeq sq = seq_of(q.i);
      const int n_new = (c.seqs ? c.seqs[q.i + 1].row0 : prm.seqs[q.i + 1].row0) - sq.row0;
      const int v = lane >> 4, ch = (lane & 15) * 8;
      const void* from = v ? c.v_new : c.k_new;
      const int r_hi = min(sq.len0 + n_new, q.pe * kGqaPageTok);
      for (int pos = max(sq.len0, q.pb * kGqaPageTok); pos < r_hi; pos++) {
        const int32_t pg = __ldg(c.table + (size_t)sq.seq * c.table_stride + pos / kGqaPageTok);
        const int idx = pos - sq.len0;
        const size_t src = c.head_major ? (size_t)sq.row0 * c.Hkv * kGqaD + ((size_t)q.kvh * n_new + idx) * kGqaD + ch
                                        : ((size_t)(sq.row0 + idx) * c.Hkv + q.kvh) * kGqaD + ch;
        uint4 w;
        if (c.new_f32) {
          const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(from) + src);
          const float4 a = s[0], b = s[1];
          w = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
        } else {
          w = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(from) + src);
        }
        if (pg < 0 || pg >= c.num_pages) continue;   // reported by the producer
        uint16_t* dst = (v ? c.v_base : c.k_base) + (((size_t)pg * c.Hkv + q.kvh) * kGqaPageTok + (pos & (kGqaPageTok - 1))) * kGqaD + ch;
        *reinterpret_cast<uint4*>(dst) = w;
      }
    }
    fence_proxy_async_all();   // the rows are read back by the producer's TMA loads
    __syncwarp();
    if (lane == 0) mbar_arrive(rows_done);
  };
  const Piece p_first = p;
  Piece p_last = p;
  if (warp < kConsumers) {
    // ---------------- consumers ----------------
    const int grp = warp >> 2, tb = (warp & 3) * 16;   // this warp's tokens inside a page
    const int row0 = MT == 1 ? 0 : grp * 16;           // first query row of this warp
    chain_wait();
    write_new_rows();
    int g = 0, n = 0;
    bool alive = true;
    for (; p.us < u_end; p_last = p, p = next_piece(p), n++) {
      const GqaSeq sq = seq_of(p.i);
      const int n_new = c.advance && c.k_new ? (c.seqs ? c.seqs[p.i + 1].row0 : prm.seqs[p.i + 1].row0) - sq.row0 : 0;
      const int T = sq.len0 + n_new + c.extra;
      if (alive) alive = timed_wait(&q_full[n % kQBufs], (n / kQBufs) & 1);
      uint32_t qa[1][8][4];
      gqa_load_q<1>(qa, reinterpret_cast<const uint16_t*>(smem + SM::kQ + (n % kQBufs) * SM::kQBytes) + row0 * kGqaQStride, lane);
      GqaState<1> state;
      state.clear();
      for (int page = p.pb; page < p.pe; page++, g++) {
        if (MT == 1 && (g & 1) != grp) continue;
        const int st = g % kStages;
        if (alive) alive = timed_wait(&full[st], (g / kStages) & 1);
        if (alive) {
          gqa_consume_page<1>(state, qa, smem_u32(smem + st * kGqaStageBytes), tb, page * kGqaPageTok + tb, T, c.S, c.g, c.causal,
                              c.scale_log2, lane, row0);
          __syncwarp();
          if (lane == 0) mbar_arrive(&empty[st]);
        }
      }
      const int sb = n % kStateBufs;
      if (n >= kStateBufs && alive) alive = timed_wait(&state_empty[sb], (n / kStateBufs - 1) & 1);
      gqa_store_state<1>(state, mb + sb * SM::kStateFloats + (size_t)warp * RS * kGqaStateStride, RS, lane, alive);
      __syncwarp();
      if (lane == 0) mbar_arrive(&state_full[sb]);
    }
  } else {
    // ---------------- finishers ----------------
    const int fw = warp - kConsumers, ft = threadIdx.x - 32 * kConsumers;
    // Q rows of a piece's kv head as bf16 into buffer b; row r = s * g + head in group
    auto load_queries = [&](const Piece& q, int b) {
      uint16_t* qs = reinterpret_cast<uint16_t*>(smem + SM::kQ + b * SM::kQBytes);
      constexpr int kAtOnce = 3;   // loads in flight per thread
      const int total = c.R * (kGqaD / 8);
      for (int e0 = ft; e0 < total; e0 += kAtOnce * 32 * kFinishers) {
        uint4 w[kAtOnce];
#pragma unroll
        for (int k = 0; k < kAtOnce; k++) {
          const int e = e0 + k * 32 * kFinishers;
          if (e >= total) break;
          const int r = e >> 4, ch = (e & 15) * 8;
          const int s = r / c.g, hq = r - s * c.g;
          const size_t off = (((size_t)q.i * c.S + s) * c.H + (size_t)q.kvh * c.g + hq) * kGqaD + ch;
          if (c.q_bf16) {
            w[k] = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(c.q) + off);
          } else {
            const float4* f = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(c.q) + off);
            const float4 a = f[0], b2 = f[1];
            w[k] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b2.x, b2.y), pack_bf16x2(b2.z, b2.w));
          }
        }
#pragma unroll
        for (int k = 0; k < kAtOnce; k++) {
          const int e = e0 + k * 32 * kFinishers;
          if (e < total) *reinterpret_cast<uint4*>(qs + (e >> 4) * kGqaQStride + (e & 15) * 8) = w[k];
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[b]);
    };
    chain_wait();
    if (ft == 0) stamp_begin(c.time);
    Piece p_ahead = p;   // the next piece whose queries have not been requested
    for (int b = 0; b < 2 && p_ahead.us < u_end; b++, p_ahead = next_piece(p_ahead)) load_queries(p_ahead, b);
    write_new_rows();
    // The pieces of a stream are one each of the workers w0 .. w1, and a row belongs to the same finisher warp in all of
    // them: each warp counts for itself (no block-wide barrier), and the warp that counts last merges its own rows of all of
    // them.  (The fence takes up to 10 us under full load; the query buffers cover it.)
    auto publish = [&](const Piece& pc) -> bool {
      uint32_t last = 0;
      if (lane == 0) {
        __threadfence();
        uint32_t* ctr = c.done + ((size_t)pc.i * c.Hkv + pc.kvh) * kFinishers + fw;
        last = atomicAdd(ctr, 1u) == (uint32_t)(worker_of(pc.us + pc.pages - 1) - worker_of(pc.us));
        if (last) *ctr = 0u;
        __threadfence();
      }
      return __shfl_sync(0xffffffffu, last, 0) != 0;
    };
    int n = 0;
    bool alive = true;
    uint32_t due = 0;   // bit 0: this warp's rows of the range's first piece are to be merged here, bit 1: of its last
    for (; p.us < u_end; p_last = p, p = next_piece(p), n++) {
      if (p_ahead.us < u_end) {   // two pieces ahead; that buffer was last read for piece n - 1, whose states have arrived
        load_queries(p_ahead, (n + 2) % kQBufs);
        p_ahead = next_piece(p_ahead);
      }
      if (alive) alive = timed_wait(&state_full[n % kStateBufs], (n / kStateBufs) & 1);
      // combine the warps' states: a warp per row, four dims per lane
      const bool whole = p.pb == 0 && p.pe == p.pages;
      const int slot = 2 * (int)blockIdx.x + (p.us + p.pb == u_begin ? 0 : 1);
      constexpr int kW = MT == 1 ? 8 : 4;   // warps that hold a state of a row
      // two rows at a time: a row is a chain of shuffles, about 1.1 us whatever its loads
      const float* states = mb + (n % kStateBufs) * SM::kStateFloats;
#pragma unroll 1
      for (int r0 = fw; r0 < c.R; r0 += 2 * kFinishers) {
        const int r1 = r0 + kFinishers < c.R ? r0 + kFinishers : r0;   // the same row twice where there is no second
        const float* src[2];
        float M[2], L[2], wgt[2];
        float4 o[2];
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const int r = k ? r1 : r0;
          src[k] = states + ((size_t)(MT == 1 ? 0 : (r >> 4) * 4) * RS + (MT == 1 ? r : (r & 15))) * kGqaStateStride;
          // lane j (mod kW) weighs warp j's state
          const float2 ml = *reinterpret_cast<const float2*>(src[k] + (size_t)(lane & (kW - 1)) * RS * kGqaStateStride + kGqaD);
          M[k] = ml.x;
          L[k] = ml.y;
          wgt[k] = ml.x;
          o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 1; i < kW; i <<= 1)
#pragma unroll
          for (int k = 0; k < 2; k++) M[k] = fmaxf(M[k], __shfl_xor_sync(0xffffffffu, M[k], i));
#pragma unroll
        for (int k = 0; k < 2; k++) {
          wgt[k] = wgt[k] == -INFINITY ? 0.f : gqa_ex2(wgt[k] - M[k]);
          L[k] *= wgt[k];
        }
#pragma unroll
        for (int i = 1; i < kW; i <<= 1)
#pragma unroll
          for (int k = 0; k < 2; k++) L[k] += __shfl_xor_sync(0xffffffffu, L[k], i);
#pragma unroll
        for (int w = 0; w < kW; w++)
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const float f = __shfl_sync(0xffffffffu, wgt[k], w);
            const float4 x = *reinterpret_cast<const float4*>(src[k] + (size_t)w * RS * kGqaStateStride + lane * 4);
            o[k].x = fmaf(x.x, f, o[k].x); o[k].y = fmaf(x.y, f, o[k].y); o[k].z = fmaf(x.z, f, o[k].z); o[k].w = fmaf(x.w, f, o[k].w);
          }
#pragma unroll
        for (int k = 0; k < 2; k++) {
          const int r = k ? r1 : r0;
          if (k && r1 == r0) break;
          if (whole) {
            const float inv = (L[k] > 0.f) ? 1.f / L[k] : 0.f;
            store_out(p, r, make_float4(o[k].x * inv, o[k].y * inv, o[k].z * inv, o[k].w * inv));
          } else {
            const size_t row = (size_t)slot * c.R + r;
            __stcg(reinterpret_cast<float4*>(c.part_o + row * kGqaD + lane * 4), o[k]);
            if (lane == 0) __stcg(reinterpret_cast<float2*>(c.part_ml + row * 2), make_float2(M[k], L[k]));
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&state_empty[n % kStateBufs]);
      if (!whole && publish(p)) due |= p.us + p.pb == p_first.us + p_first.pb ? 1u : 2u;
    }
    if (lane == 0) {
      merge_flags[fw] = due;
      mbar_arrive(merge_go);
    }
  }

  // ---------------- merge of split streams: consumers and finishers, a row per warp ----------------
  // A row's arithmetic is a chain of shuffles and a division, about 1.1 us whatever its loads; three warps took 3-12 us.
  // One row of a piece's stream: all partials of it, in range order.
  auto merge_row = [&](const Piece& pc, int r) {
    const int w0 = worker_of(pc.us), np = worker_of(pc.us + pc.pages - 1) - w0 + 1;
    // the partial of worker w0 + j lies in slot 2 (w0 + j), but for w0's own when its range begins before the stream
    const int stride = 2 * c.R, first = range_begin(w0) == pc.us ? 0 : c.R;   // in rows
    const float2* ml0 = reinterpret_cast<const float2*>(c.part_ml) + (size_t)w0 * stride;
    const float4* o0 = reinterpret_cast<const float4*>(c.part_o) + (size_t)w0 * stride * (kGqaD / 4) + lane;
    auto ml_of = [&](int j, int r) -> float2 {
      return (j < np && r < c.R) ? __ldcg(ml0 + (j ? j * stride : first) + r) : make_float2(-INFINITY, 0.f);
    };
    auto o_of = [&](int j, int r) -> float4 {
      return (j < np && r < c.R) ? __ldcg(o0 + ((j ? j * stride : first) + r) * (kGqaD / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    float2 ml = ml_of(lane, r);
    float M = ml.x, L = 0.f;
#pragma unroll 1
    for (int j = 32 + lane; j < np; j += 32) M = fmaxf(M, ml_of(j, r).x);
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float w = 0.f;
#pragma unroll 1
    for (int j = 0; j < np; j += 8) {
      float4 x[8];
#pragma unroll
      for (int q = 0; q < 8; q++) x[q] = o_of(j + q, r);
      if ((j & 31) == 0) {   // the weights of the next 32 partials, one per lane
        if (j == 0) M = warp_max(M);
        else ml = ml_of(j + lane, r);
        w = (ml.x == -INFINITY) ? 0.f : gqa_ex2(ml.x - M);
        L += ml.y * w;
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const float f = __shfl_sync(0xffffffffu, w, (j + q) & 31);
        o.x = fmaf(x[q].x, f, o.x); o.y = fmaf(x[q].y, f, o.y);
        o.z = fmaf(x[q].z, f, o.z); o.w = fmaf(x[q].w, f, o.w);
      }
    }
    L = warp_sum(L);
    const float inv = (L > 0.f) ? 1.f / L : 0.f;
    store_out(pc, r, make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv));
  };
  timed_wait(merge_go, 0);
#pragma unroll 1
  for (int e = warp; e < 2 * c.R; e += kConsumers + kFinishers) {
    const int k = e >= c.R, r = k ? e - c.R : e;
    if (merge_flags[r % kFinishers] >> k & 1u) merge_row(k ? p_last : p_first, r);
  }
  if (lane == 0 && atomicAdd(&merge_flags[kFinishers], 1u) == kConsumers + kFinishers - 1) stamp_end(c.time);   // the last of them
  if (c.out_bf16) fence_chained_writes();   // a projection's operand
}


template <int MT, int RS, int N>
int32_t launch(Pool* p, const GqaStreamCommon& c, const GqaSeq* seqs, int workers) {
  using SM = StreamSmem<MT, RS>;
  GqaStreamParams<N> prm;
  prm.c = c;
  if (!c.seqs) memcpy(prm.seqs, seqs, sizeof(GqaSeq) * ((size_t)c.n_seqs + 1));
  if (int32_t rc = allow_smem(p->dev, gqa_stream_kernel<MT, RS, N>, SM::kTotal)) return rc;
  RELUX_CUDA_TRY(launch_chained(p->tune.get(RELUX_TUNE_CHAINED_LAUNCHES) != 0, gqa_stream_kernel<MT, RS, N>, dim3(workers), dim3(kThreads),
                                (size_t)SM::kTotal, p->dev->stream, p->tmap_gqa, prm));
  time_stamp_done(p->attn_times, c.time);
  count_launch(p->dev);
  return RELUX_OK;
}
template <int N>
int32_t launch_rows(Pool* p, const GqaStreamCommon& c, const GqaSeq* seqs, int workers) {
  if (c.R <= 8) return launch<1, 8, N>(p, c, seqs, workers);
  if (c.R <= 16) return launch<1, 16, N>(p, c, seqs, workers);
  return launch<2, 16, N>(p, c, seqs, workers);
}

}  // namespace

bool gqa_stream_eligible(const Pool* p, const relux_attn_args& a) {
  const relux_pool_params& prm = p->prm;
  const int g = a.num_heads / std::max(1, prm.gqa_num_kv_heads);
  return p->has_tmap && prm.page_tokens == kGqaPageTok && prm.gqa_head_dim == kGqaD && g >= 1 && g <= 32 && a.q_tokens >= 1 &&
         a.q_tokens <= 32 / g;
}

// A step's new rows can ride in the attention launch: the pages it loads must cover them (rows past the visible tokens of
// a sequence would be nobody's), and the bookkeeping of reference-compat pools stays with the plain append.
bool gqa_append_fusable(const Pool* p, const relux_attn_args& a, int max_new_rows, bool advance) {
  return !p->compat && a.mode == RELUX_ATTN_FAST && gqa_stream_eligible(p, a) && (advance || max_new_rows <= a.extra_tokens);
}

// q: device [n][S][H][128] token-major (f32 or bf16).  out: device, same shape, f32 or bf16.  With `app` (advance = 1) the
// host lengths already count the new rows.
int32_t launch_gqa_stream(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const void* d_q, void* d_out, bool out_bf16,
                          const GqaAppend* app) {
  const relux_pool_params& prm = p->prm;
  const int n = sb.n_seqs, Hkv = prm.gqa_num_kv_heads, g = a.num_heads / Hkv, R = g * a.q_tokens;
  GqaStreamCommon c{};
  GqaSeq inl[kInlineLarge + 1];
  GqaSeq* seqs = inl;
  int slot_index = 0;
  if (n > kInlineLarge) {
    int32_t* slot = nullptr;
    if (int32_t rc = stage_acquire(p, &slot, &slot_index)) return rc;
    seqs = (GqaSeq*)slot;
  }
  int64_t units64 = 0;
  int rows = 0;
  for (int i = 0; i < n; i++) {
    const int s = sb.seq[i], len = p->h_len[(size_t)a.layer * prm.max_seqs + s], n_new = app ? app->rows[i] : 0;
    seqs[i] = GqaSeq{s, app && app->advance ? len - n_new : len, (int32_t)units64, rows};
    units64 += (len + a.extra_tokens + kGqaPageTok - 1) / kGqaPageTok + kStreamUnits;
    rows += n_new;
  }
  seqs[n] = GqaSeq{0, 0, (int32_t)units64, rows};
  units64 *= Hkv;
  if (units64 >= ((int64_t)1 << 31)) { set_error("more cached pages than one attention launch addresses"); return RELUX_ERR_UNSUPPORTED; }
  const int units = (int)units64;
  // One range per SM; ranges of fewer than two units do not pay for their share of the merge.  Where streams are a page or two,
  // some ranges hold no page and their CTAs leave at once; that costs nothing: one sequence of 60 to 120 tokens, 8 kv heads, takes
  // 4.1 us on 20 or 24 CTAs, and 6.1 with one unit a stream, whose ranges split the two pages.
  int workers = std::max(1, std::min(p->dev->sm_count, units / 2));
  if (const int ov = p->tune.get(RELUX_TUNE_CHUNK_PAGES)) workers = std::max(1, std::min(units, (units + ov - 1) / ov));   // tuning knob
  const size_t part_rows = (size_t)2 * workers * R;
  int32_t rc = grow(p->dev, p->part_o, part_rows * (kGqaD + 2) * sizeof(float));
  if (rc) return rc;
  const size_t ctr_bytes = (size_t)n * Hkv * kFinishers * sizeof(uint32_t);
  if (ctr_bytes > p->stream_done.cap) {
    if ((rc = grow(p->dev, p->stream_done, ctr_bytes))) return rc;
    RELUX_CUDA_TRY(cudaMemsetAsync(p->stream_done.p, 0, p->stream_done.cap, p->dev->stream));
  }
  if (seqs != inl) {
    const size_t bytes = sizeof(GqaSeq) * ((size_t)n + 1);
    if ((rc = grow(p->dev, p->seq_list, bytes))) return rc;
    RELUX_CUDA_TRY(cudaMemcpyAsync(p->seq_list.p, seqs, bytes, cudaMemcpyHostToDevice, p->dev->stream));
    if ((rc = stage_release(p, slot_index))) return rc;
    c.seqs = (const GqaSeq*)p->seq_list.p;
  }
  c.table = p->d_table;
  c.table_stride = prm.max_pages_per_seq;
  c.num_pages = prm.num_pages;
  c.n_seqs = n;
  c.range = units / workers;
  c.range_more = units % workers;
  c.Hkv = Hkv;
  c.H = a.num_heads;
  c.g = g;
  c.S = a.q_tokens;
  c.R = R;
  c.extra = a.extra_tokens;
  c.causal = a.causal;
  const int64_t rows_per_block = (int64_t)prm.num_pages * Hkv * kGqaPageTok;
  c.krow0 = (int32_t)((int64_t)a.layer * 2 * rows_per_block);
  c.vrow0 = (int32_t)((int64_t)a.layer * 2 * rows_per_block + rows_per_block);
  c.streams = (units64 - (int64_t)kStreamUnits * n * Hkv) * kGqaStageBytes > kResidentBytes;
  c.scale_log2 = a.scale * 1.4426950408889634f;
  c.q = d_q;
  c.q_bf16 = a.q_dtype == RELUX_DTYPE_BF16;
  c.out_bf16 = out_bf16;
  c.out = d_out;
  c.part_o = (float*)p->part_o.p;
  c.part_ml = c.part_o + part_rows * kGqaD;
  c.done = (uint32_t*)p->stream_done.p;
  if (app && rows > 0) {
    c.k_new = app->k;
    c.v_new = app->v;
    c.new_f32 = app->dtype == RELUX_DTYPE_F32;
    c.head_major = app->layout == RELUX_LAYOUT_HEAD_MAJOR;
    c.advance = app->advance;
  }
  c.k_base = p->storage + (size_t)a.layer * p->layer_elems;
  c.v_base = c.k_base + p->page_elems * prm.num_pages;
  c.len = p->d_len + (size_t)a.layer * prm.max_seqs;
  c.status = p->d_status;
  c.time = time_stamp_next(p, p->attn_times);
  return n <= kInlineSmall || c.seqs ? launch_rows<kInlineSmall>(p, c, seqs, workers) : launch_rows<kInlineLarge>(p, c, seqs, workers);
}

}  // namespace relux
