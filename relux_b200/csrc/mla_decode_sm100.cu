// Absorbed MLA flash-decode on the 5th-generation tensor cores (tcgen05 + TMEM), fed by TMA page loads.
// Shape: 128 query heads, latent 512, rope key 64 (row = 576 bf16 = 1152 B), 64-token pages.
//
// Why a CTA PAIR per worker.  The 128 heads that share one latent row are the M dimension of both
// contractions (S = Q~ K^T, O = P C).  O alone is 128 x 512 f32 = all 512 TMEM columns of one SM, and
// Q~ (128 x 576 bf16 = 144 KB) would leave no shared memory for KV tiles.  With cta_group::2 each CTA owns
// 64 heads: Q~ is 72 KB per CTA, O is 64 x 512 f32 = 256 TMEM columns (lanes 0-63 hold output dims
// [0,128) of each 256-wide block, lanes 64-127 dims [128,256)), and the B operand (the KV rows) is split between
// the two CTAs' shared memories and read by both tensor cores.  No TMA multicast is used anywhere: each CTA
// issues its own loads (`.cta_group::2` only routes the completion bytes to the leader's mbarrier).
//
// Persistent workers over a stream partition (or, short calls, a piece of one sequence each: cheapest_plan in stream_plan.h).  The pages of all sequences of the call, laid end to end, are cut
// into as many equal ranges as CTA pairs fit on the GPU; a worker (one pair) walks its range once.  An ITEM is
// the part of one sequence inside one range, so a worker changes item (new Q~, new accumulator, one split-KV
// partial written) only where a sequence ends inside its range.  The tile pipeline does not drain at an item
// boundary: Q~ of the next item is loaded as soon as the last QK^T of the current one has completed, and the
// first QK^T of the next item is issued right behind the last PV of the current one.
//
// Per 128-token tile (two pages; page r of the tile belongs to CTA r):
//   S[128 x 128]  = Q~[128 x 576] . K[128 tok x 576]^T      36 MMAs M128 N128 K16, K-major A and B
//   softmax warps : S from TMEM -> scaled exp2 with a lazily updated running max -> P (bf16) to shared memory
//   O[128 x 512] += P[128 x 128 tok] . C[128 tok x 512]      16 MMAs M128 N256 K16, B is MN-major (the same
//                                                              row-major page data, read "transposed" by descriptor)
// Shared memory per CTA: Q~ 72 KB | K slots 9 x 8 KB (own page, 64-dim column blocks) | V slots 4 x 16 KB
// (both pages x own 256 output dims) | P 16 KB | barriers.  Every slot has a full barrier (in the leader CTA,
// counting the bytes of both CTAs' loads) and an empty barrier (in each CTA, armed by tcgen05.commit multicast).
// Tiles are numbered g = 0, 1, ... over the worker's whole range; every barrier completes one phase per tile
// (s_full[b] one per tile with g & 1 == b; q_full one per item), which gives all wait parities.
// Issue order of the MMA warp: QK(0); then for each tile g: QK(g+1), PV(g) -- so the softmax of tile g+1
// overlaps PV(g) and QK(g+2).
//
// All waits are bounded; a wait that runs out sets RELUX_ERR_TIMEOUT in the status word, raises a shared abort
// flag so the other warps stop waiting too, and the CTA pair still meets at the final cluster barrier and frees
// its tensor memory.
#include <algorithm>
#include <cstdlib>
#include <cuda_bf16.h>
#include "common.cuh"
#include "internal.h"
#include "splitkv.h"
#include "softmax_parts.cuh"
#include "umma.cuh"

namespace relux {

namespace {

constexpr int kMaxHeads = 128, kDC = 512, kDR = 64, kRow = kDC + kDR;  // 576
constexpr int kPage = 64;
constexpr int kBlk = 8192;                  // one [64 rows x 64 cols] bf16 block, 128-byte swizzled
constexpr int kNumKB = kRow / 64;           // 9 column blocks per row
constexpr int kSmemQ = 0;
constexpr int kSmemK = kSmemQ + kNumKB * kBlk;        // 73728
constexpr int kSmemV = kSmemK + kNumKB * kBlk;        // 147456
constexpr int kSmemP = kSmemV + 4 * 2 * kBlk;         // 212992
constexpr int kSmemBar = kSmemP + 2 * kBlk;           // 229376
constexpr int kSmemTotal = kSmemBar + 2048;           // 231424 of the 232448 bytes a CTA may use
constexpr int kKGroups = 3, kKPerGroup = kNumKB / kKGroups;  // K slots are armed / released in groups of 3 blocks
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kTmemO = 0, kTmemS = 256;          // O: 2 x 128 columns; S: 2 buffers x 64 columns
constexpr float kRescaleThreshold = 8.0f;             // log2 units: rescale O only when the max grew by > 2^8
constexpr int kPrefetchTiles = 2;                     // of a worker's end, before which it asks for its share of W_UV
constexpr int kMaxInterleavedQ = 8;                   // up to this many query tokens work side by side on one range

struct Bars {
  uint64_t k_full[kKGroups], k_empty[kKGroups];
  uint64_t v_full[4], v_empty[4];
  uint64_t s_full[2];
  uint64_t p_full, pv_done, q_full;
  uint32_t tmem_base;
  volatile int32_t abort_flag;
  float rowmax[2][2][64];   // [tile parity][token half][row]
  float lsum[128];                    // an item's row sums, of both halves of the tokens
};
static_assert(sizeof(Bars) <= 2048, "barrier block too large");

struct MlaSm100Params {
  const StreamItem* items;
  const int32_t* worker_first;   // [workers + 1]
  const int32_t* table;
  int32_t table_stride;
  int32_t num_pages, S, sx, causal;   // sx: query tokens interleaved along grid x (their workers share the range through L2)
  int32_t H;                          // query heads, <= 128: the M = 128 tile is padded with whatever rows follow in q~
                                      // (finite values, computed and thrown away; rows past the end of q~ are zero-filled by TMA)
  int32_t layer_row0;
  float scale_log2;
  int32_t form;                       // of the partial rows (PartialForm)
  void* part_o;
  float* part_ml;
  const uint8_t* w_uv;                // brought into L2 while the last tiles run, w_uv_each bytes a CTA (0: they will be there)
  uint32_t w_uv_bytes, w_uv_each;
  int32_t* status;
  TimeStamp time;
};

// Bounded wait.  The common case (phase already complete) is a single try_wait.  When the bound runs out the
// waiter records RELUX_ERR_TIMEOUT, raises the CTA's abort flag and RETURNS: nobody leaves a loop early, every
// later wait sees the flag on its first failed poll and returns at once, so all warps still reach the named
// barriers and the final cluster barrier with garbage results and a non-zero status word.
__device__ __noinline__ void wait_slow(uint64_t* bar, uint32_t parity, Bars* b, int32_t* status) {
  for (uint32_t i = 0; i < kSpinLimit; i++) {
    if (mbar_try_wait(bar, parity)) return;
    if ((i & 255) == 255 && b->abort_flag) return;
    if (i > 512) __nanosleep(20);
  }
  b->abort_flag = 1;
  set_status(status, RELUX_ERR_TIMEOUT);
}
__device__ __forceinline__ void wait_bar(uint64_t* bar, uint32_t parity, Bars* b, int32_t* status) {
  if (!mbar_try_wait(bar, parity)) wait_slow(bar, parity, b, status);
}

__device__ __forceinline__ StreamItem load_item(const StreamItem* p) {
  const int4 a = load_chained(reinterpret_cast<const int4*>(p));
  const int4 b = load_chained(reinterpret_cast<const int4*>(p) + 1);
  StreamItem it;
  it.seq_index = a.x; it.seq = a.y; it.page_begin = a.z; it.page_end = a.w;
  it.tokens = b.x; it.first = b.y; it.n = b.z; it.pad = 0;
  return it;
}

// The same from the arguments.
__device__ __forceinline__ StreamItem listed_item(const ListedItem& l) {
  StreamItem it;
  it.seq_index = l.seq_index; it.seq = l.seq; it.page_begin = l.page_begin; it.page_end = l.page_end;
  it.tokens = l.tokens; it.first = l.first; it.n = l.n; it.pad = 0;
  return it;
}

// Page ids of an item as the producer warp holds them: lane l keeps the first pool row (TMA y coordinate) of
// pages 32 * blk + l (`cur`) and 32 * (blk + 1) + l (`nxt`); positions past the item's last page repeat the last page.
struct PageWin {
  int32_t cur, nxt, blk;
};

// The partial result of a warp: its 32 rows (heads) x 256 of the 512 latent columns of O, in eight chunks of 16 rows x 64 columns.  The
// 16x256b loads give four lanes a row.  What a row is, kForm says.  The bf16 forms are operands of the up-projection: every 32 columns in
// the order in which a lane holds them, column 8 i + 2 q + e at place 8 q + 2 i + e (mla_vup_pieces_kernel loads W_UV's rows in that
// order), and a chunk passes through 4 KB of the P tile that belong to the warp, so that its stores are whole lines and no warp waits for
// another.  Two halves (hi = the upper 16 bits of x, lo = bf16(x - hi), which is off by less than 2^-16 of x) where rows have several
// pieces.  Where every row has one, that is its whole attention: over its sum (`l_row`) it is the up-projection's operand, and is rounded to bf16
// here, float32 up to then.  (Rounded ahead of the norm, the error was 0.997-1.002 times as large.)  merge_splits_kernel reads float32.
// Bound: an SM writes 32 bytes a clock, whether by stores of whole lines (128 KB in 4.0 k clocks, one CTA or all) or by TMA (4.3-5.2 k);
// stores of 64 bytes a row take twice as long, and so did 64 TMA stores of 2 KB.  An
// item takes 3.1 us as two halves, as it did in float32, and 1.8 in one.
template <int kForm>
__device__ __forceinline__ void write_partial(uint8_t* smem, uint32_t tmem_o, void* part_o, int H, int piece, int head0, float m_used, float l_row, bool ok) {
  constexpr int kRowElems = kForm == kPartialOne ? kDC : 2 * kDC;   // bf16 forms
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3;
  // The partial results (256 KB an item at 128 heads: 17 MB in 64 pieces, 36 MB in 138 items of ranges) wait for the merge while cached
  // rows stream through L2, and came back from HBM: stored to be evicted last, a step of 64 x 4096 takes 89.2 us instead of 90.5, 40 x
  // <= 2500 45.2 instead of 46.2, 20 x 16000 94.5 instead of 95.8; shorter ones the same.  They stay while the pool is in use: a program's
  // own pass over 96 MB behind a step of 64 x 1000 then takes 40 us instead of 37.5 (48 MB: no difference), and no less with a merge that
  // reads them to be evicted first, which itself takes 1 us longer.  (Cached rows loaded to be evicted first were gone before their second
  // load, as values: 114 -> 127 us.)
  const uint64_t policy = make_evict_last_policy();
  uint8_t* stage = smem + kSmemP + warp * 4096;
  // two rows of 64 bytes to every eight lanes that write, one of 128 to every eight that read: no bank twice either way
  auto place = [](int row, int chunk16) { return (uint32_t)(row * 128 + ((chunk16 ^ ((row & 1) << 2 | (row >> 1 & 3))) << 4)); };
  uint32_t v[32];
  auto load = [&](int u) { tmem_ld_16x256b_x8(tmem_o + ((uint32_t)(warp * 32 + (u >> 2) * 16) << 16) + (u & 3) * 64, v); };
  load(0);
  float norms[4] = {1.f, 1.f, 1.f, 1.f};   // of this lane's rows
  if constexpr (kForm == kPartialOne) {
    const float norm = l_row > 0.f ? rcp_normal(l_row) : 0.f;
#pragma unroll
    for (int k = 0; k < 4; k++) norms[k] = __shfl_sync(0xffffffffu, norm, (lane >> 2) + 8 * k);
  }
#pragma unroll 1
  for (int u = 0; u < 8; u++) {   // 4 * (half of the rows) + 64-column chunk
    tmem_ld_wait_for(v);
    const int dim = 128 * (warp >> 1) + 256 * ((u & 3) >> 1) + 64 * (u & 1);
    const int head = head0 + (warp & 1) * 32 + (u >> 2) * 16;   // the chunk's first
    if constexpr (kForm == kPartialFloat32) {
      const int r32 = (u >> 2) * 16 + (lane >> 2);              // of the warp's 32 rows, the first of this lane's two
      const bool seen[2] = {ok && __shfl_sync(0xffffffffu, m_used, r32) != -INFINITY,   // a row without a visible key is zero
                            ok && __shfl_sync(0xffffffffu, m_used, r32 + 8) != -INFINITY};
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int r = head + (lane >> 2) + 8 * k;
        if (r >= H) continue;
        float* dst = reinterpret_cast<float*>(part_o) + ((size_t)piece * H + r) * kDC + dim + 2 * q;
#pragma unroll
        for (int i = 0; i < 8; i++)
          *reinterpret_cast<uint2*>(dst + 8 * i) = seen[k] ? make_uint2(v[4 * i + 2 * k], v[4 * i + 2 * k + 1]) : make_uint2(0u, 0u);
      }
      if (u < 7) load(u + 1);
    } else {
      // A row without a visible key may hold anything: the up-projection leaves it out by its maximum.
      uint32_t hi[16], lo[16];   // [row of two][32 columns of two][4]
      float big[4] = {0.f, 0.f, 0.f, 0.f};
      const float na = u < 4 ? norms[0] : norms[2], nb = u < 4 ? norms[1] : norms[3];
      const uint64_t norm2[2] = {pack2(na, na), pack2(nb, nb)};
#pragma unroll
      for (int w = 0; w < 16; w++) {
        const uint32_t x = v[4 * (w & 7) + 2 * (w >> 3)], y = v[4 * (w & 7) + 2 * (w >> 3) + 1];
        if constexpr (kForm == kPartialOne) {
          float a, b;
          unpack2(mul2(pack2(__uint_as_float(x), __uint_as_float(y)), norm2[w >> 3]), a, b);
          hi[w] = round_bf16x2(a, b);
        } else {
          hi[w] = __byte_perm(x, y, 0x7632);
          lo[w] = round_bf16x2(__uint_as_float(x) - bf16_hi(x), __uint_as_float(y) - bf16_hi(y));
          big[w & 3] = max3(big[w & 3], fabsf(__uint_as_float(x)), fabsf(__uint_as_float(y)));
        }
      }
      if (kForm == kPartialHalves && fmaxf(fmaxf(big[0], big[1]), fmaxf(big[2], big[3])) == INFINITY) {   // infinite less infinite is no number
#pragma unroll
        for (int w = 0; w < 16; w++) lo[w] &= ((hi[w] & 0x7fffu) == 0x7f80u ? 0u : 0xffffu) | ((hi[w] & 0x7fff0000u) == 0x7f800000u ? 0u : 0xffff0000u);
      }
      if (u < 7) load(u + 1);   // under the stores of this one
#pragma unroll
      for (int k = 0; k < 2; k++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint32_t at = place((lane >> 2) + 8 * k, 4 * h + q);
          const int w = 8 * k + 4 * h;
          *reinterpret_cast<uint4*>(stage + at) = make_uint4(hi[w], hi[w + 1], hi[w + 2], hi[w + 3]);
          if constexpr (kForm == kPartialHalves) *reinterpret_cast<uint4*>(stage + 2048 + at) = make_uint4(lo[w], lo[w + 1], lo[w + 2], lo[w + 3]);
        }
      __syncwarp();
      uint16_t* dst = reinterpret_cast<uint16_t*>(part_o) + ((size_t)piece * H + head + (lane >> 3)) * kRowElems + dim + (lane & 7) * 8;
      uint4 a[4], b[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {   // eight lanes a row
        a[k] = *reinterpret_cast<const uint4*>(stage + place(4 * k + (lane >> 3), lane & 7));
        if constexpr (kForm == kPartialHalves) b[k] = *reinterpret_cast<const uint4*>(stage + 2048 + place(4 * k + (lane >> 3), lane & 7));
      }
      __syncwarp();   // before the next chunk
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (head + 4 * k + (lane >> 3) < H) {
          store_hint(dst + (size_t)(4 * k) * kRowElems, a[k], policy);
          if constexpr (kForm == kPartialHalves) store_hint(dst + (size_t)(4 * k) * kRowElems + kDC, b[k], policy);
        }
    }
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1)
    mla_decode_sm100_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_q,
                            const __grid_constant__ MlaSm100Params prm, const __grid_constant__ ListedPlan list) {
  extern __shared__ __align__(1024) uint8_t smem[];
  Bars* bars = reinterpret_cast<Bars*>(smem + kSmemBar);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cluster = blockIdx.x >> 1;
  const int worker = cluster / prm.sx;
  const int sq = blockIdx.y * prm.sx + cluster % prm.sx;   // query token of this worker
  chain_release();
  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled layouts need a 1024-byte aligned base
    chain_wait();
    if (threadIdx.x == 0) set_status(prm.status, RELUX_ERR_UNSUPPORTED);
    return;
  }
  // the set-up needs nothing of the kernel before this one, whose tail hides it
  if (threadIdx.x == 0) {
    for (int i = 0; i < kKGroups; i++) { mbar_init(&bars->k_full[i], 1); mbar_init(&bars->k_empty[i], 1); }
    for (int i = 0; i < 4; i++) { mbar_init(&bars->v_full[i], 1); mbar_init(&bars->v_empty[i], 1); }
    mbar_init(&bars->s_full[0], 1);
    mbar_init(&bars->s_full[1], 1);
    mbar_init(&bars->p_full, 8);    // one arrival per softmax warp of each CTA of the pair
    mbar_init(&bars->pv_done, 1);
    mbar_init(&bars->q_full, 1);
    bars->abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    tma_prefetch_desc(&tmap_q);
  }
  if (warp == 0) {
    tmem_alloc<2>(&bars->tmem_base, kTmemCols);
    tmem_relinquish<2>();
  }
  tc_fence_before();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  // The absorbed queries, the step's new rows and (unless they are arguments) the ranges come from the kernel before this one.  The producer
  // warp waits for them further down, behind its requests for a first tile of older rows: those were complete before the head of this
  // chain began, like the page table.
  const bool listed = list.listed != 0;
  if (warp != 4 || !listed) chain_wait();
  int it0 = listed ? list.worker_first[worker] : load_chained(prm.worker_first + worker);
  int it1 = listed ? list.worker_first[worker + 1] : load_chained(prm.worker_first + worker + 1);
  if (sq >= prm.S) it1 = it0;   // an empty range: nothing to do, and the CTA pair still meets at the end
  auto item_at = [&](int it) { return listed ? listed_item(list.items[it]) : load_item(prm.items + it); };
  if (threadIdx.x == 0 && it0 < it1) stamp_begin(prm.time);

  if (it0 >= it1) {
    if (warp == 4 && listed) chain_wait();
  } else if (warp == 4) {
    // =============================== producer: TMA loads into this CTA's slots ===============================
    // The whole warp stays converged and one elected lane issues: operands that every lane computes identically
    // live in uniform registers, which is what keeps the issue rate of TMA / tcgen05 instructions high.
    const bool el = elect_one();
    const uint32_t lead_q = mapa_u32(smem_u32(&bars->q_full), 0);
    auto win_load = [&](const StreamItem& it, int blk) -> int32_t {
      const int lp = min(32 * blk + lane, it.page_end - it.page_begin - 1);
      int32_t pg = __ldg(prm.table + (size_t)it.seq * prm.table_stride + it.page_begin + lp);
      if (pg < 0 || pg >= prm.num_pages) {   // reported, and replaced by page 0 so that no load leaves the pool
        set_status(prm.status, RELUX_ERR_BAD_PAGE);
        pg = 0;
      }
      return prm.layer_row0 + pg * (kNumKB * kPage);
    };
    auto win_get = [&](const PageWin& w, int lp) -> int32_t {
      if ((lp >> 5) == w.blk) return __shfl_sync(0xffffffffu, w.cur, lp & 31);
      return __shfl_sync(0xffffffffu, w.nxt, lp & 31);
    };
    // g = worker-wide index of the tile being loaded
    auto load_q = [&](const StreamItem& it) {
      const int qrow = (it.seq_index * prm.S + sq) * prm.H + 64 * (int)rank;   // Q~ rows of this CTA's 64 heads
      if (el) {
        if (rank == 0) mbar_expect_tx(&bars->q_full, 2 * kNumKB * kBlk);
        for (int grp = 0; grp < kKGroups; grp++) tma_load_3d_2sm(smem + kSmemQ + grp * kKPerGroup * kBlk, &tmap_q, 0, qrow, grp * kKPerGroup, lead_q);
      }
      __syncwarp();
    };
    auto load_k = [&](const PageWin& w, int tile, int g) {
      const int32_t y = win_get(w, 2 * tile + (int)rank);   // the tile's page held by this CTA
#pragma unroll
      for (int grp = 0; grp < kKGroups; grp++) {
        if (g > 0) wait_bar(&bars->k_empty[grp], (g - 1) & 1, bars, prm.status);
        const uint32_t lead = mapa_u32(smem_u32(&bars->k_full[grp]), 0);
        if (el) {
          if (rank == 0) mbar_expect_tx(&bars->k_full[grp], 2 * kKPerGroup * kBlk);
          tma_load_2d_2sm(smem + kSmemK + grp * kKPerGroup * kBlk, &tmap_k, 0, y + grp * kKPerGroup * kPage, lead);
        }
        __syncwarp();
      }
    };
    auto load_v = [&](const PageWin& w, int tile, int g) {
      const int32_t y0 = win_get(w, 2 * tile), y1 = win_get(w, 2 * tile + 1);
#pragma unroll
      for (int u = 0; u < 4; u++) {  // u = nb * 2 + kb
        const int nb = u >> 1, kb = u & 1;
        if (g > 0) wait_bar(&bars->v_empty[u], (g - 1) & 1, bars, prm.status);
        const int32_t y = kb ? y1 : y0;
        const uint32_t lead = mapa_u32(smem_u32(&bars->v_full[u]), 0);
        const int blk0 = 4 * nb + 2 * (int)rank;   // this CTA's 128 output dims of block nb = column blocks blk0, blk0 + 1
        if (el) {
          if (rank == 0) mbar_expect_tx(&bars->v_full[u], 4 * kBlk);
          tma_load_2d_2sm(smem + kSmemV + u * 2 * kBlk, &tmap_v, 0, y + blk0 * kPage, lead);
        }
        __syncwarp();
      }
    };
    StreamItem cur = item_at(it0);
    PageWin w;
    w.cur = win_load(cur, 0);
    w.nxt = win_load(cur, 1);
    w.blk = 0;
    // (the first values too, early or behind the queries: no difference)
    const bool early = listed && (cur.page_begin + 2) * kPage <= cur.tokens - list.new_rows;   // no row of the first tile is new
    if (early) load_k(w, 0, 0);
    if (listed) chain_wait();
    load_q(cur);
    if (!early) load_k(w, 0, 0);
    int g = 0;
    for (int it = it0; it < it1; ++it) {
      const bool has_next = it + 1 < it1;
      StreamItem nxt = cur;
      PageWin wn = w;
      if (has_next) {   // fetched now, used at the end of this item
        nxt = item_at(it + 1);
        wn.cur = win_load(nxt, 0);
        wn.nxt = win_load(nxt, 1);
        wn.blk = 0;
      }
      const int npages = cur.page_end - cur.page_begin;
      const int ntiles = (npages + 1) >> 1;
      for (int i = 0; i < ntiles; i++, g++) {
        if (!has_next && i == max(0, ntiles - kPrefetchTiles) && prm.w_uv_each > 0) {
          const uint32_t first = (blockIdx.y * gridDim.x + blockIdx.x) * prm.w_uv_each;
          if (el && first < prm.w_uv_bytes) prefetch_l2(prm.w_uv + first, min(prm.w_uv_each, prm.w_uv_bytes - first));
          __syncwarp();
        }
        if (i + 1 < ntiles) {
          load_k(w, i + 1, g + 1);
        } else if (has_next) {
          // the next item's first K tile goes group by group behind QK^T(g) like any other tile; Q~ may be replaced once
          // the last QK^T of this item (tile g) has completed, which the last group's slot being free says
          load_k(wn, 0, g + 1);
          wait_bar(&bars->k_empty[kKGroups - 1], g & 1, bars, prm.status);
          load_q(nxt);
        }
        load_v(w, i, g);
        if (((2 * i + 2) >> 5) > w.blk) {
          w.cur = w.nxt;
          w.blk++;
          w.nxt = win_load(cur, w.blk + 1);
        }
      }
      cur = nxt;
      w = wn;
    }
  } else if (warp == 5) {
    // =============================== MMA issuer (leader CTA only, converged warp + elected lane) ===============================
    if (rank == 0) {
      const bool el = elect_one();
      const uint32_t idesc_qk = make_idesc_bf16(128, 128, false, false);
      const uint32_t idesc_pv = make_idesc_bf16(128, 256, false, true);
      // descriptors of the region bases; an operand at +bytes is base + (bytes >> 4) in the low word
      const uint64_t dQ = make_desc_kmajor_sw128(smem_u32(smem + kSmemQ));
      const uint64_t dK = make_desc_kmajor_sw128(smem_u32(smem + kSmemK));
      const uint64_t dP = make_desc_kmajor_sw128(smem_u32(smem + kSmemP));
      const uint64_t dV = make_desc_mnmajor_sw128(smem_u32(smem + kSmemV), kBlk);
      auto issue_qk = [&](int g) {
        const uint32_t d = tmem + kTmemS + (g & 1) * 64;
#pragma unroll
        for (int grp = 0; grp < kKGroups; grp++) {
          wait_bar(&bars->k_full[grp], g & 1, bars, prm.status);
          if (el) {
#pragma unroll
            for (int j = 0; j < kKPerGroup * 4; j++) {
              const uint32_t off = (uint32_t)((grp * kKPerGroup + (j >> 2)) * kBlk + (j & 3) * 32) >> 4;
              umma_ss<2>(d, dQ + off, dK + off, idesc_qk, (grp | j) != 0);
            }
            umma_commit_mc<2>(&bars->k_empty[grp], 0x3);
          }
          __syncwarp();
        }
        if (el) umma_commit_mc<2>(&bars->s_full[g & 1], 0x3);
        __syncwarp();
      };
      auto issue_pv = [&](int g, bool first) {
        wait_bar(&bars->p_full, g & 1, bars, prm.status);
        tc_fence_after();   // P rows, a possible O rescale and the previous item's O read-out were done by the softmax warps
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int nb = u >> 1, kb = u & 1;
          wait_bar(&bars->v_full[u], g & 1, bars, prm.status);
          if (el) {
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
              umma_ss<2>(tmem + kTmemO + nb * 128, dP + ((uint32_t)(kb * kBlk + kk * 32) >> 4),
                         dV + ((uint32_t)(u * 2 * kBlk + kk * 2048) >> 4), idesc_pv, !first || (kb | kk) != 0);
            umma_commit_mc<2>(&bars->v_empty[u], 0x3);
          }
          __syncwarp();
        }
        if (el) umma_commit_mc<2>(&bars->pv_done, 0x3);
        __syncwarp();
      };
      auto tiles_of = [&](int it) -> int {
        const StreamItem a = item_at(it);
        return (a.page_end - a.page_begin + 1) >> 1;
      };
      int ntiles = tiles_of(it0);
      int g = 0, n = 0;
      wait_bar(&bars->q_full, 0, bars, prm.status);
      issue_qk(0);
      for (int it = it0; it < it1; ++it, ++n) {
        const bool has_next = it + 1 < it1;
        const int next_tiles = has_next ? tiles_of(it + 1) : 0;
        for (int i = 0; i < ntiles; i++, g++) {
          if (i + 1 < ntiles) {
            issue_qk(g + 1);
          }
          issue_pv(g, i == 0);
          if (i + 1 == ntiles && has_next) {
            // at an item end PV(g) goes first: the next Q~ lands a memory latency after QK^T(g), later than P(g) is ready,
            // and the softmax warps can start writing the item out as soon as PV(g) has completed
            wait_bar(&bars->q_full, (n + 1) & 1, bars, prm.status);
            issue_qk(g + 1);
          }
        }
        ntiles = next_tiles;
      }
    }
  } else {
    // =============================== softmax / correction / epilogue (warps 0-3) ===============================
    const int L = warp * 32 + lane;   // TMEM lane
    const int row = L & 63;           // head index inside this CTA
    const int hf = L >> 6;            // token half of the tile (= which CTA's page)
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    const uint32_t p_full_lead = mapa_u32(smem_u32(&bars->p_full), 0);
    StreamItem cur = item_at(it0);
    int g = 0;
    for (int it = it0; it < it1; ++it) {
      StreamItem nxt = cur;
      if (it + 1 < it1) nxt = item_at(it + 1);   // fetched now, used after this item
      const int limit_tok = prm.causal ? (cur.tokens - prm.S + sq + 1) : cur.tokens;   // tokens [0, limit_tok) are visible
      const int tok_end = min(limit_tok, cur.page_end * kPage);
      const int ntiles = (cur.page_end - cur.page_begin + 1) >> 1;
      float m_used = -INFINITY, l_run = 0.f;
      for (int i = 0; i < ntiles; i++, g++) {
        // no thread leaves this loop early: every thread must reach the same named barriers
        wait_bar(&bars->s_full[g & 1], (g >> 1) & 1, bars, prm.status);
        tc_fence_after();
        uint32_t sv[2][32];
        tmem_ld_32x32b_x32(tmem + lane_addr + kTmemS + (g & 1) * 64, sv[0]);
        tmem_ld_32x32b_x32(tmem + lane_addr + kTmemS + (g & 1) * 64 + 32, sv[1]);
        tmem_ld_wait();
        // valid tokens of this thread's 64: [0, nvalid); only the last tile(s) of an item are partial
        const int tok0 = (cur.page_begin + 2 * i + hf) * kPage;
        const int nvalid = (cur.page_begin + 2 * i + hf < cur.page_end) ? max(0, min(kPage, tok_end - tok0)) : 0;
        if (nvalid < kPage) {
#pragma unroll
          for (int h2 = 0; h2 < 2; h2++)
#pragma unroll
            for (int j = 0; j < 32; j++)
              if (h2 * 32 + j >= nvalid) sv[h2][j] = 0xFF800000u;  // -inf
        }
        // row max of the raw scores (the softmax scale is positive, so it commutes with max); four chains of three-input maxima
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int h2 = 0; h2 < 2; h2++)
#pragma unroll
          for (int j = 0; j < 32; j += 8)
#pragma unroll
            for (int k = 0; k < 4; k++) mx4[k] = max3(mx4[k], __uint_as_float(sv[h2][j + 2 * k]), __uint_as_float(sv[h2][j + 2 * k + 1]));
        float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * prm.scale_log2;
        // (a barrier that votes first, with the exchange only behind a yes, took as long per tile and 1 % longer per item: every
        // item's first tile is one)
        bars->rowmax[g & 1][hf][row] = mx;
        asm volatile("bar.sync 1, 128;" ::: "memory");
        mx = fmaxf(mx, bars->rowmax[g & 1][hf ^ 1][row]);
        // lazily updated running max: both threads of a row take the same decision
        float alpha = 1.f;
        bool rescale = false;
        if (mx > m_used + kRescaleThreshold) {   // also true on the first tile with a visible token (m_used = -inf)
          alpha = (m_used == -INFINITY) ? 0.f : exp2f(m_used - mx);
          rescale = (m_used != -INFINITY);
          m_used = mx;
        }
        // p = 2^(s * scale_log2 - m), two scores an instruction but for the exponentials
        const float neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
        const uint64_t scale2 = pack2(prm.scale_log2, prm.scale_log2), neg_m2 = pack2(neg_m, neg_m);
        uint64_t ps2[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
        uint32_t pk[32];
#pragma unroll
        for (int h2 = 0; h2 < 2; h2++)
#pragma unroll
          for (int j = 0; j < 32; j += 2) {
            float x0, x1;
            unpack2(fma2(pack2(__uint_as_float(sv[h2][j]), __uint_as_float(sv[h2][j + 1])), scale2, neg_m2), x0, x1);
            const float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
            ps2[(j >> 1) & 1] = add2(ps2[(j >> 1) & 1], pack2(p0, p1));
            __nv_bfloat162 b2 = __floats2bfloat162_rn(p0, p1);
            pk[h2 * 16 + j / 2] = *reinterpret_cast<uint32_t*>(&b2);
          }
        float ps0, ps1;
        unpack2(add2(ps2[0], ps2[1]), ps0, ps1);
        l_run = l_run * alpha + (ps0 + ps1);
        // P(g) may overwrite the buffer, and O may be rescaled, only after PV(g-1) has completed
        if (g > 0) wait_bar(&bars->pv_done, (g - 1) & 1, bars, prm.status);
        // TMEM loads and stores are warp-collective: the decision is taken for the whole warp, and the rows that keep their
        // maximum multiply by one
        if (__any_sync(0xffffffffu, rescale && i > 0)) {
          const float a_row = rescale ? alpha : 1.f;
          tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 256; c += 32) {
            uint32_t ov[32];
            tmem_ld_32x32b_x32(tmem + lane_addr + kTmemO + c, ov);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j++) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * a_row);
            tmem_st_32x32b_x32(tmem + lane_addr + kTmemO + c, ov);
          }
          tmem_st_wait();
          tc_fence_before();
        }
        // P row: 64 tokens = 128 bytes = one swizzled row of block hf
        uint8_t* prow = smem + kSmemP + hf * kBlk + row * 128;
#pragma unroll
        for (int c = 0; c < 8; c++)
          *reinterpret_cast<uint4*>(prow + ((c ^ (row & 7)) << 4)) = make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(p_full_lead);
      }
      // ---- item epilogue: O (unnormalised), running max and sum -> split-KV partial of this item ----
      wait_bar(&bars->pv_done, (g - 1) & 1, bars, prm.status);
      const bool ok = !__any_sync(0xffffffffu, bars->abort_flag != 0);   // the TMEM loads below are warp-collective
      tc_fence_after();
      bars->lsum[L] = l_run;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const float l_row = bars->lsum[row] + bars->lsum[64 + row];
      const bool real_head = 64 * (int)rank + row < prm.H;   // padding rows of the tile are not written
      // the pieces of a row lie one behind another where the up-projection reads them, item by item where merge_splits_kernel does
      const int piece = prm.form != kPartialFloat32 ? cur.first * prm.S + sq * cur.n + (it - cur.first) : it * prm.S + sq;
      if (hf == 0 && real_head) {
        const size_t prow = (size_t)piece * prm.H + 64 * rank + row;
        prm.part_ml[prow * 2] = ok ? m_used : -INFINITY;
        prm.part_ml[prow * 2 + 1] = !ok ? 0.f : prm.form != kPartialOne ? l_row : l_row > 0.f ? 1.f : 0.f;
      }
      if (64 * (int)rank + 32 * (warp & 1) >= prm.H) {   // none of the warp's rows is a head
      } else if (prm.form == kPartialHalves) write_partial<kPartialHalves>(smem, tmem + kTmemO, prm.part_o, prm.H, piece, 64 * (int)rank, m_used, l_row, ok);
      else if (prm.form == kPartialOne) write_partial<kPartialOne>(smem, tmem + kTmemO, prm.part_o, prm.H, piece, 64 * (int)rank, m_used, l_row, ok);
      else write_partial<kPartialFloat32>(smem, tmem + kTmemO, prm.part_o, prm.H, piece, 64 * (int)rank, m_used, l_row, ok);
      tc_fence_before();   // the O read-out is ordered before this thread's next p_full arrival, which releases the first PV of the next item
      cur = nxt;
    }
  }
  if (warp < 4) fence_chained_writes();   // the up-projection reads the partial rows by TMA
  tc_fence_before();
  cluster_sync_relaxed();   // nothing is handed over: the pair's barriers and tensor memory outlive what the other CTA does with them
  if (threadIdx.x == 0 && it0 < it1) stamp_end(prm.time);
  if (warp == 0) tmem_dealloc<2>(tmem, kTmemCols);
}

}  // namespace

bool mla_sm100_eligible(const Pool* p, const relux_attn_args& a) {
  const relux_pool_params& prm = p->prm;
  if (p->tune.get(RELUX_TUNE_MLA_GENERIC)) return false;
  // fewer than 128 heads run on the same M = 128 tile (padded); below 16 heads the CUDA-core kernel is the better fit
  return p->has_tmap && p->mla_blocked && prm.page_tokens == kPage && prm.mla_dc == kDC && prm.mla_dhr == kDR && a.num_heads <= kMaxHeads &&
         a.num_heads >= 16;
}


// Number of ranges the stream of pages is cut into: one per CTA pair that can be resident at the same time,
// divided among the query tokens that run side by side.
int mla_sm100_workers(Pool* p, int q_tokens) {
  static int max_clusters = 0;
  if (!max_clusters) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * 74, 1, 1);
    cfg.blockDim = dim3(192, 1, 1);
    cfg.dynamicSmemBytes = kSmemTotal;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(mla_decode_sm100_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemTotal) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, mla_decode_sm100_kernel, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = std::max(1, p->dev->sm_count / 2);
    }
    max_clusters = n;
  }
  int mc = max_clusters;
  if (const int ov = p->tune.get(RELUX_TUNE_MLA_WORKERS)) mc = std::max(1, ov);   // tuning knob
  if (q_tokens > kMaxInterleavedQ) {
    // A long multi-token call (a prompt) has one row of workers per query token: the rows already fill the device, so a
    // row needs only enough workers for about two waves in total, and each worker walks a long piece of the stream
    // (2048 tokens, one sequence: 3.2 ms with a full row of workers per token, 0.94 ms with one).
    return std::min(mc, std::max(1, (2 * mc + q_tokens - 1) / q_tokens));
  }
  return std::max(1, mc / q_tokens);
}

int32_t launch_mla_decode_sm100(Pool* p, const SeqBatch& sb, const relux_attn_args& a, const SplitPlan& plan, const uint16_t* q_abs,
                                const ListedPlan& list, int form, TimeStamp time) {
  const relux_pool_params& prm = p->prm;
  if (plan.num_items == 0) return RELUX_OK;   // every sequence is empty: the merge writes zeros
  CUtensorMap tq;   // the absorbed queries [rows][576] in boxes of three blocks of 64 columns x 64 rows
  const uint64_t q_dims[3] = {64, (uint64_t)sb.n_seqs * a.q_tokens * a.num_heads, kNumKB}, q_strides[2] = {kRow, 64};
  const uint32_t q_box[3] = {64, 64, kKPerGroup};
  if (!make_tmap_view(&tq, (void*)q_abs, 3, q_dims, q_strides, q_box)) {
    set_error("tensor map for the absorbed queries could not be encoded");
    return RELUX_ERR_CUDA;
  }
  const int sx = a.q_tokens <= kMaxInterleavedQ ? a.q_tokens : 1;
  MlaSm100Params k;
  k.items = plan.stream_items;
  k.worker_first = plan.worker_first;
  k.table = p->d_table;
  k.table_stride = prm.max_pages_per_seq;
  k.num_pages = prm.num_pages;
  k.S = a.q_tokens;
  k.sx = sx;
  k.causal = a.causal;
  k.layer_row0 = (int32_t)((int64_t)a.layer * prm.num_pages * kNumKB * kPage);
  k.scale_log2 = a.scale * 1.4426950408889634f;
  k.form = form;
  k.part_o = p->part_o.p;
  k.part_ml = (float*)p->part_ml.p;
  k.H = a.num_heads;
  k.status = p->d_status;
  k.time = time;
  // Cached rows of more than half of L2 have pushed the weights of the next launch out of it.
  int64_t cached = 0;
  for (int i = 0; i < sb.n_seqs; i++) cached += (int64_t)p->h_len[(size_t)a.layer * prm.max_seqs + sb.seq[i]] * kRow * 2;
  const uint32_t ctas = 2 * plan.num_workers * sx * (a.q_tokens / sx);
  k.w_uv = (const uint8_t*)a.w_uv;
  k.w_uv_bytes = (uint32_t)kDC * a.num_heads * a.head_dim * 2;
  k.w_uv_each = form != kPartialFloat32 && cached > kResidentBytes ? ((k.w_uv_bytes + ctas - 1) / ctas + 127) / 128 * 128 : 0;
  if (int32_t rc = allow_smem(p->dev, mla_decode_sm100_kernel, kSmemTotal)) return rc;
  dim3 grid(2 * plan.num_workers * sx, a.q_tokens / sx);
  RELUX_CUDA_TRY(launch_chained(p->tune.get(RELUX_TUNE_CHAINED_LAUNCHES) != 0, mla_decode_sm100_kernel, grid, dim3(192), (size_t)kSmemTotal,
                                p->dev->stream, p->tmap_mla_3, p->tmap_mla_2, tq, k, list));
  time_stamp_done(p->attn_times, time);
  return RELUX_OK;
}

}  // namespace relux
