// Whole attention layer steps on the device: the work of MLA.forwardCached (internal/transformer/mla.go:272-397) and
// MHA.forwardCached (mha.go:245-369) either side of the cached attention, so that a caller hands over the layer
// input x and gets the layer output back.  For MLA:
//   1. projections  q^C = x W_Q, q^R = x W_QR, c^KV = x W_DKV, k^R = x W_KR          mla.go:285-288
//   2. decoupled RoPE on q^R and k^R at position cacheLen + s                          mla.go:297-307, rope.go:130-180
//   3. append (c^KV, k^R) to the paged latent cache                                    mla.go:309-314
//   4. absorbed attention over the cache (the kernels of mla_decode.cu)                mla.go:317-377
//   5. output projection  out = o W_O                                                  mla.go:380-389
// and for GQA: q, k, v = x Wq, x Wk, x Wv (mha.go:251-258), RoPE on q and k (mha.go:272-282), append k / v
// (mha.go:284-289), attention (mha.go:292-348), Wo (mha.go:351-355).
// The projections are skinny GEMMs (M = sequences x new tokens, at most a few hundred rows) against bf16 weight
// matrices of up to 16384 x 16384: they are bound by streaming the weights from HBM once.  FAST mode runs them on
// tcgen05 (activations rounded to bf16, f32 accumulation in tensor memory, split along K so that every SM streams an
// equal share of the weights); REFERENCE mode runs them in the reference's own float32 operation order
// (matmulBatched3D, matmul.go: k ascending, multiply then add, never fused), bit for bit.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include "common.cuh"
#include "internal.h"
#include "umma.cuh"

namespace relux {

int32_t stage_in(Pool* p, GrowBuf& buf, const void* src, size_t bytes, int mem, const void** dptr);

namespace {

constexpr int kMaxWeights = 4;   // weight matrices that share one activation matrix in a launch
constexpr int kTileN = 128, kTileK = 64;
constexpr int kStageW = kTileK * kTileN * 2;   // 16 KB of weights: two [64 k][64 n] blocks, 128-byte swizzle, MN-major
constexpr int kMaxTok = 256;                   // activation rows of one block

// How a launch's tiles (128 weight columns x one block of rows) are dealt out.  `full` rounds of whole tiles, neighbouring tiles
// side by side: the workers then walk K in step and together read whole weight rows, which DRAM serves faster than 256-byte
// pieces of rows that lie far apart (0.54 GB: 86.8 us so, 90.1 us with every worker somewhere else in K; 0.82 GB: 128.5 against
// 130.8 us).  The tiles that are left are cut along K, `split` equal parts each (also in step), or (split = 0) their K steps,
// laid end to end, are cut into ranges that differ by at most one step.  A PIECE is the part of a tile that one worker does;
// piece j of a tile (in K order) is split j of the result.
// With more rows than a block holds, `beside` blocks have workers of their own that walk the same columns of weights in step, so
// that a column is read once for all of them; the blocks after those are further tiles of the same workers.
struct GemmRanges {
  int32_t workers, steps, full, split;   // of one of the blocks beside each other.  steps: K steps per tile (0: one piece per tile)
  int32_t range, more;                   // split = 0: steps per worker, one more for the first `more` of them
  int32_t rest;                          // tiles that are left after the full rounds
  int32_t beside, row_blocks, block_rows, col_tiles;
  bool in_turns() const { return row_blocks != beside; }
  __host__ __device__ int tile_of(int col, int row) const { return row / block_rows / beside * col_tiles + col; }
  __host__ __device__ int begin(int w) const {   // in steps of the tiles that are left
    if (!split) return w * range + (w < more ? w : more);
    return w < rest * split ? w / split * steps + w % split * steps / split : rest * steps;
  }
  __host__ __device__ int worker_of(int u) const {   // split = 0
    const int big = more * (range + 1);
    return u < big ? (int)((unsigned)u / (unsigned)(range + 1)) : more + (int)((unsigned)(u - big) / (unsigned)range);
  }
  __host__ __device__ int pieces(int tile) const {
    const int t = tile - full * workers;
    if (!steps || t < 0) return 1;
    return split ? split : worker_of((t + 1) * steps - 1) - worker_of(t * steps) + 1;
  }
};
// The pieces of one worker: GemmWalk walk(rg, w); while (walk.next()) ... walk.col, walk.block, steps [k0, k1), split.
// kBlocks: there may be more than one row block.
template <bool kBlocks>
struct GemmWalk {
  const GemmRanges& g;
  int w, n, u, u1, col, block, block0, k0, k1, split;
  __device__ GemmWalk(const GemmRanges& rg, int id)
      : g(rg), w(kBlocks ? id / rg.beside : id), n(0), u(rg.begin(w)), u1(rg.begin(w + 1)), col(0), block(0), block0(kBlocks ? id - w * rg.beside : 0),
        k0(0), k1(0), split(0) {}
  __device__ int total() const { return g.full * g.steps + g.begin(w + 1) - g.begin(w); }
  __device__ bool next() {
    int tile;
    split = 0;
    if (n < g.full) {
      tile = n++ * g.workers + w;
      k0 = 0;
      k1 = g.steps;
    } else {
      if (u >= u1) return false;
      const int t = u / g.steps;
      tile = g.full * g.workers + t;
      k0 = u - t * g.steps;
      u = min(u1, (t + 1) * g.steps);
      k1 = u - t * g.steps;
      split = g.split ? w - t * g.split : w - g.worker_of(t * g.steps);
    }
    col = tile;
    if constexpr (kBlocks) {
      block = block0;
      if (g.row_blocks != g.beside) {
        const int turn = tile / g.col_tiles;
        col = tile - turn * g.col_tiles;
        block += turn * g.beside;
      }
    }
    return true;
  }
};

struct GemmMaps {
  CUtensorMap a;                 // activations [M][K] bf16, box: 64 k x NT rows
  CUtensorMap w[kMaxWeights];    // weights [K][N_j] bf16
};
struct GemmParams {
  int32_t n_weights;
  int32_t tile_first[kMaxWeights + 1];   // first 128-column tile of every weight
  int32_t n_cols[kMaxWeights];           // N_j
  int32_t col_first[kMaxWeights];        // first output column of weight j in the concatenated result
  int32_t M, n_total;
  GemmRanges rg;
  float* part;                           // [piece][M][n_total] f32
  // With one block of rows every weight is read once; of more than 16 MB of them, they are loaded to be evicted first, and push out each
  // other and not the activations, partials and cached rows around them: MLA layer of 16 x 4096, 1.36 GB, 266.3 -> 258.4 us, GQA layers of
  // 84 MB, with the cached rows loaded so too, 66.6 -> 65.1 (24 x 2048), 76.4 -> 73.3 (128 x 300), 35.2 -> 34.3 (2 x 400).  Fewer may stay
  // in L2 from call to call.
  int32_t streams;
  // The result of more than 32 rows, in all its pieces no more than half of L2, is stored to stay there until it is summed (layer steps:
  // 100 x 1000 of d_model 4096 113 -> 107.6 us, 60 x 1000 of 16384 281 -> 278; up to 32 rows 1 % slower so).  More cannot stay, and would
  // push out what can (layer prompts of 2 x 2048 and 4 x 2048 tokens, 100 and 201 MB: 523 and 1013 us so, 521 and 1007 without).
  int32_t keeps;
  int32_t* status;
  TimeStamp time;                        // input projections only
};

// NT: activation rows of a block (the N of the MMA).  As many stages as shared memory holds.
template <int NT>
struct GemmShape {
  static constexpr int kStageX = NT * kTileK * 2;   // [NT rows][64 k] bf16, 128-byte swizzle, K-major
  static constexpr int kStage = kStageW + kStageX;
  static constexpr int kStages = (232448 - 1024) / kStage;
  static constexpr int kSmem = kStages * kStage + 1024;
  static constexpr int kAcc = NT < 32 ? 32 : NT;    // columns of one of the two accumulators
};

struct GemmBars {
  uint64_t full[12], empty[12], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  volatile int32_t abort_flag;
};
static_assert(GemmShape<16>::kStages <= 12 && sizeof(GemmBars) <= 1024, "barrier block too small");

__device__ __noinline__ void gemm_wait_slow(uint64_t* bar, uint32_t parity, GemmBars* b, int32_t* status) {
  for (uint32_t i = 0; i < kSpinLimit; i++) {
    if (mbar_try_wait(bar, parity)) return;
    if ((i & 255) == 255 && b->abort_flag) return;
    if (i > 512) __nanosleep(20);
  }
  b->abort_flag = 1;
  set_status(status, RELUX_ERR_TIMEOUT);
}
// Bounded wait: a wait that runs out records RELUX_ERR_TIMEOUT and raises the CTA's abort flag; nobody leaves a loop early.
__device__ __forceinline__ void gemm_wait(uint64_t* bar, uint32_t parity, GemmBars* b, int32_t* status) {
  if (!mbar_try_wait(bar, parity)) gemm_wait_slow(bar, parity, b, status);
}

// part[piece][m][n] = x [M][K] x [W_0 | W_1 | ...] over the piece's K steps.  Bound: HBM, every weight is read once.
// grid (workers), 192 threads: warps 0-3 epilogue, warp 4 TMA producer, warp 5 MMA issuer.
//   * The WEIGHTS are the M = 128 operand (MN-major: the row-major rows as they lie in HBM) and the activations, 16 to 256
//     rows, the N operand, so that a stage is 16 KB of weights and no more activations than there are: with the
//     activations as the M = 128 operand a stage of 16 rows was half padding, read from L2 for every step.
//   * One CTA per SM walks its pieces (GemmRanges) without draining its pipeline in between (two accumulators: a piece is
//     written out while the next one's MMAs run).
//   * The weights do not depend on the launches before this one, whose tail and launch gap they hide: the producer
//     fills its stages with them before chain_wait().  The first kernel of a layer step (cast_bf16_kernel) releases its
//     successors only when everything before the step is complete, so that weights written earlier in the stream are there.
// Measured with the chained launches around it (a layer step, before -> now): 16 rows of d_model 16384, 1.36 GB of weights,
// 308 -> 272 us; 24 rows of d_model 4096, 84 MB, 82.8 -> 67.0 us.
template <int NT>
__global__ void __launch_bounds__(192, 1) skinny_gemm_sm100_kernel(const __grid_constant__ GemmMaps maps, const __grid_constant__ GemmParams prm) {
  using SH = GemmShape<NT>;
  constexpr int kStages = SH::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  GemmBars* bars = reinterpret_cast<GemmBars*>(smem + kStages * SH::kStage);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr bool kBlocks = NT >= 128;   // smaller blocks hold all rows
  GemmWalk<kBlocks> walk(prm.rg, blockIdx.x);
  auto weight_of = [&](int tile) -> int {
    int j = 0;
    while (j + 1 < prm.n_weights && tile >= prm.tile_first[j + 1]) j++;
    return j;
  };
  chain_release();
  if ((smem_u32(smem) & 1023u) != 0) {
    chain_wait();
    if (threadIdx.x == 0) set_status(prm.status, RELUX_ERR_UNSUPPORTED);
    return;
  }
  if (threadIdx.x == 0) {
    stamp_begin(prm.time);   // the launch that cleared the slot is complete: see cast_bf16_kernel
    for (int s = 0; s < kStages; s++) { mbar_init(&bars->full[s], 1); mbar_init(&bars->empty[s], 1); }
    for (int b = 0; b < 2; b++) { mbar_init(&bars->acc_full[b], 1); mbar_init(&bars->acc_empty[b], 4); }
    bars->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc<1>(&bars->tmem_base, 2 * SH::kAcc);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;

  if (warp == 4) {
    const bool el = elect_one();
    const uint64_t policy = prm.streams ? make_evict_first_policy() : make_evict_normal_policy();   // (a branch around the loads cost 3 %)
    if (el) tma_prefetch_desc(&maps.a);
    const int n = walk.total(), ahead = min(n, kStages);
    auto wx = walk;   // the activations' place, up to kStages steps behind
    walk.next();
    wx.next();
    int k = walk.k0, kx = wx.k0, j = weight_of(walk.col);
    auto load_w = [&](int g) {   // the weights of step g of this worker; arms the stage for both operands
      const int s = g % kStages;
      if (el) {
        uint8_t* sw = smem + s * SH::kStage;
        const int n0 = (walk.col - prm.tile_first[j]) * kTileN;
        mbar_expect_tx(&bars->full[s], SH::kStage);   // out-of-range parts of a box are zero-filled and still counted
        tma_load_2d_hint(sw, &maps.w[j], n0, k * kTileK, &bars->full[s], policy);
        tma_load_2d_hint(sw + kStageW / 2, &maps.w[j], n0 + 64, k * kTileK, &bars->full[s], policy);
      }
      __syncwarp();
      if (++k == walk.k1 && walk.next()) {
        k = walk.k0;
        j = weight_of(walk.col);
      }
    };
    auto load_x = [&](int g) {
      const int s = g % kStages;
      if (el) tma_load_2d(smem + s * SH::kStage + kStageW, &maps.a, kx * kTileK, kBlocks ? wx.block * NT : 0, &bars->full[s]);
      __syncwarp();
      if (++kx == wx.k1 && wx.next()) kx = wx.k0;
    };
    for (int g = 0; g < ahead; g++) load_w(g);
    chain_wait();
    for (int g = 0; g < n; g++) {
      if (g >= ahead) {
        gemm_wait(&bars->empty[g % kStages], (g / kStages - 1) & 1, bars, prm.status);
        load_w(g);
      }
      load_x(g);
    }
  } else if (warp == 5) {
    chain_wait();
    const bool el = elect_one();
    const uint32_t idesc = make_idesc_bf16(kTileN, NT, true, false);
    int g = 0;
    for (int piece = 0; walk.next(); piece++) {
      const uint32_t d = tmem + (piece & 1) * SH::kAcc;
      if (piece >= 2) gemm_wait(&bars->acc_empty[piece & 1], ((piece >> 1) - 1) & 1, bars, prm.status);
      tc_fence_after();
      for (int k = walk.k0; k < walk.k1; k++, g++) {
        const int s = g % kStages;
        gemm_wait(&bars->full[s], (g / kStages) & 1, bars, prm.status);
        tc_fence_after();
        if (el) {
          const uint32_t sw = smem_u32(smem + s * SH::kStage);
          const uint64_t dW = make_desc_mnmajor_sw128(sw, kStageW / 2);
          const uint64_t dX = make_desc_kmajor_sw128(sw + kStageW);
#pragma unroll
          for (int kk = 0; kk < kTileK / 16; kk++)
            umma_ss<1>(d, dW + ((uint32_t)(kk * 2048) >> 4), dX + ((uint32_t)(kk * 32) >> 4), idesc, k != walk.k0 || kk != 0);
          umma_commit<1>(&bars->empty[s]);
        }
        __syncwarp();
      }
      if (el) umma_commit<1>(&bars->acc_full[piece & 1]);
      __syncwarp();
    }
  } else {
    // epilogue: thread = weight column, accumulator column = activation row; a warp writes 128 bytes of a row at once
    constexpr bool kKeep = NT >= 64;
    const uint64_t stay = !kKeep ? 0 : prm.keeps ? make_evict_last_policy() : make_evict_normal_policy();
    chain_wait();
    for (int piece = 0; walk.next(); piece++) {
      const int j = weight_of(walk.col), m0 = kBlocks ? walk.block * NT : 0;
      const int n = (walk.col - prm.tile_first[j]) * kTileN + warp * 32 + lane;
      const int m_end = min(NT, prm.M - m0);
      float* dst = prm.part + ((size_t)walk.split * prm.M + m0) * prm.n_total + prm.col_first[j] + n;
      gemm_wait(&bars->acc_full[piece & 1], (piece >> 1) & 1, bars, prm.status);
      tc_fence_after();
      const bool ok = !bars->abort_flag, mine = n < prm.n_cols[j];
#pragma unroll 1
      for (int c = 0; c < m_end; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem + ((uint32_t)(warp * 32) << 16) + (piece & 1) * SH::kAcc + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 32; q++)
          if (mine && c + q < m_end) {
            float* to = dst + (size_t)(c + q) * prm.n_total;
            const float x = ok ? __uint_as_float(v[q]) : 0.f;
            if constexpr (kKeep) store_hint(to, x, stay);
            else *to = x;
          }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[piece & 1]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) stamp_end(prm.time);
  if (warp == 0) tmem_dealloc<1>(tmem, 2 * SH::kAcc);
}

// The reference's matmulBatched3D in its own operation order: out[m][n] = sum over k ascending of x[m][k] * w[k][n],
// float32, multiply then add, never fused.  One thread per output element; threads of a warp read consecutive n.
__global__ void gemm_reference_kernel(const float* __restrict__ x, const uint16_t* __restrict__ w, float* __restrict__ out, int M, int K,
                                      int N, int out_stride, int col_first) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
  if (n >= N || m >= M) return;
  const float* xr = x + (size_t)m * K;
  float acc = 0.f;
  for (int k = 0; k < K; k++) acc = __fadd_rn(acc, __fmul_rn(xr[k], f32_from_bf16_bits(w[(size_t)k * N + n])));
  out[(size_t)m * out_stride + col_first + n] = acc;
}

// The first kernel of a layer step.  It waits before it releases the launch after it, which may therefore rely on
// everything that was queued before the step without a wait of its own.
__global__ void cast_bf16_kernel(const float* __restrict__ src, uint16_t* __restrict__ dst, size_t n8) {
  chain_wait();
  chain_release();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n8) return;
  const float4 a = load_chained(reinterpret_cast<const float4*>(src) + 2 * i), b = load_chained(reinterpret_cast<const float4*>(src) + 2 * i + 1);
  reinterpret_cast<uint4*>(dst)[i] = make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  fence_chained_writes();
}

// Sums the K splits of the projection result (fixed order, so the result does not depend on scheduling), applies
// RoPE (rope.go:168-176: pairs (2i, 2i+1) of a head, out0 = x0 c - x1 s, out1 = x1 c + x0 s, unfused) at position
// len[seq] + s to the segments that ask for it, and scatters every segment to its own buffer.
// One thread per pair of adjacent columns of the concatenated result.
struct ProjSeg {
  int32_t n;          // columns of this segment (= of its weight matrix)
  int32_t rope_dim;   // 0: no rotation; else the per-head width the rotation works on
  void* dst;          // [M][n], f32 or bf16
  int32_t bf16;
  int32_t by_tma;     // the next launch reads it by TMA
};
struct FinishParams {
  const float* part;
  GemmRanges rg;
  int32_t tile_first[kMaxWeights];   // first 128-column tile of every segment
  int32_t M, n_total, S, n_segs;
  ProjSeg seg[kMaxWeights];
  const int32_t* len;              // this layer's lengths BEFORE the append
  const int32_t* seq_ids;
  const float* rope_cos;           // [positions][rope_dim / 2]
  const float* rope_sin;
  int32_t rope_positions;
  int32_t same_pos;                // the reference's own rule (rope.go:151-158): on a non-empty cache every new row takes position len
  int32_t* status;
};
template <bool kTurns>   // the row blocks come in turns (GemmRanges): a tile is a column and a row
__global__ void proj_finish_kernel(const FinishParams p) {
  const int pair = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y;
  const int col = 2 * pair;
  chain_release();
  chain_wait();
  if (col >= p.n_total || m >= p.M) return;
  int c = col, j = 0;
  while (j + 1 < p.n_segs && c >= p.seg[j].n) {
    c -= p.seg[j].n;
    j++;
  }
  const int col_tile = p.tile_first[j] + c / kTileN;
  const int pieces = p.rg.pieces(kTurns ? p.rg.tile_of(col_tile, m) : col_tile);
  float v0 = 0.f, v1 = 0.f;
#pragma unroll 4
  for (int s = 0; s < pieces; s++) {
    const float2 t = load_chained(reinterpret_cast<const float2*>(p.part + ((size_t)s * p.M + m) * p.n_total + col));
    v0 += t.x;
    v1 += t.y;
  }
  const ProjSeg sg = p.seg[j];
  if (sg.rope_dim > 0) {
    const int i = m / p.S, s = m % p.S;
    const int seq = p.seq_ids ? p.seq_ids[i] : i;
    const int len0 = load_chained(p.len + seq);
    const int pos = (p.same_pos && len0 > 0) ? len0 : len0 + s;
    if (pos >= p.rope_positions) {
      set_status(p.status, RELUX_ERR_OVERFLOW);   // the reference panics: position >= maxSeqLen (rope.go:160-162)
    } else {
      const int half = sg.rope_dim / 2, idx = (c % sg.rope_dim) >> 1;
      const float cs = p.rope_cos[(size_t)pos * half + idx], sn = p.rope_sin[(size_t)pos * half + idx];
      const float r0 = __fsub_rn(__fmul_rn(v0, cs), __fmul_rn(v1, sn));
      const float r1 = __fadd_rn(__fmul_rn(v1, cs), __fmul_rn(v0, sn));
      v0 = r0;
      v1 = r1;
    }
  }
  if (sg.bf16) {
    reinterpret_cast<uint32_t*>(sg.dst)[((size_t)m * sg.n + c) >> 1] = pack_bf16x2(v0, v1);
    if (sg.by_tma) fence_chained_writes();
  } else {
    *reinterpret_cast<float2*>(reinterpret_cast<float*>(sg.dst) + (size_t)m * sg.n + c) = make_float2(v0, v1);
  }
}

// out [M][N] = sum over the pieces of one weight's tiles; a thread sums four adjacent columns.
template <bool kTurns>
__global__ void sum_splits_kernel(const float* __restrict__ part, GemmRanges rg, int N, size_t n4, float* __restrict__ out) {
  chain_release();
  chain_wait();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const int col_tile = (int)(4 * i % (unsigned)N) / kTileN;
  const int pieces = rg.pieces(kTurns ? rg.tile_of(col_tile, (int)(4 * i / (unsigned)N)) : col_tile);
  float4 acc = load_chained(reinterpret_cast<const float4*>(part) + i);
#pragma unroll 4
  for (int s = 1; s < pieces; s++) {
    const float4 t = load_chained(reinterpret_cast<const float4*>(part) + (size_t)s * n4 + i);
    acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
  }
  reinterpret_cast<float4*>(out)[i] = acc;
}

struct WeightRef {
  const void* w;
  int n;
};

template <int NT>
int32_t launch_skinny_gemm_rows(Pool* p, const GemmMaps& maps, const GemmParams& g, int workers) {
  if (int32_t rc = allow_smem(p->dev, skinny_gemm_sm100_kernel<NT>, GemmShape<NT>::kSmem)) return rc;
  RELUX_CUDA_TRY(launch_chained(p->tune.get(RELUX_TUNE_CHAINED_LAUNCHES) != 0, skinny_gemm_sm100_kernel<NT>, dim3(workers), dim3(192),
                                (size_t)GemmShape<NT>::kSmem, p->dev->stream, maps, g));
  count_launch(p->dev);
  return RELUX_OK;
}

// Deals the tiles to one worker per SM, `beside` blocks of `block_rows` rows beside each other.  max_pieces: pieces of a tile that
// the scratch holds.  *cost_us: what this takes beyond what every dealing takes, from measured parts (4 to 25600 rows against
// weights of 1024 x 1024 to 16384 x 16384): a step takes an SM 0.28 us whatever the rows of its block, and a tenth more where the
// workers don't walk in step; the weights come at 7 TB/s, again for every turn of blocks when they exceed L2; the last piece of
// a worker is written at 16 ns per row with nothing to hide it; pieces are written and read at 3 TB/s.
GemmRanges deal_tiles(int sms, int col_tiles, int M, int block_rows, int beside, int K, int cols, int max_pieces, int split_knob, double* cost_us) {
  GemmRanges r{};
  r.steps = (K + kTileK - 1) / kTileK;
  r.col_tiles = col_tiles;
  r.row_blocks = (M + block_rows - 1) / block_rows;
  r.block_rows = block_rows;
  r.beside = beside;
  const int turns = (r.row_blocks + beside - 1) / beside, tiles = col_tiles * turns, units = tiles * r.steps;
  r.workers = std::max(1, std::min(std::max(1, sms / beside), units / 4));   // pieces of fewer than four steps do not pay for their share of the result
  if (split_knob) r.workers = std::max(1, (int)std::min<int64_t>(units, (int64_t)tiles * split_knob));
  r.full = tiles / r.workers;
  r.rest = tiles % r.workers;
  r.range = r.rest * r.steps / r.workers;
  r.more = r.rest * r.steps % r.workers;
  const double step = 0.28, write = 0.016 * std::min(block_rows, M), per_piece = (double)M * cols * 4 / tiles / 3e6, bytes = (double)K * cols * 2;
  const double weights = bytes * (bytes > 60e6 ? turns : 1) / 7e6;
  auto cost = [&](double steps, double pieces) { return std::max((r.full * r.steps + steps) * step, weights) + write + pieces * per_piece; };
  if (!r.rest) {
    *cost_us = cost(0, tiles);
    return r;
  }
  const int fits = std::max(1, std::min(r.workers / r.rest, max_pieces)), most_split = std::max(1, r.steps / 4);
  const bool even = r.range > 0 && (r.steps - 2) / r.range + 2 <= max_pieces;   // may the ranges be even?
  const double even_cost = cost(1.1 * r.rest * r.steps / r.workers, tiles + r.workers) + std::max(0.0, write - r.range * step / 2);
  auto split_cost = [&](int s) { return cost((r.steps + s - 1) / s, tiles + (double)r.rest * (s - 1)); };
  if (block_rows <= 64) {
    // few rows: results are small, and what counts is that no SM idles
    if (fits >= most_split) r.split = most_split;
    else if (!even || 6 * fits * r.rest >= 5 * r.workers) r.split = fits;
  } else {
    r.split = 1;
    for (int s = 2; s <= std::min(fits, most_split); s++)
      if (split_cost(s) < split_cost(r.split)) r.split = s;
    if (even && even_cost < split_cost(r.split)) r.split = 0;
  }
  *cost_us = r.split ? split_cost(r.split) : even_cost;
  return r;
}

// part[piece][M][n_total] = A[M][K] x [W_0 | W_1 | ...]; returns the ranges, which say how many pieces every tile has.
int32_t launch_skinny_gemm(Pool* p, const uint16_t* a_bf16, int M, int K, const WeightRef* ws, int nw, float* part, size_t part_cap_bytes,
                           GemmRanges* ranges, TimeStamp time = TimeStamp{nullptr, nullptr}) {
  GemmMaps maps;
  GemmParams g;
  memset(&g, 0, sizeof(g));
  int tiles = 0, cols = 0;
  for (int j = 0; j < nw; j++) {
    if (!make_tmap_2d(&maps.w[j], (void*)ws[j].w, (uint64_t)K, (uint64_t)ws[j].n, 64, kTileK)) {
      set_error("tensor map for a weight matrix could not be encoded");
      return RELUX_ERR_CUDA;
    }
    g.tile_first[j] = tiles;
    g.n_cols[j] = ws[j].n;
    g.col_first[j] = cols;
    tiles += (ws[j].n + kTileN - 1) / kTileN;
    cols += ws[j].n;
  }
  for (int j = nw; j < kMaxWeights; j++) maps.w[j] = maps.w[0];
  g.tile_first[nw] = tiles;
  g.n_weights = nw;
  g.M = M;
  g.n_total = cols;
  const int steps = (K + kTileK - 1) / kTileK;
  if ((int64_t)tiles * ((M + 127) / 128) * steps >= (int64_t)1 << 31) { set_error("a projection of more than 2^31 steps"); return RELUX_ERR_UNSUPPORTED; }
  // Rows of a block: the smallest tile that holds them all (padding costs L2 reads and shared memory), up to 256; more than 128
  // rows also as blocks of 128 where that keeps more SMs busy or leaves less padding (256 rows of 4096 x 1024: 14.8 us, one block
  // of 256 20.2).  Up to 16 blocks beside each other, whichever number leaves the fewest SMs idle: with all of them beside
  // each other 19200 rows had 75 workers (4096 x 4096: 1.28 ms, now 0.71).
  int nt = 16;
  while (nt < M && nt < kMaxTok) nt *= 2;
  const int max_pieces = (int)std::min<size_t>(std::max<size_t>(1, part_cap_bytes / ((size_t)M * cols * 4)), 1 << 20);
  double best = 0;
  for (int rows = nt; rows >= std::min(nt, 128); rows /= 2)
    for (int beside = std::min(16, (M + rows - 1) / rows); beside >= 1; beside--) {
      double cost = 0;
      const GemmRanges r = deal_tiles(p->dev->sm_count, tiles, M, rows, beside, K, cols, max_pieces, p->tune.get(RELUX_TUNE_GEMM_SPLIT), &cost);
      if (!g.rg.workers || cost < best) {
        g.rg = r;
        best = cost;
      }
    }
  nt = g.rg.block_rows;
  if (!make_tmap_2d(&maps.a, (void*)a_bf16, (uint64_t)M, (uint64_t)K, kTileK, nt)) {
    set_error("tensor map for the activations could not be encoded");
    return RELUX_ERR_CUDA;
  }
  const int workers = g.rg.workers * g.rg.beside;
  g.part = part;
  g.streams = g.rg.row_blocks == 1 && (int64_t)K * cols * 2 > ((int64_t)16 << 20);
  const int tiles_of_block = g.rg.full * g.rg.workers + g.rg.rest;
  const int pieces_of_block = g.rg.full * g.rg.workers + (g.rg.split ? g.rg.rest * g.rg.split : g.rg.rest ? g.rg.rest + g.rg.workers : 0);
  g.keeps = (int64_t)M * cols * 4 * pieces_of_block / tiles_of_block <= kResidentBytes;
  g.status = p->d_status;
  g.time = time;
  *ranges = g.rg;
  switch (nt) {
    case 16: return launch_skinny_gemm_rows<16>(p, maps, g, workers);
    case 32: return launch_skinny_gemm_rows<32>(p, maps, g, workers);
    case 64: return launch_skinny_gemm_rows<64>(p, maps, g, workers);
    case 128: return launch_skinny_gemm_rows<128>(p, maps, g, workers);
    default: return launch_skinny_gemm_rows<kMaxTok>(p, maps, g, workers);
  }
}

bool gemm_sm100_eligible(int K, const WeightRef* ws, int nw) {
  if (K % 8 != 0 || nw > kMaxWeights) return false;
  for (int j = 0; j < nw; j++)
    if (ws[j].n % 8 != 0 || ((uintptr_t)ws[j].w & 15) != 0) return false;
  return true;
}

int32_t launch_gemm_reference(Pool* p, const float* x, int M, int K, const WeightRef* ws, int nw, float* out, int out_stride) {
  int col = 0;
  for (int j = 0; j < nw; j++) {
    dim3 grid((ws[j].n + 127) / 128, M);
    gemm_reference_kernel<<<grid, 128, 0, p->dev->stream>>>(x, (const uint16_t*)ws[j].w, out, M, K, ws[j].n, out_stride, col);
    RELUX_CUDA_TRY(cudaGetLastError());
    count_launch(p->dev);
    col += ws[j].n;
  }
  return RELUX_OK;
}

// cos / sin tables of the decoupled RoPE exactly as NewRotaryEmbedding builds them (rope.go:59-68):
// theta = float32(1) / float32(pow(base, 2i / headDim)), angle = float32(pos * theta), cos / sin in float64, rounded.
int32_t ensure_rope_table(Pool* p, int dHR, float base, int positions) {
  if (p->rope_dim == dHR && p->rope_base == base && p->rope_positions >= positions) return RELUX_OK;
  const int half = dHR / 2;
  std::vector<float> tab((size_t)2 * positions * half);
  for (int pos = 0; pos < positions; pos++)
    for (int i = 0; i < half; i++) {
      const float theta = 1.0f / (float)std::pow((double)base, (double)(2 * i) / (double)dHR);
      const float angle = (float)((double)pos * (double)theta);
      tab[(size_t)pos * half + i] = (float)std::cos((double)angle);
      tab[(size_t)positions * half + (size_t)pos * half + i] = (float)std::sin((double)angle);
    }
  int32_t rc = grow(p->dev, p->rope_tab, tab.size() * 4);
  if (rc) return rc;
  RELUX_CUDA_TRY(cudaMemcpyAsync(p->rope_tab.p, tab.data(), tab.size() * 4, cudaMemcpyHostToDevice, p->dev->stream));
  RELUX_CUDA_TRY(cudaStreamSynchronize(p->dev->stream));   // `tab` goes out of scope
  p->rope_dim = dHR;
  p->rope_base = base;
  p->rope_positions = positions;
  return RELUX_OK;
}

int32_t launch_cast(Pool* p, const float* src, uint16_t* dst, size_t n) {
  RELUX_CUDA_TRY(launch_chained(p->tune.get(RELUX_TUNE_CHAINED_LAUNCHES) != 0, cast_bf16_kernel, dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0,
                                p->dev->stream, src, dst, n / 8));
  count_launch(p->dev);
  return RELUX_OK;
}

// x [M][K] f32 -> every segment's buffer: cast + split-K tensor-core GEMM (or the reference-order GEMM), then the
// finish kernel.  The GEMM's device time goes to the pool's projection ring.
int32_t project_and_finish(Pool* p, const SeqBatch& sb, int layer, const float* dx, int M, int K, int S, const WeightRef* ws,
                           const ProjSeg* segs, int nw, bool mma, uint16_t* a_bf16, float* part, size_t part_cap, bool same_pos = false) {
  cudaStream_t st = p->dev->stream;
  const bool chained = p->tune.get(RELUX_TUNE_CHAINED_LAUNCHES) != 0;
  int n_total = 0;
  for (int j = 0; j < nw; j++) n_total += ws[j].n;
  GemmRanges ranges{};
  if (mma) {
    int32_t rc = launch_cast(p, dx, a_bf16, (size_t)M * K);
    const TimeStamp time = time_stamp_next(p, p->proj_times);
    if (!rc) rc = launch_skinny_gemm(p, a_bf16, M, K, ws, nw, part, part_cap, &ranges, time);
    if (rc) return rc;
    time_stamp_done(p->proj_times, time);
  } else {
    int32_t rc = time_events_begin(p, p->proj_times);
    if (rc) return rc;
    rc = launch_gemm_reference(p, dx, M, K, ws, nw, part, n_total);
    if (rc) return rc;
    if ((rc = time_events_end(p, p->proj_times))) return rc;
  }
  FinishParams f;
  memset(&f, 0, sizeof(f));
  f.part = part;
  f.rg = ranges;
  for (int j = 1; j < nw; j++) f.tile_first[j] = f.tile_first[j - 1] + (ws[j - 1].n + kTileN - 1) / kTileN;
  f.M = M;
  f.n_total = n_total;
  f.S = S;
  f.n_segs = nw;
  int rope_dim = 0;
  for (int j = 0; j < nw; j++) {
    f.seg[j] = segs[j];
    if (segs[j].rope_dim) rope_dim = segs[j].rope_dim;
  }
  f.len = p->d_len + (size_t)layer * p->prm.max_seqs;
  f.seq_ids = sb.d_seq_ids;
  f.rope_cos = (const float*)p->rope_tab.p;
  f.rope_sin = f.rope_cos ? f.rope_cos + (size_t)p->rope_positions * (rope_dim / 2) : nullptr;
  f.rope_positions = p->rope_positions;
  f.same_pos = same_pos ? 1 : 0;
  f.status = p->d_status;
  dim3 grid((n_total / 2 + 255) / 256, M);
  RELUX_CUDA_TRY(launch_chained(chained, ranges.in_turns() ? proj_finish_kernel<true> : proj_finish_kernel<false>, grid, dim3(256), 0, st, f));
  count_launch(p->dev);
  return RELUX_OK;
}

// out [M][N] f32 = attn [M][K] x W_O [K][N]; `out` is the caller's buffer (host or device).  d_attn: float32, or nullptr when
// the rows are in a_bf16 already (mma).
int32_t output_projection(Pool* p, const float* d_attn, int M, int K, const void* w_o, int N, bool mma, uint16_t* a_bf16, float* part,
                          size_t part_cap, void* out, int out_mem) {
  cudaStream_t st = p->dev->stream;
  const bool direct = out_mem == RELUX_MEM_DEVICE;
  float* d_out = direct ? (float*)out : nullptr;
  if (!direct) {
    int32_t rc = grow(p->dev, p->out_buf, (size_t)M * N * 4);
    if (rc) return rc;
    d_out = (float*)p->out_buf.p;
  }
  const WeightRef outp[1] = {{w_o, N}};
  if (mma) {
    GemmRanges ranges{};
    int32_t rc = d_attn ? launch_cast(p, d_attn, a_bf16, (size_t)M * K) : RELUX_OK;
    if (!rc) rc = launch_skinny_gemm(p, a_bf16, M, K, outp, 1, part, part_cap, &ranges);
    if (rc) return rc;
    const size_t n4 = (size_t)M * N / 4;
    RELUX_CUDA_TRY(launch_chained(p->tune.get(RELUX_TUNE_CHAINED_LAUNCHES) != 0, ranges.in_turns() ? sum_splits_kernel<true> : sum_splits_kernel<false>,
                                  dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, st, (const float*)part, ranges, N, n4, d_out));
    count_launch(p->dev);
  } else {
    int32_t rc = launch_gemm_reference(p, d_attn, M, K, outp, 1, d_out, N);
    if (rc) return rc;
  }
  if (!direct) {
    RELUX_CUDA_TRY(cudaMemcpyAsync(out, d_out, (size_t)M * N * 4, cudaMemcpyDeviceToHost, st));
    RELUX_CUDA_TRY(cudaStreamSynchronize(st));
  }
  return RELUX_OK;
}

// Validation shared by the two layer entry points; fills the batch with S rows per sequence.
int32_t layer_batch(Pool* p, int layer, int n_seqs, const int32_t* seq_ids, int S, const char* what, SeqBatch* sb) {
  const relux_pool_params& prm = p->prm;
  if (layer < 0 || layer >= prm.num_layers) {
    set_error("layerIdx=%d out of range [0, %d)", layer, prm.num_layers);
    return RELUX_ERR_INVALID_ARG;
  }
  if (n_seqs <= 0 || n_seqs > prm.max_seqs) {
    set_error("n_seqs=%d outside [1, max_seqs=%d]", n_seqs, prm.max_seqs);
    return RELUX_ERR_INVALID_ARG;
  }
  int32_t rc = stage_batch(p, n_seqs, seq_ids, nullptr, S, sb);
  if (rc) return rc;
  for (int i = 0; i < sb->n_seqs; i++) {   // the reference panics on overflow (kvcache.go:282-285, mla_cache.go:160-164)
    const int s = sb->seq[i];
    const int len = p->h_len[(size_t)layer * prm.max_seqs + s], cap = p->seq_pages[s] * prm.page_tokens;
    if (len + S > cap) {
      set_error("%s: layer %d overflow: total=%d + newLen=%d > capacity=%d (sequence %d)", what, layer, len, S, cap, s);
      return RELUX_ERR_OVERFLOW;
    }
  }
  return RELUX_OK;
}

struct LayerScratch {
  uint16_t* a_bf16;
  float* part;
  size_t part_cap;
  char* rest;
};
// [activations as bf16 (M x max_k) | split partials | caller's buffers (rest_bytes)]
int32_t layer_scratch(Pool* p, int M, int max_k, int max_n, size_t rest_bytes, LayerScratch* out) {
  const size_t part_cap = std::max<size_t>((size_t)64 << 20, (size_t)M * max_n * 4 * 4);
  const size_t off_part = ((size_t)M * max_k * 2 + 255) & ~(size_t)255;
  const size_t off_rest = off_part + part_cap;
  int32_t rc = grow(p->dev, p->layer_buf, off_rest + rest_bytes);
  if (rc) return rc;
  char* base = (char*)p->layer_buf.p;
  out->a_bf16 = (uint16_t*)base;
  out->part = (float*)(base + off_part);
  out->part_cap = part_cap;
  out->rest = base + off_rest;
  return RELUX_OK;
}
inline size_t pad256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace

int32_t do_mla_layer(Pool* p, const relux_mla_layer_args* a) {
  if (!a || !a->w) { set_error("nil argument struct"); return RELUX_ERR_INVALID_ARG; }
  const relux_pool_params& prm = p->prm;
  if (prm.kind != RELUX_POOL_MLA) { set_error("pool kind does not match this call (MLA pool needed)"); return RELUX_ERR_INVALID_ARG; }
  const relux_mla_layer_weights& w = *a->w;
  if (!a->x || !a->out || !w.w_q || !w.w_qr || !w.w_dkv || !w.w_kr || !w.w_uk || !w.w_uv || !w.w_o) {
    set_error("nil input, output or weight pointer");
    return RELUX_ERR_INVALID_ARG;
  }
  const int H = a->num_heads, D = a->d_model, S = a->q_tokens, dC = prm.mla_dc, dHR = prm.mla_dhr;
  if (H <= 0 || D <= 0 || S <= 0 || D % H != 0) {   // NewMLA, mla.go:69-74
    set_error("NewMLA: dModel=%d not divisible by numHeads=%d (or non-positive sizes)", D, H);
    return RELUX_ERR_INVALID_ARG;
  }
  if (dHR % 2 != 0) { set_error("NewMLA: dHR=%d must be even for paired RoPE rotation", dHR); return RELUX_ERR_INVALID_ARG; }
  if (a->mode != RELUX_ATTN_FAST && a->mode != RELUX_ATTN_REFERENCE && a->mode != RELUX_ATTN_REFERENCE_FAITHFUL) { set_error("bad mode"); return RELUX_ERR_INVALID_ARG; }
  const bool faithful = a->mode == RELUX_ATTN_REFERENCE_FAITHFUL;
  if (faithful && !p->compat) { set_error("RELUX_ATTN_REFERENCE_FAITHFUL needs a pool created with RELUX_POOL_FLAG_REFERENCE_COMPAT"); return RELUX_ERR_INVALID_ARG; }
  if (a->x_dtype != RELUX_DTYPE_F32) { set_error("x must be float32"); return RELUX_ERR_UNSUPPORTED; }
  const int Dh = D / H;
  const float rope_base = a->rope_base == 0.f ? 10000.f : a->rope_base;   // NewMLA, mla.go:78-80
  SeqBatch sb;
  int32_t rc = layer_batch(p, a->layer, a->n_seqs, a->seq_ids, S, "MLACache.Append", &sb);
  if (rc) return rc;
  const int M = sb.n_seqs * S;
  rc = ensure_rope_table(p, dHR, rope_base, prm.max_pages_per_seq * prm.page_tokens);
  if (rc) return rc;
  const void* dx = nullptr;
  rc = stage_in(p, p->in_a, a->x, (size_t)M * D * 4, a->x_mem, &dx);
  if (rc) return rc;

  const WeightRef proj[4] = {{w.w_q, H * Dh}, {w.w_qr, H * dHR}, {w.w_dkv, dC}, {w.w_kr, dHR}};
  const WeightRef outp[1] = {{w.w_o, D}};
  const int n_total = H * Dh + H * dHR + dC + dHR;
  const bool fast = a->mode == RELUX_ATTN_FAST;
  const bool mma = fast && !p->tune.get(RELUX_TUNE_GEMM_GENERIC) && gemm_sm100_eligible(D, proj, 4) && gemm_sm100_eligible(H * Dh, outp, 1);
  const size_t q_es = fast ? 2 : 4;
  const size_t b_qc = pad256((size_t)M * H * Dh * q_es), b_qr = pad256((size_t)M * H * dHR * q_es), b_c = pad256((size_t)M * dC * 4),
               b_kr = pad256((size_t)M * dHR * 4);
  LayerScratch sc;
  rc = layer_scratch(p, M, std::max(D, H * Dh), std::max(n_total, D), b_qc + b_qr + b_c + b_kr + (size_t)M * H * Dh * 4, &sc);
  if (rc) return rc;
  void* d_qc = sc.rest;
  void* d_qr = sc.rest + b_qc;
  float* d_c = (float*)(sc.rest + b_qc + b_qr);
  float* d_kr = (float*)(sc.rest + b_qc + b_qr + b_c);
  float* d_attn = (float*)(sc.rest + b_qc + b_qr + b_c + b_kr);
  // 1 + 2. projections, RoPE on q^R and k^R
  const ProjSeg segs[4] = {{H * Dh, 0, d_qc, fast ? 1 : 0, 1}, {H * dHR, dHR, d_qr, fast ? 1 : 0, S > 1}, {dC, 0, d_c, 0, 0}, {dHR, dHR, d_kr, 0, 0}};
  rc = project_and_finish(p, sb, a->layer, (const float*)dx, M, D, S, proj, segs, 4, mma, sc.a_bf16, sc.part, sc.part_cap, faithful);
  if (rc) return rc;
  // 3. append (advances the cursors).  A one-token step on the tensor-core path leaves the append to the attention's
  //    preparation launch (absorb + append + stream partition in one kernel, as relux_mla_step does).
  relux_attn_args probe;
  memset(&probe, 0, sizeof(probe));
  probe.mode = a->mode;
  probe.num_heads = H;
  probe.head_dim = Dh;
  probe.q_tokens = S;
  const bool fused_append = fast && S == 1 && mla_step_fusable(p, probe);
  if (!fused_append) {
    rc = launch_mla_append(p, sb, a->layer, d_c, d_kr, RELUX_DTYPE_F32, 1);
    if (rc) return rc;
  }
  for (int i = 0; i < sb.n_seqs; i++) {
    int32_t& len = p->h_len[(size_t)a->layer * prm.max_seqs + sb.seq[i]];
    note_append(p, a->layer, sb.seq[i], len, S);
    len += S;
  }
  // 4. attention over the cache, the S new rows included
  relux_attn_args aa;
  memset(&aa, 0, sizeof(aa));
  aa.layer = a->layer;
  aa.n_seqs = sb.n_seqs;
  aa.seq_ids = a->seq_ids;
  aa.q_tokens = S;
  aa.extra_tokens = 0;
  aa.causal = a->causal;
  aa.num_heads = H;
  aa.head_dim = Dh;
  aa.scale = (float)(1.0 / std::sqrt((double)(Dh + dHR)));   // mla.go:344-345
  aa.q_dtype = fast ? RELUX_DTYPE_BF16 : RELUX_DTYPE_F32;
  aa.q_layout = RELUX_LAYOUT_TOKEN_MAJOR;
  aa.w_uk = w.w_uk;
  aa.w_uv = w.w_uv;
  aa.mode = a->mode;
  const StepAppend step{d_c, d_kr, RELUX_DTYPE_F32, nullptr, 1, 1, mma};   // one row per sequence
  const bool o_bf16 = mma && mla_writes_bf16(p, sb, aa);   // the output projection's operand, rounded by the kernel that makes it
  rc = fast ? launch_mla_decode_fast(p, sb, aa, d_qc, d_qr, o_bf16 ? (void*)sc.a_bf16 : d_attn, o_bf16, fused_append ? &step : nullptr)
            : launch_attn_reference_mla(p, sb, aa, (const float*)d_qc, (const float*)d_qr, d_attn);
  if (rc) {
    if (fused_append) take_rows_back(p, sb, a->layer);   // nobody appended them
    return rc;
  }
  // 5. output projection
  return output_projection(p, o_bf16 ? nullptr : d_attn, M, H * Dh, w.w_o, D, mma, sc.a_bf16, sc.part, sc.part_cap, a->out, a->out_mem);
}

// MHA.forwardCached (mha.go:245-369) for a batch of independent sequences: projections with Wq / Wk / Wv, RoPE on q
// and k at position cacheLen + s (when the layer has a rotary embedding), append of k / v, GQA attention, Wo.
int32_t do_gqa_layer(Pool* p, const relux_gqa_layer_args* a) {
  if (!a || !a->w) { set_error("nil argument struct"); return RELUX_ERR_INVALID_ARG; }
  const relux_pool_params& prm = p->prm;
  if (prm.kind != RELUX_POOL_GQA) { set_error("pool kind does not match this call (GQA pool needed)"); return RELUX_ERR_INVALID_ARG; }
  const relux_gqa_layer_weights& w = *a->w;
  if (!a->x || !a->out || !w.w_q || !w.w_k || !w.w_v || !w.w_o) {
    set_error("nil input, output or weight pointer");
    return RELUX_ERR_INVALID_ARG;
  }
  const int H = a->num_heads, D = a->d_model, S = a->q_tokens, Hkv = prm.gqa_num_kv_heads, hd = prm.gqa_head_dim;
  if (H <= 0 || D <= 0 || S <= 0 || D % H != 0 || D / H != hd || H % Hkv != 0) {   // NewMHAGQA, mha.go
    set_error("dModel=%d / numHeads=%d must equal the pool's head_dim=%d, numHeads a multiple of numKVHeads=%d", D, H, hd, Hkv);
    return RELUX_ERR_INVALID_ARG;
  }
  if (a->rope && hd % 2 != 0) { set_error("NewRotaryEmbedding: headDim=%d, must be even and > 0", hd); return RELUX_ERR_INVALID_ARG; }
  if (a->mode != RELUX_ATTN_FAST && a->mode != RELUX_ATTN_REFERENCE && a->mode != RELUX_ATTN_REFERENCE_FAITHFUL) { set_error("bad mode"); return RELUX_ERR_INVALID_ARG; }
  const bool faithful = a->mode == RELUX_ATTN_REFERENCE_FAITHFUL;
  if (faithful && (!p->compat || !a->advance)) { set_error("RELUX_ATTN_REFERENCE_FAITHFUL needs a pool created with RELUX_POOL_FLAG_REFERENCE_COMPAT and advance != 0"); return RELUX_ERR_INVALID_ARG; }
  if (a->x_dtype != RELUX_DTYPE_F32) { set_error("x must be float32"); return RELUX_ERR_UNSUPPORTED; }
  if (a->mode == RELUX_ATTN_FAST && (!p->has_tmap || prm.page_tokens != 64 || hd != 128 || H / Hkv > 32)) {
    // checked before anything is written to the cache
    set_error("GQA FAST kernels need page_tokens=64, head_dim=128 and num_heads/num_kv_heads <= 32 "
              "(got page_tokens=%d head_dim=%d group=%d); use RELUX_ATTN_REFERENCE for other shapes", prm.page_tokens, hd, H / Hkv);
    return RELUX_ERR_UNSUPPORTED;
  }
  const float rope_base = a->rope_base == 0.f ? 10000.f : a->rope_base;
  SeqBatch sb;
  int32_t rc = layer_batch(p, a->layer, a->n_seqs, a->seq_ids, S, "Append", &sb);
  if (rc) return rc;
  const int M = sb.n_seqs * S;
  if (a->rope) {
    rc = ensure_rope_table(p, hd, rope_base, prm.max_pages_per_seq * prm.page_tokens);
    if (rc) return rc;
  }
  const void* dx = nullptr;
  rc = stage_in(p, p->in_a, a->x, (size_t)M * D * 4, a->x_mem, &dx);
  if (rc) return rc;
  const WeightRef proj[3] = {{w.w_q, H * hd}, {w.w_k, Hkv * hd}, {w.w_v, Hkv * hd}};
  const WeightRef outp[1] = {{w.w_o, D}};
  const int n_total = (H + 2 * Hkv) * hd;
  const bool fast = a->mode == RELUX_ATTN_FAST;
  const bool mma = fast && !p->tune.get(RELUX_TUNE_GEMM_GENERIC) && gemm_sm100_eligible(D, proj, 3) && gemm_sm100_eligible(H * hd, outp, 1);
  const size_t q_es = fast ? 2 : 4;
  const size_t b_q = pad256((size_t)M * H * hd * q_es), b_kv = pad256((size_t)M * Hkv * hd * 4);
  LayerScratch sc;
  rc = layer_scratch(p, M, std::max(D, H * hd), std::max(n_total, D), b_q + 2 * b_kv + (size_t)M * H * hd * 4, &sc);
  if (rc) return rc;
  void* d_q = sc.rest;
  float* d_k = (float*)(sc.rest + b_q);
  float* d_v = (float*)(sc.rest + b_q + b_kv);
  float* d_attn = (float*)(sc.rest + b_q + 2 * b_kv);
  const int rd = a->rope ? hd : 0;
  const ProjSeg segs[3] = {{H * hd, rd, d_q, fast ? 1 : 0, S > 1}, {Hkv * hd, rd, d_k, 0, 0}, {Hkv * hd, 0, d_v, 0, 0}};
  rc = project_and_finish(p, sb, a->layer, (const float*)dx, M, D, S, proj, segs, 3, mma, sc.a_bf16, sc.part, sc.part_cap, faithful);
  if (rc) return rc;
  // append: the GEMM rows are token-major [row][Hkv][hd]; advance = 0 leaves the rows past the cursor (verify).  A short
  // step leaves the append to the attention launch.
  relux_attn_args aa;
  memset(&aa, 0, sizeof(aa));
  aa.mode = a->mode;
  aa.num_heads = H;
  aa.q_tokens = S;
  aa.extra_tokens = a->advance ? 0 : S;
  const bool fused_append = fast && gqa_append_fusable(p, aa, S, a->advance != 0);
  if (!fused_append) {
    rc = launch_gqa_append(p, sb, a->layer, d_k, d_v, RELUX_DTYPE_F32, RELUX_LAYOUT_TOKEN_MAJOR, a->advance);
    if (rc) return rc;
  }
  if (a->advance)
    for (int i = 0; i < sb.n_seqs; i++) {
      int32_t& len = p->h_len[(size_t)a->layer * prm.max_seqs + sb.seq[i]];
      note_append(p, a->layer, sb.seq[i], len, S);
      len += S;
    }
  aa.layer = a->layer;
  aa.n_seqs = sb.n_seqs;
  aa.seq_ids = a->seq_ids;
  aa.causal = a->causal;
  aa.head_dim = hd;
  aa.scale = (float)(1.0 / std::sqrt((double)hd));   // mha.go:319
  aa.q_dtype = fast ? RELUX_DTYPE_BF16 : RELUX_DTYPE_F32;
  aa.q_layout = RELUX_LAYOUT_TOKEN_MAJOR;
  const GqaAppend app{d_k, d_v, RELUX_DTYPE_F32, RELUX_LAYOUT_TOKEN_MAJOR, a->advance ? 1 : 0, sb.rows.data()};
  const bool o_bf16 = mma && fused_append;   // the output projection's operand, rounded by the kernel that makes it
  rc = fused_append ? launch_gqa_stream(p, sb, aa, d_q, o_bf16 ? (void*)sc.a_bf16 : d_attn, o_bf16, &app)
       : fast       ? launch_gqa_decode_fast(p, sb, aa, d_q, d_attn)
                    : launch_attn_reference_gqa(p, sb, aa, (const float*)d_q, d_attn);
  if (rc) {
    if (fused_append && a->advance) take_rows_back(p, sb, a->layer);   // nobody appended them
    return rc;
  }
  return output_projection(p, o_bf16 ? nullptr : d_attn, M, H * hd, w.w_o, D, mma, sc.a_bf16, sc.part, sc.part_cap, a->out, a->out_mem);
}

// ComputeBackend.MatMulFloat32 as matmulBatched3D uses it (interface.go:25-29, mha.go:759-785): C = A x B with A, C float32
// and B a bf16 weight matrix [K][N] on the device.
int32_t do_matmul(Pool* p, const relux_matmul_args* a) {
  if (!a || !a->a || !a->b || !a->c) { set_error("nil argument"); return RELUX_ERR_INVALID_ARG; }
  const int M = a->m, K = a->k, N = a->n;
  if (M <= 0 || K <= 0 || N <= 0) { set_error("MatMulFloat32: M=%d K=%d N=%d must be positive", M, K, N); return RELUX_ERR_INVALID_ARG; }
  if (a->mode != RELUX_ATTN_FAST && a->mode != RELUX_ATTN_REFERENCE) { set_error("bad mode"); return RELUX_ERR_INVALID_ARG; }
  for (int i = 0; i < 4; i++)
    if (a->reserved[i]) { set_error("reserved fields must be zero"); return RELUX_ERR_INVALID_ARG; }
  int32_t rc;
  if ((rc = check_dev_align(a->b, "B"))) return rc;
  if (a->a_mem == RELUX_MEM_DEVICE && (rc = check_dev_align(a->a, "A"))) return rc;
  if (a->c_mem == RELUX_MEM_DEVICE && (rc = check_dev_align(a->c, "C"))) return rc;
  const WeightRef w[1] = {{a->b, N}};
  const bool fast = a->mode == RELUX_ATTN_FAST;
  if (fast && (p->tune.get(RELUX_TUNE_GEMM_GENERIC) || !gemm_sm100_eligible(K, w, 1) || N % 4 != 0)) {
    set_error("MatMulFloat32 FAST needs K and N multiples of 8 (got K=%d N=%d); use RELUX_ATTN_REFERENCE", K, N);
    return RELUX_ERR_UNSUPPORTED;
  }
  const void* dA = nullptr;
  rc = stage_in(p, p->in_a, a->a, (size_t)M * K * 4, a->a_mem, &dA);
  if (rc) return rc;
  LayerScratch sc;
  rc = layer_scratch(p, M, K, N, 0, &sc);
  if (rc) return rc;
  return output_projection(p, (const float*)dA, M, K, a->b, N, fast, sc.a_bf16, sc.part, sc.part_cap, a->c, a->c_mem);
}

}  // namespace relux
