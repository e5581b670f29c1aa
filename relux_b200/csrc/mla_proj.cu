// The two small per-head GEMMs around the absorbed MLA decode, on tensor cores (mma.sync m16n8k16, bf16 in,
// f32 accumulate):
//   absorb:  q~[row][h][0:dC]  = q_nope[row][h][:] . W_UK[:, h*Dh:(h+1)*Dh]^T      M = rows, N = dC,  K = Dh
//            q~[row][h][dC: ]  = q_rope[row][h][:]
//   up-proj: out[row][h][:]    = O_lat[row][h][:] . W_UV[:, h*Dh:(h+1)*Dh]          M = rows, N = Dh,  K = dC
// Both are about 1 GFLOP per step at batch 64 (1.5 % of the decode's work) and move ~30 MB; they are written to stay
// out of the way of the decode kernel, not to chase the tensor peak: one CTA per (head, 128-wide slice, 64 rows),
// operands staged in shared memory by a few TMA boxes (every load of a CTA in flight at once), fragments through
// ldmatrix (the up-projection of more than 16 rows runs on tcgen05).  The up-projection also performs the split-KV merge while it
// builds its operand.
// Shapes: Dh = 128, dC a multiple of 128.  Other shapes use the scalar kernels in mla_decode.cu.
#include "common.cuh"
#include "internal.h"
#include "prep_parts.cuh"
#include "umma.cuh"

namespace relux {

namespace {

constexpr int kDh = 128;
constexpr int kStride = kDh + 8;  // bf16 elements per shared-memory row (272 B: conflict-free ldmatrix)
constexpr int kMergeBlk = 8192;   // 64 rows x 64 columns of the merged operand
constexpr int kMaxChunks = 4;     // the fused merge + up-projection keeps at most 4 x 128 latent columns in shared memory

// 64 rows x 128 latent columns of the absorb for one head, by 128 threads.  W_UK's tile [128 c][128 d] and (bf16) the query
// tile [64 rows][128 d] come as four TMA boxes from one thread: as 3072 cp.async of 16 bytes they took 2.2 us to issue.  Both
// lie as two 64-column blocks with the 128-byte swizzle.  Up to 32 rows, the warps share the row groups that hold a row.
// Measured (the whole preparation launch, before -> now): 3 rows 8.1 -> 4.7 us, 64 rows 12.6 -> 12.0 us.
// The result leaves through shared memory as 16-byte row-contiguous stores.
constexpr int kAbsorbSmem = 32768 + 16384 + 1024;
__device__ __forceinline__ void absorb_block(uint8_t* sm_raw, const CUtensorMap* tmap_w, const CUtensorMap* tmap_q, const void* __restrict__ q_nope,
                                             const void* __restrict__ q_rope, int q_bf16, uint16_t* __restrict__ q_abs, int rows, int H, int dC,
                                             int dHR, int bx, int by, int bz, int32_t* status, bool chained, bool wait_for_queries) {
  __shared__ __align__(8) uint64_t landed;
  uint8_t* sm = (uint8_t*)(((uintptr_t)sm_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* Bs = sm;             // [2 halves of d][128 c][64], swizzled
  uint8_t* As = sm + 32768;     // [2 halves of d][64 rows][64], swizzled
  const int h = bx, c0 = by * 128, r0 = bz * 64;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_here = min(64, rows - r0), groups = rows_here <= 16 ? 1 : rows_here <= 32 ? 2 : 4;
  if (threadIdx.x == 0) {
    mbar_init(&landed, 1);
    fence_mbar_init();
    mbar_expect_tx(&landed, 32768 + (q_bf16 ? 16384 : 0));
    tma_load_2d(Bs, tmap_w, h * kDh, c0, &landed);
    tma_load_2d(Bs + 16384, tmap_w, h * kDh + 64, c0, &landed);
  }
  if (wait_for_queries) chain_wait();
  if (q_bf16) {
    if (threadIdx.x == 0) {   // rows past the batch are zero-filled
      tma_load_2d(As, tmap_q, h * kDh, r0, &landed);
      tma_load_2d(As + 8192, tmap_q, h * kDh + 64, r0, &landed);
    }
  } else {
#pragma unroll 4
    for (int e = threadIdx.x; e < groups * 16 * (kDh / 8); e += blockDim.x) {
      const int r = e / (kDh / 8), v = e % (kDh / 8);
      uint4 w = make_uint4(0, 0, 0, 0);
      if (r < rows_here) {
        const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q_nope) + ((size_t)(r0 + r) * H + h) * kDh + (size_t)v * 8);
        const float4 x = load_chained(s), y = load_chained(s + 1);
        w = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
      }
      *reinterpret_cast<uint4*>(As + (v >> 3) * 8192 + swz128(r, v & 7)) = w;
    }
  }
  const int roww = dC + dHR;
  if (by == 0) {   // the rope part of q~ is a copy (with the same rounding when the source is float32)
    const int vecs = dHR / 8;
    for (int e = threadIdx.x; e < rows_here * vecs; e += blockDim.x) {
      const int r = e / vecs, v = e % vecs;
      const size_t off = ((size_t)(r0 + r) * H + h) * dHR + (size_t)v * 8;
      uint4 w;
      if (q_bf16) w = load_chained(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(q_rope) + off));
      else {
        const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q_rope) + off);
        const float4 x = load_chained(s), y = load_chained(s + 1);
        w = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
      }
      *reinterpret_cast<uint4*>(q_abs + ((size_t)(r0 + r) * H + h) * roww + dC + (size_t)v * 8) = w;
    }
  }
  __syncthreads();   // the barrier and the float32 rows are visible
  if (!mbar_wait(&landed, 0)) set_status(status, RELUX_ERR_TIMEOUT);   // bounded: a load that never lands is reported
  // warp: 16 rows x 32 * groups columns
  const int m = lane >> 3, row_w = (warp % groups) * 16, col_w = (warp / groups) * 32 * groups;
  const uint32_t a_base = smem_u32(As), b_base = smem_u32(Bs);
  float acc[16][4];
#pragma unroll
  for (int i = 0; i < 16; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 8; ks++) {
    uint32_t a[4];
    const int ka = ks * 2 + (m >> 1), kb = ks * 2 + (m & 1);   // 16-byte chunk of the row
    ldmatrix_x4(a[0], a[1], a[2], a[3], a_base + (ka >> 3) * 8192 + swz128(row_w + (m & 1) * 8 + (lane & 7), ka & 7));
#pragma unroll
    for (int n2 = 0; n2 < 8; n2++) {
      if (n2 >= 2 * groups) break;
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4(b0, b1, b2, b3, b_base + (kb >> 3) * 16384 + swz128(col_w + n2 * 16 + (m >> 1) * 8 + (lane & 7), kb & 7));
      mma_bf16_16816(acc[2 * n2], a, b0, b1);
      mma_bf16_16816(acc[2 * n2 + 1], a, b2, b3);
    }
  }
  __syncthreads();   // every warp is done with As / Bs: Bs becomes the output staging tile
  uint16_t* Os = reinterpret_cast<uint16_t*>(Bs);
#pragma unroll
  for (int hf = 0; hf < 2; hf++) {
    const int r = row_w + hf * 8 + (lane >> 2);
#pragma unroll
    for (int nt = 0; nt < 16; nt++) {
      if (nt >= 4 * groups) break;
      *reinterpret_cast<uint32_t*>(Os + r * kStride + col_w + nt * 8 + 2 * (lane & 3)) = pack_bf16x2(acc[nt][hf * 2], acc[nt][hf * 2 + 1]);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < rows_here * 16; e += blockDim.x) {
    const int r = e / 16, v = e % 16;
    *reinterpret_cast<uint4*>(q_abs + ((size_t)(r0 + r) * H + h) * roww + c0 + v * 8) = *reinterpret_cast<const uint4*>(Os + r * kStride + v * 8);
  }
  if (chained) fence_chained_writes();
}

// grid (H, dC/128, ceil(rows/64)), 128 threads.  A plain launch that releases nobody early: the decode kernel reads its rows by TMA
// behind its end.
__global__ void __launch_bounds__(128) mla_absorb_mma_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_q,
                                                             const void* __restrict__ q_nope, const void* __restrict__ q_rope, int q_bf16,
                                                             uint16_t* __restrict__ q_abs, int rows, int H, int dC, int dHR, int32_t* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  absorb_block(smem_raw, &tmap_w, &tmap_q, q_nope, q_rope, q_bf16, q_abs, rows, H, dC, dHR, blockIdx.x, blockIdx.y, blockIdx.z, status, false, false);
}

// The preparation of one MLA decode step in ONE launch: blocks 0 .. n_seqs - 1 append the step's new rows (a sequence
// each), block n_seqs builds the stream partition, and the blocks after them are the absorb grid (head fastest, then the
// dC / 128 latent slices, then 64 rows each).  The three jobs are independent of one another: the append reads the lengths
// before it writes, the partition counts every sequence's new rows itself, and the last of those blocks to finish advances
// the lengths.  They come first because theirs is the longer chain of dependent reads.
// The kernel releases the launches after it only when everything before it is complete (the up-projection fetches its
// weights without a wait of its own), unless the launches before it in the call have seen to that (weights_ready): its own
// weights are then fetched ahead of its wait too.
__global__ void __launch_bounds__(128) mla_prep_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_q,
                                                       const void* __restrict__ q_nope, const void* __restrict__ q_rope, int q_bf16,
                                                       uint16_t* __restrict__ q_abs, int rows, int H, int dC, int dHR, int weights_ready,
                                                       const __grid_constant__ PrepAppend ap, const __grid_constant__ PrepPlan pl) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int e = blockIdx.x;
  if (!weights_ready) chain_wait();   // also: the kernel before this one may still be reading what this one overwrites
  chain_release();
  if (e > ap.n_seqs) {
    const int a = e - ap.n_seqs - 1, slices = dC / 128;
    absorb_block(smem_raw, &tmap_w, &tmap_q, q_nope, q_rope, q_bf16, q_abs, rows, H, dC, dHR, a % H, a / H % slices, a / H / slices, ap.status,
                 true, weights_ready != 0);
    return;
  }
  if (weights_ready) chain_wait();
  if (e < ap.n_seqs) prep_append_seq(ap, e);
  else prep_build_stream(ap, pl);
  prep_arrive_and_advance(ap, (uint32_t)ap.n_seqs + 1u);
}

// 16 rows x 16 columns of a warp, over one 128-wide k chunk: A rows at As (kStride), B [128 k][128 n] at Bs as two 64-column
// blocks with the 128-byte swizzle (n contiguous -> ldmatrix.trans).
__device__ __forceinline__ void tile_mma_16x16(const uint16_t* As, uint32_t Bs, float (&acc)[2][4], int col0, int lane) {
  const int m = lane >> 3;
#pragma unroll
  for (int ks = 0; ks < 8; ks++) {
    uint32_t a[4];
    ldmatrix_x4(a[0], a[1], a[2], a[3], smem_u32(As + ((m & 1) * 8 + (lane & 7)) * kStride + ks * 16 + (m >> 1) * 8));
    const int krow = ks * 16 + (m & 1) * 8 + (lane & 7);
    const int col = col0 + (m >> 1) * 8;
    uint32_t b0, b1, b2, b3;
    ldmatrix_x4_trans(b0, b1, b2, b3, Bs + (col >> 6) * 16384 + swz128(krow, (col & 63) >> 3));
    mma_bf16_16816(acc[0], a, b0, b1);
    mma_bf16_16816(acc[1], a, b2, b3);
  }
}

// Merges the split-KV partials of the tile's rows into the bf16 A operand, one warp per row at a time: a lane owns the
// same 4 of every 128 latent columns, so every load instruction of a warp is 512 contiguous bytes of one partial row
// (four threads per row with 128 bytes each, the first layout, put 32 different cache lines into every load
// instruction: the kernel spent most of its time in the load unit's address stage).  The weights of a row's items come
// from one round trip: lane j reads (max, sum) of item j, the warp reduces.
// kChunks: 128-column chunks of a warp, 4 / kChunks warps share a row; 16 / kChunks items are in flight per lane.  A call of
// up to four rows has more warps than rows, and its rows the most items (each worker holds a piece of some sequence).
// Rows past the batch are zero rows of the MMA tile.  The pointers have come through behind_wait().
constexpr int kMergeWarps = 16;
template <int kChunks>
__device__ __forceinline__ void merge_rows_warp(uint16_t* As, const float* part_o, const float* part_ml, const int32_t* chunk_off,
                                                int rows, int S, int H, int h, int dC, int nk_all, int rows_total) {
  constexpr int kParts = kMaxChunks / kChunks, kItems = 16 / kChunks, kRowStep = kMergeWarps / kParts;
  const int warp = (int)(threadIdx.x >> 5) / kParts, lane = threadIdx.x & 31;   // the warp's first row of the tile
  const int k0 = (int)(threadIdx.x >> 5) % kParts * kChunks, nk = min(kChunks, nk_all - k0);
  if (nk <= 0) return;
  part_o += k0 * 128;
  As += (size_t)k0 * 16 * kStride;
  // The item range of a row is the first of two dependent round trips to L2, so it is requested one row ahead.
  int c0_next = 0, c1_next = 0;
  if (warp < rows) {
    const int i = warp / S;
    c0_next = load_settled(chunk_off + i);
    c1_next = load_settled(chunk_off + i + 1);
  }
  for (int r = warp; r < 16; r += kRowStep) {
    const int c0 = c0_next, c1 = c1_next;
    c0_next = c1_next = 0;
    if (r + kRowStep < rows) {
      const int i = (r + kRowStep) / S;
      c0_next = load_settled(chunk_off + i);
      c1_next = load_settled(chunk_off + i + 1);
    }
    float4 acc[kChunks];
#pragma unroll
    for (int k = 0; k < kChunks; k++) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) {
      const size_t prow = (size_t)(r % S) * H + h;
      // (max, sum) of this lane's item of every group of 32, and at the same time the partial rows of the first
      // items: one memory round trip serves the common case of a sequence cut into a handful of items
      const int n_items = c1 - c0;
      if (n_items <= 0) goto store_row;   // no partial to merge: a zero row
      float2 ml = make_float2(-INFINITY, 0.f);
      if (lane < n_items) ml = load_settled(reinterpret_cast<const float2*>(part_ml + ((size_t)(c0 + lane) * rows_total + prow) * 2));
      float4 x[kItems][kChunks];
      const int ng0 = min(32, n_items);
#pragma unroll
      for (int u = 0; u < kItems; u++) {
        // a slot past the group's last item stays zero (its weight is zero too): the load unit's data path, 128 bytes
        // per clock for all 16 warps, is what a row's requests queue on, so no load is spent on padding
        const float4* src = reinterpret_cast<const float4*>(part_o + ((size_t)(c0 + u) * rows_total + prow) * dC) + lane;
#pragma unroll
        for (int k = 0; k < kChunks; k++)
          if (k < nk) x[u][k] = load_settled_if(src + k * 32, u < ng0);
      }
      // global maximum and normaliser over all items of the sequence
      float M = ml.x;
      for (int c = c0 + 32 + lane; c < c1; c += 32) M = fmaxf(M, load_settled(part_ml + ((size_t)c * rows_total + prow) * 2));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
      float L = (ml.x != -INFINITY) ? ml.y * exp2f(ml.x - M) : 0.f;
      for (int c = c0 + 32 + lane; c < c1; c += 32) {
        const float2 t = load_settled(reinterpret_cast<const float2*>(part_ml + ((size_t)c * rows_total + prow) * 2));
        if (t.x != -INFINITY) L += t.y * exp2f(t.x - M);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
      const float inv = (L > 0.f) ? 1.0f / L : 0.f;
      for (int cb = c0; cb < c1; cb += 32) {
        // this lane's item of the group of 32: its weight; then kItems at a time, weights by shuffle
        float w_mine = 0.f;
        if (cb == c0) {
          w_mine = (ml.x == -INFINITY) ? 0.f : exp2f(ml.x - M) * inv;
        } else if (cb + lane < c1) {
          const float m = load_settled(part_ml + ((size_t)(cb + lane) * rows_total + prow) * 2);
          w_mine = (m == -INFINITY) ? 0.f : exp2f(m - M) * inv;
        }
        const int ng = min(32, c1 - cb);
        for (int j = 0; j < ng; j += kItems) {
          if (cb != c0 || j != 0) {   // the first items of the row are in flight already
#pragma unroll
            for (int u = 0; u < kItems; u++) {
              const float4* src = reinterpret_cast<const float4*>(part_o + ((size_t)(cb + j + u) * rows_total + prow) * dC) + lane;
#pragma unroll
              for (int k = 0; k < kChunks; k++)
                if (k < nk) x[u][k] = load_settled_if(src + k * 32, j + u < ng);
            }
          }
#pragma unroll
          for (int u = 0; u < kItems; u++) {
            float w = __shfl_sync(0xffffffffu, w_mine, min(j + u, 31));
            if (j + u >= ng) w = 0.f;
#pragma unroll
            for (int k = 0; k < kChunks; k++)
              if (k < nk) {
                acc[k].x = fmaf(x[u][k].x, w, acc[k].x);
                acc[k].y = fmaf(x[u][k].y, w, acc[k].y);
                acc[k].z = fmaf(x[u][k].z, w, acc[k].z);
                acc[k].w = fmaf(x[u][k].w, w, acc[k].w);
              }
          }
        }
      }
    }
  store_row:
#pragma unroll
    for (int k = 0; k < kChunks; k++)
      if (k < nk)
        *reinterpret_cast<uint2*>(As + ((size_t)k * 16 + r) * kStride + lane * 4) =
            make_uint2(pack_bf16x2(acc[k].x, acc[k].y), pack_bf16x2(acc[k].z, acc[k].w));
  }
}

// Split-KV merge fused into the value up-projection, for up to 16 rows and one head: the A operand (the merged, normalised latent
// output as bf16) is built straight from the per-item partials
//   part_o [item][S * H][dC] f32 (unnormalised), part_ml [item][S * H][2] = (max in the log2 domain, sum),
// items of sequence i = [chunk_off[i], chunk_off[i + 1]).
// All of W_UV's slice for this head (dC x 128 bf16) is fetched by one thread as 2 * nk TMA boxes before chain_wait(): the
// weights do not depend on the decode kernel, and the launches before it have waited for everything older (as 512 bulk
// copies of a row each, issued behind the merge's first loads, they took 2-3 us to be accepted).  Eight warps share the MMAs, chunk by
// chunk as the boxes land.
// grid (H), 512 threads, row = seq_index * S + query token.  dC = 128 * nk, nk <= 4.
__global__ void __launch_bounds__(32 * kMergeWarps) mla_merge_vup_mma_kernel(const __grid_constant__ CUtensorMap tmap_w, const float* part_o,
                                                                const float* part_ml, const int32_t* chunk_off,
                                                                void* __restrict__ out, int out_bf16, int rows, int S, int H, int dC,
                                                                int32_t* __restrict__ status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t w_full[kMaxChunks];   // chunk k of W_UV has landed (bytes counted by the TMA loads)
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int nk = dC / 128;
  const uint32_t Bs = smem_u32(smem);                                       // [nk][2 halves of 64 columns][128][64], swizzled
  uint16_t* As = reinterpret_cast<uint16_t*>(smem + (size_t)nk * 32768);    // [nk][16][kStride]
  const int h = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_total = S * H;
  chain_release();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    for (int k = 0; k < nk; k++) mbar_init(&w_full[k], 1);
    fence_mbar_init();
    for (int k = 0; k < nk; k++) {
      mbar_expect_tx(&w_full[k], 32768);
      tma_load_2d(smem + (size_t)k * 32768, &tmap_w, h * kDh, k * 128, &w_full[k]);
      tma_load_2d(smem + (size_t)k * 32768 + 16384, &tmap_w, h * kDh + 64, k * 128, &w_full[k]);
    }
  }
  chain_wait();   // the partial results come from the kernel before this one
  part_o = behind_wait(part_o);
  part_ml = behind_wait(part_ml);
  chunk_off = behind_wait(chunk_off);
  if (rows <= 4) merge_rows_warp<1>(As, part_o, part_ml, chunk_off, rows, S, H, h, dC, nk, rows_total);
  else if (rows <= 8) merge_rows_warp<2>(As, part_o, part_ml, chunk_off, rows, S, H, h, dC, nk, rows_total);
  else merge_rows_warp<4>(As, part_o, part_ml, chunk_off, rows, S, H, h, dC, nk, rows_total);
  float acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
  __syncthreads();   // the merged A tiles are complete, and the barriers visible
  const int col0 = warp * 16;
  if (col0 >= kDh) return;
  for (int k = 0; k < nk; k++) {
    if (!mbar_wait(&w_full[k], 0)) set_status(status, RELUX_ERR_TIMEOUT);   // bounded: a copy that never lands is reported, not waited for
    tile_mma_16x16(As + (size_t)k * 16 * kStride, Bs + k * 32768, acc, col0, lane);
  }
#pragma unroll
  for (int hf = 0; hf < 2; hf++) {
    const int r = hf * 8 + (lane >> 2);
    if (r >= rows) continue;
    const size_t off = ((size_t)r * H + h) * kDh + col0 + 2 * (lane & 3);
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      const float x = acc[nt][hf * 2], y = acc[nt][hf * 2 + 1];
      if (out_bf16) *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(out) + off + nt * 8) = pack_bf16x2(x, y);
      else *reinterpret_cast<float2*>(reinterpret_cast<float*>(out) + off + nt * 8) = make_float2(x, y);
    }
  }
  if (out_bf16) fence_chained_writes();   // a projection's operand
}

// The same for a tile of up to 64 rows, a warp a row: the item range of the warp's row is requested two rows ahead, (max, sum) of its
// items one row ahead, and the partial rows, two items at a time, before the ones they follow are added up.  The loop over the rows
// stays a loop: unrolled, the kernel waited for its own instructions.  Rows past rows_here are left as they are.
__device__ __forceinline__ void merge_rows_piped(uint8_t* As, const float* part_o, const float* part_ml, const int32_t* chunk_off,
                                                int r0, int rows_here, int S, int H, int h, int dC, int nk, int rows_total) {
  constexpr int kChunks = kMaxChunks, kItems = 2, kRowStep = kMergeWarps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;   // the warp's first row of the tile
  part_o += lane * 4;
  struct Row {
    int c0, n;   // first item, items
    int pr;      // row of an item's partial block
  };
  auto row_at = [&](int row) -> Row {   // a row past the tile has no items
    Row r{0, 0, 0};
    if (row < rows_here) {
      const int i = (r0 + row) / S;
      r.c0 = load_settled(chunk_off + i);
      r.n = load_settled(chunk_off + i + 1);   // its end, for now
      r.pr = (r0 + row) % S * H + h;
    }
    return r;
  };
  auto ml_of = [&](const Row& r, int j) {
    return load_settled(reinterpret_cast<const float2*>(part_ml + ((size_t)(r.c0 + j) * rows_total + r.pr) * 2));
  };
  float4 x[kItems][kChunks], y[kItems][kChunks];
  auto fetch = [&](float4 (&z)[kItems][kChunks], const Row& r, int j) {   // a slot past the row's last item stays zero: no load is spent on it
    const float* src = part_o + ((size_t)(r.c0 + j) * rows_total + r.pr) * dC;
#pragma unroll
    for (int u = 0; u < kItems; u++) {
#pragma unroll
      for (int k = 0; k < kChunks; k++)
        if (k < nk) z[u][k] = load_settled_if(reinterpret_cast<const float4*>(src) + k * 32, j + u < r.n);
      src += (size_t)rows_total * dC;
    }
  };
  Row cur = row_at(warp), nxt = row_at(warp + kRowStep);
  cur.n -= cur.c0;
  float2 ml = make_float2(-INFINITY, 0.f);
  if (lane < cur.n) ml = ml_of(cur, lane);
  fetch(x, cur, 0);
#pragma unroll 1
  for (int row = warp; row < rows_here; row += kRowStep) {
    nxt.n -= nxt.c0;
    float2 ml_next = make_float2(-INFINITY, 0.f);
    if (lane < nxt.n) ml_next = ml_of(nxt, lane);
    const Row after = row_at(row + 2 * kRowStep);
    // weights of the row's first 32 items: 2^(m - M) / L
    float M = ml.x;
    for (int j = 32 + lane; j < cur.n; j += 32) M = fmaxf(M, ml_of(cur, j).x);
    M = warp_max(M);
    float w = (ml.x != -INFINITY) ? exp2f(ml.x - M) : 0.f;
    float L = ml.y * w;
    for (int j = 32 + lane; j < cur.n; j += 32) {
      const float2 m = ml_of(cur, j);
      if (m.x != -INFINITY) L += m.y * exp2f(m.x - M);
    }
    L = warp_sum(L);
    const float inv = (L > 0.f) ? 1.0f / L : 0.f;
    w *= inv;
    float4 acc[kChunks];
#pragma unroll
    for (int k = 0; k < kChunks; k++) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    int j = 0;
#pragma unroll 1
    do {   // a row without items adds up the zeros that fetch left
      const bool more = j + kItems < cur.n;
      fetch(y, more ? cur : nxt, more ? j + kItems : 0);
      if (j > 0 && (j & 31) == 0) {
        w = 0.f;
        if (j + lane < cur.n) {
          const float m = ml_of(cur, j + lane).x;
          if (m != -INFINITY) w = exp2f(m - M) * inv;
        }
      }
#pragma unroll
      for (int u = 0; u < kItems; u++) {
        const float wu = __shfl_sync(0xffffffffu, w, (j + u) & 31);
#pragma unroll
        for (int k = 0; k < kChunks; k++)
          if (k < nk) {
            acc[k].x = fmaf(x[u][k].x, wu, acc[k].x);
            acc[k].y = fmaf(x[u][k].y, wu, acc[k].y);
            acc[k].z = fmaf(x[u][k].z, wu, acc[k].z);
            acc[k].w = fmaf(x[u][k].w, wu, acc[k].w);
          }
      }
#pragma unroll
      for (int u = 0; u < kItems; u++)
#pragma unroll
        for (int k = 0; k < kChunks; k++) x[u][k] = y[u][k];
      j += kItems;
    } while (j < cur.n);
#pragma unroll
    for (int k = 0; k < kChunks; k++)
      if (k < nk)
        *reinterpret_cast<uint2*>(As + (k * 2 + (lane >> 4)) * kMergeBlk + swz128(row, (lane & 15) >> 1) + (lane & 1) * 8) =
            make_uint2(pack_bf16x2(acc[k].x, acc[k].y), pack_bf16x2(acc[k].z, acc[k].w));
    cur = nxt;
    nxt = after;
    ml = ml_next;
  }
}

// Split-KV merge fused into the value up-projection, for one head and up to 64 rows: the merged, normalised latent output is built as
// bf16 straight from the per-item partials
//   part_o [item][S * H][dC] f32 (unnormalised), part_ml [item][S * H][2] = (max in the log2 domain, sum),
// items of sequence i = [chunk_off[i], chunk_off[i + 1]),
// and D[128 output dims x rows] = W_UV^T O on tcgen05: the weights are the M = 128 operand as they lie (MN-major), the rows the N
// operand (16, 32 or 64, K-major blocks of 64 columns), one tensor-memory column per row.  Rows of the tile past the batch hold
// whatever shared memory held: their columns of D are not read.
// Clock stamps at 64 sequences of 4096 tokens, 64 rows of one item each: merge 15-16 k, MMAs 3.2 k, of which their issue is 2.8 k, the
// outputs 1.5 k.  (With two items a row, the plan of equal ranges: merge 15-16.5 k, 17-22 k with one row's round trips after another; MMAs
// by mma.sync, whose fragments come from shared memory four times each, 7 k.)  The code runs once and waits for its own instructions: an
// operand more, for what the rows' rounding leaves, took 2-3 us of the launch, not the 0.4 of its MMAs, and one MMA a turn 3.
// All of W_UV's slice for this head (dC x 128 bf16) is fetched by one thread as 2 * nk TMA boxes before chain_wait(): the
// weights do not depend on the decode kernel, and the launches before it have waited for everything older (as 512 bulk
// copies of a row each, issued behind the merge's first loads, they took 2-3 us to be accepted).
// grid (H, ceil(rows/64)), 512 threads, row = seq_index * S + query token.  dC = 128 * nk, nk <= 4.
__global__ void __launch_bounds__(32 * kMergeWarps, 1) mla_merge_vup_sm100_kernel(const __grid_constant__ CUtensorMap tmap_w, const float* part_o,
                                                                const float* part_ml, const int32_t* chunk_off,
                                                                void* __restrict__ out, int out_bf16, int rows, int S, int H, int dC,
                                                                int32_t* __restrict__ status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t w_full[kMaxChunks], done;   // chunk k of W_UV has landed (bytes counted by the TMA loads); D is complete
  __shared__ uint32_t tmem_slot;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int nk = dC / 128;
  uint8_t* Ws = smem;                           // [nk][2 halves of 64 columns][128][64], swizzled
  uint8_t* As = smem + (size_t)nk * 32768;      // [2 nk][64 rows][64], swizzled
  const int h = blockIdx.x, r0 = blockIdx.y * 64;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  chain_release();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmap_w);
    for (int k = 0; k < nk; k++) mbar_init(&w_full[k], 1);
    mbar_init(&done, 1);
    fence_mbar_init();
    for (int k = 0; k < nk; k++) {
      mbar_expect_tx(&w_full[k], 32768);
      tma_load_2d(Ws + (size_t)k * 32768, &tmap_w, h * kDh, k * 128, &w_full[k]);
      tma_load_2d(Ws + (size_t)k * 32768 + 16384, &tmap_w, h * kDh + 64, k * 128, &w_full[k]);
    }
  }
  if (warp == 1) {
    tmem_alloc<1>(&tmem_slot, 64);
    tmem_relinquish<1>();
  }
  chain_wait();   // the partial results come from the kernel before this one
  part_o = behind_wait(part_o);
  part_ml = behind_wait(part_ml);
  chunk_off = behind_wait(chunk_off);
  const int rows_here = min(64, rows - r0), n_tile = rows_here <= 16 ? 16 : rows_here <= 32 ? 32 : 64;
  merge_rows_piped(As, part_o, part_ml, chunk_off, r0, rows_here, S, H, h, dC, nk, S * H);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();   // the merged rows are complete, the barriers and the tensor memory's address visible
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (warp == 0) {
    const bool el = elect_one();
    const uint32_t idesc = make_idesc_bf16(128, n_tile, true, false);
    const uint64_t dW = make_desc_mnmajor_sw128(smem_u32(Ws), 16384), dA = make_desc_kmajor_sw128(smem_u32(As));
    for (int k = 0; k < nk; k++) {
      if (!mbar_wait(&w_full[k], 0)) set_status(status, RELUX_ERR_TIMEOUT);   // bounded: a copy that never lands is reported, not waited for
      __syncwarp();
      if (el) {
#pragma unroll
        for (int ks = 0; ks < 8; ks++)
          umma_ss<1>(tmem, dW + ((uint32_t)(k * 32768 + ks * 2048) >> 4), dA + ((uint32_t)((2 * k + (ks >> 2)) * kMergeBlk + (ks & 3) * 32) >> 4),
                     idesc, (k | ks) != 0);
      }
      __syncwarp();
    }
    if (el) umma_commit<1>(&done);
    __syncwarp();
  }
  if (!mbar_wait(&done, 0)) set_status(status, RELUX_ERR_TIMEOUT);
  tc_fence_after();
  // lane = output dim 32 (warp & 3) + lane, column = row: every store of a warp is 32 neighbouring dims of a row
  const uint32_t tmem_d = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  size_t off = ((size_t)(r0 + (warp >> 2) * 4) * H + h) * kDh + (warp & 3) * 32 + lane;
#pragma unroll 1
  for (int g = (warp >> 2) * 4; g < rows_here; g += 16, off += (size_t)16 * H * kDh) {
    uint32_t v[4];
    tmem_ld_32x32b_x4(tmem_d + g, v);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (g + j < rows_here) {
        if (out_bf16) reinterpret_cast<uint16_t*>(out)[off + (size_t)j * H * kDh] = (uint16_t)pack_bf16x2(__uint_as_float(v[j]), 0.f);
        else reinterpret_cast<float*>(out)[off + (size_t)j * H * kDh] = __uint_as_float(v[j]);
      }
  }
  tc_fence_before();
  if (out_bf16) fence_chained_writes();   // a projection's operand
  __syncthreads();
  if (warp == 1) tmem_dealloc<1>(tmem, 64);
}

}  // namespace

bool mla_proj_mma_eligible(int Dh, int dC) { return Dh == kDh && dC % 128 == 0; }

// W_UK [dC][H * 128] in 128 x 64 boxes; bf16 queries [rows][H * 128] in 64 x 64 boxes.
static int32_t absorb_maps(const uint16_t* W_UK, const void* q_nope, int q_bf16, int rows, int H, int dC, CUtensorMap* tw, CUtensorMap* tq) {
  if (!make_tmap_2d(tw, (void*)W_UK, (uint64_t)dC, (uint64_t)H * kDh, 64, 128) ||
      (q_bf16 && !make_tmap_2d(tq, (void*)q_nope, (uint64_t)rows, (uint64_t)H * kDh, 64, 64))) {
    set_error("tensor map for w_uk or the queries could not be encoded");
    return RELUX_ERR_CUDA;
  }
  if (!q_bf16) *tq = *tw;
  return RELUX_OK;
}

int32_t launch_mla_absorb_mma(Device* dev, const void* q_nope, const void* q_rope, int q_bf16, const uint16_t* W_UK, uint16_t* q_abs,
                              int rows, int H, int dC, int dHR, int32_t* status) {
  dim3 grid(H, dC / 128, (rows + 63) / 64);
  CUtensorMap tw, tq;
  if (int32_t rc = absorb_maps(W_UK, q_nope, q_bf16, rows, H, dC, &tw, &tq)) return rc;
  if (int32_t rc = allow_smem(dev, mla_absorb_mma_kernel, kAbsorbSmem)) return rc;
  mla_absorb_mma_kernel<<<grid, 128, kAbsorbSmem, dev->stream>>>(tw, tq, q_nope, q_rope, q_bf16, q_abs, rows, H, dC, dHR, status);
  RELUX_CUDA_TRY(cudaGetLastError());
  count_launch(dev);
  return RELUX_OK;
}

// One launch: absorb + append of the step's rows + stream partition (see mla_prep_kernel).
int32_t launch_mla_prep(Device* dev, const void* q_nope, const void* q_rope, int q_bf16, const uint16_t* W_UK, uint16_t* q_abs, int rows,
                        int H, int dC, int dHR, bool weights_ready, const PrepAppend& ap, const PrepPlan& pl, bool chained) {
  const unsigned blocks = (unsigned)ap.n_seqs + 1u + (unsigned)H * (unsigned)(dC / 128) * (unsigned)((rows + 63) / 64);
  CUtensorMap tw, tq;
  if (int32_t rc = absorb_maps(W_UK, q_nope, q_bf16, rows, H, dC, &tw, &tq)) return rc;
  if (int32_t rc = allow_smem(dev, mla_prep_kernel, kAbsorbSmem)) return rc;
  RELUX_CUDA_TRY(launch_chained(chained, mla_prep_kernel, dim3(blocks), dim3(128), (size_t)kAbsorbSmem, dev->stream, tw, tq, q_nope, q_rope, q_bf16,
                                q_abs, rows, H, dC, dHR, weights_ready ? 1 : 0, ap, pl));
  count_launch(dev);
  return RELUX_OK;
}

int32_t launch_mla_merge_vup_mma(Device* dev, const float* part_o, const float* part_ml, const int32_t* chunk_off, const uint16_t* W_UV,
                                 void* out, int out_bf16, int rows, int S, int H, int dC, int32_t* status, bool chained) {
  CUtensorMap tw;   // W_UV [dC][H * 128], 128 x 64 boxes
  if (!make_tmap_2d(&tw, (void*)W_UV, (uint64_t)dC, (uint64_t)H * kDh, 64, 128)) {
    set_error("tensor map for w_uv could not be encoded");
    return RELUX_ERR_CUDA;
  }
  dim3 grid(H, (rows + 63) / 64);
  // Up to 16 rows a warp has one row, with four items of it in flight, and eight warps' MMAs are short; beyond, rows follow one another
  // in a warp.  64 rows (64 x 4096): the call takes 98.9 us by mma.sync, 96.7 by tcgen05; 16 rows (16 x <= 32k): 97.7 against 99-102.
  if (rows > 16) {
    const size_t smem_tc = (size_t)(dC / 128) * (32768 + 2 * kMergeBlk) + 1024;
    if (int32_t rc = allow_smem(dev, mla_merge_vup_sm100_kernel, smem_tc)) return rc;
    RELUX_CUDA_TRY(launch_chained(chained, mla_merge_vup_sm100_kernel, grid, dim3(32 * kMergeWarps), smem_tc, dev->stream, tw, part_o, part_ml, chunk_off,
                                  out, out_bf16, rows, S, H, dC, status));
    count_launch(dev);
    return RELUX_OK;
  }
  const size_t smem = (size_t)(dC / 128) * (32768 + 16 * kStride * 2) + 1024;
  if (int32_t rc = allow_smem(dev, mla_merge_vup_mma_kernel, smem)) return rc;
  RELUX_CUDA_TRY(launch_chained(chained, mla_merge_vup_mma_kernel, grid, dim3(32 * kMergeWarps), smem, dev->stream, tw, part_o, part_ml, chunk_off,
                                out, out_bf16, rows, S, H, dC, status));
  count_launch(dev);
  return RELUX_OK;
}

}  // namespace relux
