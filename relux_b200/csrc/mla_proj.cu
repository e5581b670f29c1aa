// The two small per-head GEMMs around the absorbed MLA decode, on tensor cores, bf16 in, f32 accumulate:
//   absorb:  q~[row][h][0:dC]  = q_nope[row][h][:] . W_UK[:, h*Dh:(h+1)*Dh]^T      M = rows, N = dC,  K = Dh      (M = dC, N = rows on tcgen05)
//            q~[row][h][dC: ]  = q_rope[row][h][:]
//   up-proj: out[row][h][:]    = O_lat[row][h][:] . W_UV[:, h*Dh:(h+1)*Dh]          M = Dh, N = pieces of rows, K = dC   (tcgen05)
// Both are about 1 GFLOP per step at batch 64 (1.5 % of the decode's work) and move ~30 MB; they are written to stay out of the way of
// the decode kernel, not to chase the tensor peak.  Operands come by a few TMA boxes (every load of a CTA in flight at once).  The up-projection is also the split-KV
// merge: it multiplies every piece and adds the products up.
// Shapes: Dh = 128, dC a multiple of 128.  Other shapes use the scalar kernels in mla_decode.cu.
#include "common.cuh"
#include <algorithm>

#include "internal.h"
#include "prep_parts.cuh"
#include "splitkv.h"
#include "umma.cuh"
#include "vup_plan.h"

namespace relux {

namespace {

constexpr int kDh = 128;

struct AbsorbParams {
  const void* q_nope;
  const void* q_rope;
  uint16_t* q_abs;
  int32_t q_bf16, rows, H, dC, dHR, n_chunks;   // n_chunks: 128 latent columns each, of a CTA
  int32_t* status;
};

// Up to 32 rows x 128 latent columns of the absorb for one head, by 128 threads on mma.sync.  W_UK's tile [128 c][128 d] and (bf16) the query
// tile [32 rows][128 d] come as four TMA boxes from one thread: as 3072 cp.async of 16 bytes they took 2.2 us to issue.  Both
// lie as two 64-column blocks with the 128-byte swizzle; the warps share the row groups that hold a row.  The result leaves through shared
// memory as 16-byte row-contiguous stores.  Four CTAs an SM: their round trips overlap, which for few rows is all there is to gain, and one
// CTA of four chunks on tcgen05 takes 0.1-0.3 us longer (1 x 300 19.5 -> 19.7 us, 30 x 1000 layers 253.6 -> 255.9).
constexpr int kAbsorbMmaThreads = 128, kAbsorbMmaRows = 32;
constexpr size_t kAbsorbMmaSmem = 32768 + 8192 + 1024;
constexpr int kStride = kDh + 8;  // bf16 elements per shared-memory row (272 B: conflict-free ldmatrix)
__device__ __forceinline__ void absorb_block_mma(uint8_t* sm_raw, const CUtensorMap* tmap_w, const CUtensorMap* tmap_q, const AbsorbParams& prm, int bx,
                                                 int by, bool chained, bool weights_ready) {
  const void* const q_nope = prm.q_nope;
  const void* const q_rope = prm.q_rope;
  uint16_t* const q_abs = prm.q_abs;
  const int q_bf16 = prm.q_bf16, H = prm.H, dC = prm.dC, dHR = prm.dHR;
  __shared__ __align__(8) uint64_t landed;
  uint8_t* sm = (uint8_t*)(((uintptr_t)sm_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* Bs = sm;             // [2 halves of d][128 c][64], swizzled
  uint8_t* As = sm + 32768;     // [2 halves of d][32 rows][64], swizzled
  const int h = bx, c0 = by * 128;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_here = prm.rows, groups = rows_here <= 16 ? 1 : 2;
  if (threadIdx.x == 0) {
    mbar_init(&landed, 1);
    fence_mbar_init();
    tma_prefetch_desc(tmap_w);
    tma_prefetch_desc(tmap_q);
    mbar_expect_tx(&landed, 32768 + (q_bf16 ? 8192 : 0));
  }
  auto load_w = [&] {
    if (threadIdx.x == 0) {
      tma_load_2d(Bs, tmap_w, h * kDh, c0, &landed);
      tma_load_2d(Bs + 16384, tmap_w, h * kDh + 64, c0, &landed);
    }
  };
  if (weights_ready) {
    if (chained) chain_release();
    load_w();
  }
  chain_wait();   // also: the kernel before this one may still be reading what this one overwrites
  if (!weights_ready) {
    if (chained) chain_release();
    load_w();
  }
  if (q_bf16) {
    if (threadIdx.x == 0) {   // rows past the batch are zero-filled
      tma_load_2d(As, tmap_q, h * kDh, 0, &landed);
      tma_load_2d(As + 4096, tmap_q, h * kDh + 64, 0, &landed);
    }
  } else {
#pragma unroll 4
    for (int e = threadIdx.x; e < groups * 16 * (kDh / 8); e += blockDim.x) {
      const int r = e / (kDh / 8), v = e % (kDh / 8);
      uint4 w = make_uint4(0, 0, 0, 0);
      if (r < rows_here) {
        const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q_nope) + ((size_t)r * H + h) * kDh + (size_t)v * 8);
        const float4 x = load_chained(s), y = load_chained(s + 1);
        w = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
      }
      *reinterpret_cast<uint4*>(As + (v >> 3) * 4096 + swz128(r, v & 7)) = w;
    }
  }
  const int roww = dC + dHR;
  if (by == 0) {   // the rope part of q~ is a copy (with the same rounding when the source is float32)
    const int vecs = dHR / 8;
    for (int e = threadIdx.x; e < rows_here * vecs; e += blockDim.x) {
      const int r = e / vecs, v = e % vecs;
      const size_t off = ((size_t)r * H + h) * dHR + (size_t)v * 8;
      uint4 w;
      if (q_bf16) w = load_chained(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(q_rope) + off));
      else {
        const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(q_rope) + off);
        const float4 x = load_chained(s), y = load_chained(s + 1);
        w = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
      }
      *reinterpret_cast<uint4*>(q_abs + ((size_t)r * H + h) * roww + dC + (size_t)v * 8) = w;
    }
  }
  __syncthreads();   // the barrier and the float32 rows are visible
  if (!mbar_wait(&landed, 0)) set_status(prm.status, RELUX_ERR_TIMEOUT);   // bounded: a load that never lands is reported
  // warp: 16 rows x 32 * groups columns
  const int m = lane >> 3, row_w = (warp % groups) * 16, col_w = (warp / groups) * 32 * groups;
  const uint32_t a_base = smem_u32(As), b_base = smem_u32(Bs);
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 8; ks++) {
    uint32_t a[4];
    const int ka = ks * 2 + (m >> 1), kb = ks * 2 + (m & 1);   // 16-byte chunk of the row
    ldmatrix_x4(a[0], a[1], a[2], a[3], a_base + (ka >> 3) * 4096 + swz128(row_w + (m & 1) * 8 + (lane & 7), ka & 7));
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
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
    for (int nt = 0; nt < 8; nt++) {
      if (nt >= 4 * groups) break;
      *reinterpret_cast<uint32_t*>(Os + r * kStride + col_w + nt * 8 + 2 * (lane & 3)) = pack_bf16x2(acc[nt][hf * 2], acc[nt][hf * 2 + 1]);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < rows_here * 16; e += blockDim.x) {
    const int r = e / 16, v = e % 16;
    *reinterpret_cast<uint4*>(q_abs + ((size_t)r * H + h) * roww + c0 + v * 8) = *reinterpret_cast<const uint4*>(Os + r * kStride + v * 8);
  }
  if (chained) fence_chained_writes();
}

// The absorb of up to 64 rows for one head and 128, 256 or 512 latent columns (n_chunks of 128), on tcgen05: of every chunk
// D[128 x 128 latent columns] = q W_UK^T, both operands K-major as they lie, in two 64-column blocks with the 128-byte swizzle, by TMA (as 3072
// cp.async of 16 bytes a chunk took 2.2 us to issue).  The M = 128 rows are the queries' 64 twice over, so that all four warps of a group find rows in
// the quarter of tensor memory that they can read, and each takes half of the columns.  Warp 8
// loads and multiplies chunk by chunk, two groups of four warps take the chunks in turn: tensor memory to bf16, through the chunk's own
// weights' place, out by TMA.
// CTAs of one chunk each were started one an SM, by their stamps, once the kernel used tensor memory, four by mma.sync: so a CTA has as many
// chunks as leave no head waiting for a second turn.
// Bound: W_UK from memory (16.8 MB at 128 heads) behind one round trip.  By mma.sync, four CTAs of one chunk an SM, the launch took 9.3-12
// us at 64 rows of 128 heads (its products alone 2.8), so 7.1-7.7; steps of 64 x 300 31.8 -> 28.7 us, 64 x 1000 41.0 -> 39.5, 64 x 4096 83.7 -> 81.8.
constexpr int kAbsorbThreads = 288;
constexpr int kAbsorbQ = 32768, kAbsorbW = 32768, kAbsorbRows = 64;
// Unless `weights_ready` the launch is the head of a chain: it releases the next one, and reads W_UK, behind its wait.
__device__ __forceinline__ void absorb_block(uint8_t* sm_raw, const CUtensorMap* tmap_w, const CUtensorMap* tmap_q, const CUtensorMap* tmap_out,
                                             const AbsorbParams& prm, int bx, int by, int bz, bool chained, bool weights_ready) {
  __shared__ __align__(8) uint64_t landed[4], done[4], q_landed;
  __shared__ uint32_t tmem_slot;
  uint8_t* sm = (uint8_t*)(((uintptr_t)sm_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* As = sm;               // [2 halves of d][128 rows][64], swizzled
  uint8_t* Bs = sm + kAbsorbQ;    // [chunk][2 halves of d][128 c][64], swizzled; then [chunk][2 halves of c][kAbsorbRows rows][64]
  const int n_chunks = prm.n_chunks, H = prm.H, q_bf16 = prm.q_bf16;
  const int h = bx, c0 = by * 128 * n_chunks, r0 = bz * 64;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_here = min(64, prm.rows - r0);
  const uint32_t tmem_cols = n_chunks * 128;
  auto load_w = [&] {
    for (int i = 0; i < n_chunks; i++) {
      mbar_expect_tx(&landed[i], kAbsorbW);
      tma_load_2d(Bs + i * kAbsorbW, tmap_w, h * kDh, c0 + i * 128, &landed[i]);
      tma_load_2d(Bs + i * kAbsorbW + 16384, tmap_w, h * kDh + 64, c0 + i * 128, &landed[i]);
    }
  };
  // The release stands behind the allocation: a CTA of the up-projection, which allocates ahead of its wait, may share the SM, and must find this
  // one's columns taken.  Ahead of this launch's own wait it allocates only behind launches that use no tensor memory beside it.
  auto take_tmem = [&] {
    tmem_alloc<1>(&tmem_slot, tmem_cols);
    tmem_relinquish<1>();
  };
  if (warp == 8) {
    if (elect_one()) {
      tma_prefetch_desc(tmap_w);
      tma_prefetch_desc(tmap_q);
      mbar_init(&q_landed, 1);
      for (int i = 0; i < n_chunks; i++) {
        mbar_init(&landed[i], 1);
        mbar_init(&done[i], 1);
      }
      fence_mbar_init();
      if (weights_ready) load_w();
      tma_prefetch_desc(tmap_out);
    }
    if (weights_ready) {
      take_tmem();
      if (chained) chain_release();
    }
  }
  chain_wait();   // also: the kernel before this one may still be reading what this one overwrites
  if (warp == 8) {
    if (elect_one()) {
      if (q_bf16) {   // rows past the batch are zero-filled
        mbar_expect_tx(&q_landed, 32768);
        for (int r = 0; r < 128; r += kAbsorbRows) {
          tma_load_2d(As + r * 128, tmap_q, h * kDh, r0, &q_landed);
          tma_load_2d(As + 16384 + r * 128, tmap_q, h * kDh + 64, r0, &q_landed);
        }
      }
      if (!weights_ready) load_w();
    }
    if (!weights_ready) {
      take_tmem();
      if (chained) chain_release();
    }
    __syncwarp();
  }
  if (!q_bf16) {
#pragma unroll 2
    for (int e = threadIdx.x; e < rows_here * (kDh / 8); e += blockDim.x) {
      const int r = e / (kDh / 8), v = e % (kDh / 8);
      const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(prm.q_nope) + ((size_t)(r0 + r) * H + h) * kDh + (size_t)v * 8);
      const float4 x = load_chained(s), y = load_chained(s + 1);
      const uint4 w = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
      for (int k = r; k < 128; k += kAbsorbRows) *reinterpret_cast<uint4*>(As + (v >> 3) * 16384 + swz128(k, v & 7)) = w;
    }
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();   // the barriers, the tensor memory's address and the float32 rows are visible
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const int roww = prm.dC + prm.dHR;
  if (warp == 8) {
    const bool el = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
    const uint64_t dQ = make_desc_kmajor_sw128(smem_u32(As)), dW = make_desc_kmajor_sw128(smem_u32(Bs));
    if (q_bf16 && !mbar_wait(&q_landed, 0)) set_status(prm.status, RELUX_ERR_TIMEOUT);   // bounded: a load that never lands is reported
#pragma unroll 1
    for (int i = 0; i < n_chunks; i++) {
      if (!mbar_wait(&landed[i], 0)) set_status(prm.status, RELUX_ERR_TIMEOUT);
      __syncwarp();
      if (el) {
        const uint64_t w = dW + (uint32_t)(i * (kAbsorbW >> 4));
#pragma unroll
        for (int ks = 0; ks < 8; ks++)
          umma_ss<1>(tmem + i * 128, dQ + (((ks >> 2) * 16384 + (ks & 3) * 32) >> 4), w + (((ks >> 2) * 16384 + (ks & 3) * 32) >> 4), idesc, ks != 0);
        umma_commit<1>(&done[i]);
      }
      __syncwarp();
    }
  } else {
    if (by == 0) {   // the rope part of q~ is a copy (with the same rounding when the source is float32)
      const int vecs = prm.dHR / 8;
      for (int e = threadIdx.x; e < rows_here * vecs; e += 256) {
        const int r = e / vecs, v = e % vecs;
        const size_t off = ((size_t)(r0 + r) * H + h) * prm.dHR + (size_t)v * 8;
        uint4 w;
        if (q_bf16) w = load_chained(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(prm.q_rope) + off));
        else {
          const float4* s = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(prm.q_rope) + off);
          const float4 x = load_chained(s), y = load_chained(s + 1);
          w = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y), pack_bf16x2(y.z, y.w));
        }
        *reinterpret_cast<uint4*>(prm.q_abs + ((size_t)(r0 + r) * H + h) * roww + prm.dC + (size_t)v * 8) = w;
      }
    }
    const int group = warp >> 2, row = (warp & 1) * 32 + lane, first = (warp & 2) * 32;   // this warp's first column of a chunk
#pragma unroll 1
    for (int i = group; i < n_chunks; i += 2) {
      if (!mbar_wait(&done[i], 0)) set_status(prm.status, RELUX_ERR_TIMEOUT);
      tc_fence_after();
      uint8_t* Os = Bs + i * kAbsorbW;
#pragma unroll 1
      for (int c = first; c < first + 64; c += 32) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + i * 128 + c, v);
        tmem_ld_wait_for(v);
#pragma unroll
        for (int j = 0; j < 4; j++) {
          uint32_t w[4];
#pragma unroll
          for (int k = 0; k < 4; k++) w[k] = pack_bf16x2(__uint_as_float(v[8 * j + 2 * k]), __uint_as_float(v[8 * j + 2 * k + 1]));
          *reinterpret_cast<uint4*>(Os + (c >> 6) * 8192 + swz128(row, ((c & 63) >> 3) + j)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      fence_proxy_async();
      asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
      if ((threadIdx.x & 127) == 0) {   // rows past the batch lie outside the map
        tma_store_2d(tmap_out, h * roww + c0 + i * 128, r0, Os);
        tma_store_2d(tmap_out, h * roww + c0 + i * 128 + 64, r0, Os + 8192);
        tma_store_commit();
      }
    }
    if ((threadIdx.x & 127) == 0) tma_store_wait_all();
    if (chained) fence_chained_writes();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) tmem_dealloc<1>(tmem, tmem_cols);
}

// One block of either, a of the grid: head fastest, then the chunks of latent columns, then 64 rows each.
template <bool kTc>
__device__ __forceinline__ void absorb_any(uint8_t* sm_raw, const CUtensorMap* tmap_w, const CUtensorMap* tmap_q, const CUtensorMap* tmap_out,
                                           const AbsorbParams& prm, int a, bool chained, bool weights_ready) {
  const int slices = prm.dC / 128 / prm.n_chunks;
  if constexpr (kTc) absorb_block(sm_raw, tmap_w, tmap_q, tmap_out, prm, a % prm.H, a / prm.H % slices, a / prm.H / slices, chained, weights_ready);
  else absorb_block_mma(sm_raw, tmap_w, tmap_q, prm, a % prm.H, a / prm.H, chained, weights_ready);
}

// A plain launch.
template <bool kTc>
__global__ void __launch_bounds__(kTc ? kAbsorbThreads : kAbsorbMmaThreads) mla_absorb_mma_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                             const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_out,
                                                             const __grid_constant__ AbsorbParams prm) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  absorb_any<kTc>(smem_raw, &tmap_w, &tmap_q, &tmap_out, prm, blockIdx.x, false, true);
}

// The preparation of one MLA decode step in ONE launch: the first blocks append the step's new rows (a warp a sequence), the next one builds
// the stream partition (unless the decode kernel has it as arguments), and the blocks after them are the absorb grid (head fastest, then the
// chunks of latent columns, then 64 rows each).  The three jobs are independent of one another: the append reads the lengths
// before it writes, the partition counts every sequence's new rows itself, and the last of those blocks to finish advances
// the lengths (without a partition nobody else reads a sequence's length, and its warp advances it itself).  They come first because theirs is
// the longer chain of dependent reads.
// The kernel releases the launches after it only when everything before it is complete (the up-projection fetches its
// weights without a wait of its own), unless the launches before it in the call have seen to that (weights_ready): its own
// weights are then fetched ahead of its wait too.
template <bool kTc>
__global__ void __launch_bounds__(kTc ? kAbsorbThreads : kAbsorbMmaThreads) mla_prep_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_q,
                                                       const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ AbsorbParams prm,
                                                       int weights_ready, const __grid_constant__ PrepAppend ap, const __grid_constant__ PrepPlan pl) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  constexpr int kWarps = kTc ? 8 : 4;
  const int appends = (ap.n_seqs + kWarps - 1) / kWarps, chores = appends + (pl.listed ? 0 : 1), e = blockIdx.x;
  if (e >= chores) {
    absorb_any<kTc>(smem_raw, &tmap_w, &tmap_q, &tmap_out, prm, e - chores, true, weights_ready != 0);
    return;
  }
  if (weights_ready) chain_release();
  chain_wait();
  chain_release();
  if (e < appends) {
    const int i = e * kWarps + (threadIdx.x >> 5);
    if (threadIdx.x < 32 * kWarps && i < ap.n_seqs) prep_append_seq(ap, i, pl.listed != 0);
  } else {
    prep_build_stream<(kTc ? kAbsorbThreads : kAbsorbMmaThreads) / 32>(ap, pl);
  }
  if (!pl.listed) prep_arrive_and_advance(ap, (uint32_t)chores);
}

// Value up-projection of the split-KV partial results, and their sum.  For one head, with the pieces of a row (a sequence's query
// token) as columns,
//   D[128 output dims][column] = W_UV^T hi + W_UV^T lo      on tcgen05, W_UV's rows as the M = 128 operand as they lie (MN-major)
//   out[row] = sum over the row's columns of 2^(m - M) / L * D[:, column]
// part [piece][H][2 dC]: two bf16 halves of the unnormalised float32 partial (write_partial, mla_decode_generic_kernel), part_ml
// [piece][H][2] = (max in the log2 domain, sum); the pieces of row (i, q) are [first_i S + q n_i, + n_i), first_i = chunk_off[i], n_i =
// chunk_off[i + 1] - first_i, so that the columns of neighbouring rows are neighbours.
// What is summed is 128 float32 outputs a piece instead of 512 latent columns, behind the contraction instead of before it: nothing but TMA
// touches the partials (2 KB a piece and head), no row is rounded to bf16, and the row's weights are worked out meanwhile.  Adding the
// partials up first, by ordinary loads, took 15-16 k clocks of a launch at 64 rows of one piece (128 KB a CTA: every row a chain of round
// trips), rounded the sum to bf16 (the largest part of a latent step's error: 1.7e-3 of 2.4e-3), and multiplied by 3.2 k clocks of MMAs.
// From the wait to the last output, before -> now, three inputs in turn: 64 x 4096, a piece a row 12.4 -> 4.9 us; 16 x <= 32k, 90 pieces 8.0
// -> 7.2; 3 x <= 1500, 27 pieces 4.1 -> 3.5; one sequence 3.8 -> 2.4.  Bound: with many pieces what the partials take from L2 (35 bytes a clock
// and SM), else the round trips of a stage, of 32 MMAs (1.5 k clocks) and of the outputs.
// An MMA of up to 64 columns takes 40-48 clocks for its 4 KB of weights, so the halves of a block of columns stand side by side as N and the
// weights are read once for both: 32 MMAs a block.  Rows of one piece each come divided by their sum (their part_ml has 1) and rounded to bf16, without a lo.
// A launch finds its instructions in no cache, and what is executed once is waited for: clock stamps had 2 k clocks between the wait and the
// first MMA, 2.4 k for the first outputs, 4 k for the weights of three rows.  So the loops are rolled, and the warps that have nothing to do
// before the wait go through theirs once, on whatever memory holds, without storing.
// W_UV's slice of the head (dC x 128 bf16) is fetched by one thread as TMA boxes before chain_wait(): the weights do not depend on the
// decode kernel, and the launches before it have waited for everything older.
// grid (H, groups of rows), 512 threads: warp 0 loads, warp 1 issues the MMAs, the others work out the weights, all but those write the outputs.
constexpr int kVupWarps = 16;
constexpr int kVupListed = 256;                   // sequences whose first pieces travel as arguments
static_assert(kVupMaxCols >= kMaxRowItems, "a row's pieces are columns of one CTA");
static_assert(kListedItems <= kVupListed && kListedItems < 65536, "a listed plan is listed here too");
struct VupParams {
  const float* part_ml;
  const int32_t* chunk_off;
  void* out;
  int32_t rows, S, H, nk;
  int32_t rows_each;                          // rows of a group (the last may have fewer)
  int32_t halves, n_block, n_kb, n_stages;    // VupShape; a stage is one TMA box
  int32_t tmem_cols;
  int32_t n_blocks, room, all;                // blocks and columns that a CTA has room for, and columns that there are partial results for
  int32_t listed;                             // `first` holds chunk_off
  int32_t* status;
  uint16_t first[kVupListed + 1];
};
struct VupShared {
  uint64_t w_full[2], full[kVupMaxStages], empty[kVupMaxStages], done;
  uint32_t tmem_slot;
  float4 info[(kVupMaxCols + 16) / 2];        // of a column: first (max, sum), then its weight and, at a row's last, the row's place in `out` (else -1)
};
static_assert(131072 + kVupRing + sizeof(VupShared) <= 232448, "more shared memory than a CTA may use");

// Bounded, and out of line: around a loop of its own the issuing warp's operands leave their uniform registers.
__device__ __noinline__ void vup_wait_slow(uint64_t* bar, uint32_t parity, int32_t* status) {
  if (!mbar_wait(bar, parity)) set_status(status, RELUX_ERR_TIMEOUT);
}
__device__ __forceinline__ void vup_wait(uint64_t* bar, uint32_t parity, int32_t* status) {
  if (!mbar_try_wait(bar, parity)) vup_wait_slow(bar, parity, status);
  __syncwarp();
}

// kLoose (SplitPlan): the host has not counted the columns that the device's lengths make.
template <bool kOutBf16, bool kLoose>
__global__ void __launch_bounds__(32 * kVupWarps, 1) mla_vup_pieces_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                                          const __grid_constant__ CUtensorMap tmap_p,
                                                                          const __grid_constant__ VupParams prm) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int nk = prm.nk, H = prm.H, S = prm.S, nb = prm.n_block, blk_bytes = prm.halves * nb * 128, stage_bytes = prm.n_kb * blk_bytes;
  uint8_t* Ws = smem;                                             // [2 halves of 64 output dims][dC latent rows][64], swizzled
  uint8_t* ring = smem + nk * 32768;                              // [stage], swizzled
  VupShared* sh = reinterpret_cast<VupShared*>(ring + prm.n_stages * stage_bytes);
  float2* info = reinterpret_cast<float2*>(sh->info);
  const int h = blockIdx.x, r0 = blockIdx.y * prm.rows_each, rows_here = min(prm.rows_each, prm.rows - r0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int steps_each = (2 * nk + prm.n_kb - 1) / prm.n_kb;      // stages of a block of columns
  chain_release();
  if (threadIdx.x == 0) {
    if ((smem_u32(smem) & 1023u) != 0) set_status(prm.status, RELUX_ERR_UNSUPPORTED);   // the swizzled layouts
    mbar_init(&sh->w_full[0], 1);
    mbar_init(&sh->w_full[1], 1);
    for (int s = 0; s < prm.n_stages; s++) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    mbar_init(&sh->done, 1);
    fence_mbar_init();
    for (int k = 0; k < nk; k += 2) {   // 256 latent rows (128 where there are no more) in the order of a partial's columns
      mbar_expect_tx(&sh->w_full[k >> 1], nk == 1 ? 32768 : 65536);
      tma_load_5d(Ws + k * 16384, &tmap_w, h * kDh, 0, 0, 0, k * 4, &sh->w_full[k >> 1]);
      tma_load_5d(Ws + nk * 16384 + k * 16384, &tmap_w, h * kDh + 64, 0, 0, 0, k * 4, &sh->w_full[k >> 1]);
    }
    tma_prefetch_desc(&tmap_p);
  }
  if (warp == 1) {
    tmem_alloc<1>(&sh->tmem_slot, prm.tmem_cols);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();   // the barriers and the tensor memory's address are visible
  tc_fence_after();
  const uint32_t tmem = sh->tmem_slot;
  auto first_of = [&](int i) -> int { return prm.listed ? prm.first[i] : load_chained(prm.chunk_off + i); };
  auto col_of = [&](int row) -> int {   // first column of a row of the call
    const int i = S == 1 ? row : row / S, q = row - i * S, c0 = first_of(i);
    return c0 * S + (q == 0 ? 0 : q * (first_of(i + 1) - c0));
  };
  auto beyond = [&](int c0, int n) { return kLoose && (n > prm.room || c0 + n > prm.all); };   // columns that the launch was not sized for
  if (warp < 2) {
    const bool el = elect_one();
    chain_wait();   // the partial results come from the kernel before this one
    const int col0 = col_of(r0), cols = col_of(r0 + rows_here) - col0;
    int blocks = (cols + nb - 1) / nb;
    if (kLoose) blocks = min(blocks, prm.n_blocks);
    if (beyond(col0, cols) && threadIdx.x == 0) set_status(prm.status, RELUX_ERR_UNSUPPORTED);
    if (warp == 0) {
#pragma unroll 1
      for (int b = 0, s = 0, use = 0; b < blocks; b++)
#pragma unroll 1
        for (int st = 0; st < steps_each; st++) {
          if (use > 0) vup_wait(&sh->empty[s], (use - 1) & 1, prm.status);
          if (el) {
            mbar_expect_tx(&sh->full[s], stage_bytes);
            tma_load_5d(ring + s * stage_bytes, &tmap_p, 0, col0 + b * nb, 0, st * prm.n_kb, h, &sh->full[s]);
          }
          __syncwarp();
          if (++s == prm.n_stages) s = 0, use++;
        }
    } else {
      const uint32_t idesc = make_idesc_bf16(128, prm.halves * nb, true, false);
      const uint64_t dA = make_desc_kmajor_sw128(smem_u32(ring)), dW = make_desc_mnmajor_sw128(smem_u32(Ws), nk * 16384);
      vup_wait(&sh->w_full[0], 0, prm.status);
#pragma unroll 1
      for (int b = 0, s = 0, use = 0; b < blocks; b++)
#pragma unroll 1
        for (int st = 0, kb = 0; st < steps_each; st++) {
          if (kb + prm.n_kb > 4 && nk > 2) vup_wait(&sh->w_full[1], 0, prm.status);
          vup_wait(&sh->full[s], use & 1, prm.status);
          const uint64_t a0 = dA + ((uint32_t)(s * stage_bytes) >> 4);
#pragma unroll 1
          for (int k = 0; k < prm.n_kb && kb < 2 * nk; k++, kb++)
            if (el) {
              const uint64_t a = a0 + ((uint32_t)(k * blk_bytes) >> 4), w = dW + (uint32_t)(kb * 512);
              umma_ss<1>(tmem + b * prm.halves * nb, w, a, idesc, kb != 0);
              umma_ss<1>(tmem + b * prm.halves * nb, w + 128, a + 2, idesc, true);
              umma_ss<1>(tmem + b * prm.halves * nb, w + 256, a + 4, idesc, true);
              umma_ss<1>(tmem + b * prm.halves * nb, w + 384, a + 6, idesc, true);
            }
          if (el) umma_commit<1>(&sh->empty[s]);
          __syncwarp();
          if (++s == prm.n_stages) s = 0, use++;
        }
      if (kLoose && nk > 2) vup_wait(&sh->w_full[1], 0, prm.status);   // without a column nobody has, and no load may land when the CTA has gone
      if (el) umma_commit<1>(&sh->done);
      __syncwarp();
    }
  }
  // The others: weights, then outputs, four warps a lane quarter and a quarter of the rows each.
  // lane = output dim 32 (warp & 3) + lane, column = piece: every store of a warp is 32 neighbouring dims of a row
  const uint32_t tmem_d = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const size_t off0 = ((size_t)r0 * H + h) * kDh + (warp & 3) * 32 + lane;
#pragma unroll 1
  for (int pass = warp >= 2 ? 0 : 1; pass < 2; pass++) {
    const bool real = pass == 1;
    int col0 = 0, lo = 0, hi = 0;   // first column of the CTA, and columns of the warp's rows
    if (real) {
      if (warp >= 2) chain_wait();
      const int ra = rows_here * (warp >> 2) / 4, rb = rows_here * ((warp >> 2) + 1) / 4;
      col0 = col_of(r0);
      lo = col_of(r0 + ra) - col0;
      hi = col_of(r0 + rb) - col0;
      if (beyond(col0, hi)) lo = hi = 0;   // (not from `lo` on: a lane's eight columns would be beyond it too)
    }
    if (warp >= 2) {
      // the weights of a row's pieces, by 32, 8 or 4 lanes
      const int lpr = rows_here <= kVupWarps - 2 ? 32 : rows_here <= 4 * (kVupWarps - 2) ? 8 : 4;
      const int sub = lane & (lpr - 1), per_pass = (kVupWarps - 2) * (32 / lpr), rows_now = real ? rows_here : 1;
#pragma unroll 1
      for (int rw = 0; rw < rows_now; rw += per_pass) {
        const int r = rw + ((warp - 2) * 32 + lane) / lpr;
        int c = 0, n = 0;
        if (r < rows_now) {
          const int i = S == 1 ? r0 + r : (r0 + r) / S, q = r0 + r - i * S, first = first_of(i), pieces = first_of(i + 1) - first;
          n = real ? pieces : 1;
          c = real ? first * S + q * n - col0 : kVupMaxCols + 8;   // no column's place: other warps may be at theirs already
          if (real && beyond(col0, c + n)) n = 0;
        }
        float M = -INFINITY;
#pragma unroll 1
        for (int j = sub; j < n; j += lpr) {
          const float2 ml = load_chained(reinterpret_cast<const float2*>(prm.part_ml + ((size_t)((real ? col0 + c : 0) + j) * H + h) * 2));
          info[c + j] = ml;
          M = fmaxf(M, ml.x);
        }
#pragma unroll 1
        for (int o = 1; o < lpr; o <<= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
        float L = 0.f;
#pragma unroll 1
        for (int j = sub; j < n; j += lpr) {
          const float2 ml = info[c + j];
          if (ml.x != -INFINITY) L += ml.y * exp2f(ml.x - M);
        }
#pragma unroll 1
        for (int o = 1; o < lpr; o <<= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
        const float inv = (L > 0.f) ? 1.0f / L : 0.f;
#pragma unroll 1
        for (int j = sub; j < n; j += lpr) {
          const float m = info[c + j].x;
          info[c + j] = make_float2(m == -INFINITY ? 0.f : exp2f(m - M) * inv, __int_as_float(j == n - 1 ? r * H * kDh : -1));
        }
        if (r < rows_now && n <= 0)   // an empty sequence
          for (int d = sub; d < kDh; d += lpr) {
            const size_t off = ((size_t)(r0 + r) * H + h) * kDh + d;
            if (kOutBf16) reinterpret_cast<uint16_t*>(prm.out)[off] = 0;
            else reinterpret_cast<float*>(prm.out)[off] = 0.f;
          }
      }
    }
    if (real) {
      __syncthreads();   // the weights
      vup_wait(&sh->done, 0, prm.status);
      tc_fence_after();
    }
    float acc = 0.f;
#pragma unroll 1
    for (int c = lo & ~7; c < (real ? hi : 8); c += 8) {
      uint32_t v[8], w[8];   // the halves' products; a block's lie n_block apart
      const int b = c >= nb ? c / nb : 0, at = c + (prm.halves - 1) * b * nb;
      tmem_ld_32x32b_x8(tmem_d + at, v);
      tmem_ld_32x32b_x8(tmem_d + at + (prm.halves - 1) * nb, w);
      float4 f[4];
#pragma unroll
      for (int j = 0; j < 4; j++) f[j] = sh->info[c / 2 + j];
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float wt = (j & 1) ? f[j >> 1].z : f[j >> 1].x, second = prm.halves == 2 ? __uint_as_float(w[j]) : 0.f;
        const int r = __float_as_int((j & 1) ? f[j >> 1].w : f[j >> 1].y);
        const bool mine = c + j >= lo && c + j < hi, last = mine && r >= 0;
        const float x = fmaf(__uint_as_float(v[j]) + second, wt, acc);
        acc = mine && wt != 0.f ? x : acc;   // a piece without a visible key may hold anything
        if (kOutBf16) store_if(reinterpret_cast<uint16_t*>(prm.out) + off0 + r, (uint16_t)pack_bf16x2(acc, 0.f), last);
        else store_if(reinterpret_cast<float*>(prm.out) + off0 + r, acc, last);
        acc = last ? 0.f : acc;
      }
    }
  }
  tc_fence_before();
  if (kOutBf16) fence_chained_writes();   // a projection's operand
  __syncthreads();
  if (warp == 1) tmem_dealloc<1>(tmem, prm.tmem_cols);
}

}  // namespace

bool mla_proj_mma_eligible(int Dh, int dC) { return Dh == kDh && dC % 128 == 0; }

// W_UK [dC][H * 128] in 128 x 64 boxes; bf16 queries [rows][H * 128], and the result [rows][H * (dC + dHR)], in boxes of the kernel's rows.  On tcgen05 a
// CTA has as many chunks as leave the heads' CTAs one turn on the GPU.
struct AbsorbSetup {
  CUtensorMap w, q, out;
  AbsorbParams prm;
  bool tc;
  unsigned ctas;
  size_t smem;
};
static int32_t absorb_setup(Device* dev, const void* q_nope, const void* q_rope, int q_bf16, const uint16_t* W_UK, uint16_t* q_abs, int rows, int H, int dC,
                            int dHR, int32_t* status, AbsorbSetup* s) {
  s->tc = rows > kAbsorbMmaRows;
  const int n_tile = s->tc ? kAbsorbRows : kAbsorbMmaRows;
  if (!make_tmap_2d(&s->w, (void*)W_UK, (uint64_t)dC, (uint64_t)H * kDh, 64, 128) ||
      (s->tc && !make_tmap_2d(&s->out, q_abs, (uint64_t)rows, (uint64_t)H * (dC + dHR), 64, n_tile)) ||
      (q_bf16 && !make_tmap_2d(&s->q, (void*)q_nope, (uint64_t)rows, (uint64_t)H * kDh, 64, n_tile))) {
    set_error("tensor map for w_uk or the queries could not be encoded");
    return RELUX_ERR_CUDA;
  }
  if (!q_bf16) s->q = s->w;
  if (!s->tc) s->out = s->w;
  int n = 1;
  while (s->tc && n < 4 && dC / 128 % (2 * n) == 0 && H * (dC / 128 / n) > dev->sm_count) n *= 2;
  s->prm = AbsorbParams{q_nope, q_rope, q_abs, q_bf16, rows, H, dC, dHR, n, status};
  s->ctas = (unsigned)H * (unsigned)(dC / 128 / n) * (unsigned)((rows + 63) / 64);
  s->smem = s->tc ? (size_t)kAbsorbQ + (size_t)n * kAbsorbW + 1024 : kAbsorbMmaSmem;
  return RELUX_OK;
}
constexpr size_t kAbsorbSmemMost = kAbsorbQ + 4 * kAbsorbW + 1024;

int32_t launch_mla_absorb_mma(Device* dev, const void* q_nope, const void* q_rope, int q_bf16, const uint16_t* W_UK, uint16_t* q_abs,
                              int rows, int H, int dC, int dHR, int32_t* status) {
  AbsorbSetup s;
  if (int32_t rc = absorb_setup(dev, q_nope, q_rope, q_bf16, W_UK, q_abs, rows, H, dC, dHR, status, &s)) return rc;
  auto launch = [&](auto kern, int threads, size_t most) -> int32_t {
    if (int32_t rc = allow_smem(dev, kern, most)) return rc;
    kern<<<s.ctas, threads, s.smem, dev->stream>>>(s.w, s.q, s.out, s.prm);
    RELUX_CUDA_TRY(cudaGetLastError());
    count_launch(dev);
    return RELUX_OK;
  };
  return s.tc ? launch(mla_absorb_mma_kernel<true>, kAbsorbThreads, kAbsorbSmemMost) : launch(mla_absorb_mma_kernel<false>, kAbsorbMmaThreads, kAbsorbMmaSmem);
}

// One launch: absorb + append of the step's rows + stream partition (see mla_prep_kernel).
int32_t launch_mla_prep(Device* dev, const void* q_nope, const void* q_rope, int q_bf16, const uint16_t* W_UK, uint16_t* q_abs, int rows,
                        int H, int dC, int dHR, bool weights_ready, const PrepAppend& ap, const PrepPlan& pl, bool chained) {
  AbsorbSetup s;
  if (int32_t rc = absorb_setup(dev, q_nope, q_rope, q_bf16, W_UK, q_abs, rows, H, dC, dHR, ap.status, &s)) return rc;
  auto launch = [&](auto kern, int threads, size_t most) -> int32_t {
    if (int32_t rc = allow_smem(dev, kern, most)) return rc;
    const int warps = threads / 64 * 2;   // that append, of a block: 4 of 4, 8 of 9
    const unsigned blocks = (unsigned)(ap.n_seqs + warps - 1) / (unsigned)warps + (pl.listed ? 0u : 1u) + s.ctas;
    RELUX_CUDA_TRY(launch_chained(chained, kern, dim3(blocks), dim3(threads), s.smem, dev->stream, s.w, s.q, s.out, s.prm, weights_ready ? 1 : 0, ap, pl));
    count_launch(dev);
    return RELUX_OK;
  };
  return s.tc ? launch(mla_prep_kernel<true>, kAbsorbThreads, kAbsorbSmemMost) : launch(mla_prep_kernel<false>, kAbsorbMmaThreads, kAbsorbMmaSmem);
}

int32_t launch_mla_vup_pieces(Device* dev, const void* part, const float* part_ml, const SplitPlan& plan, const VupShape& sh, int form, bool natural,
                              const uint16_t* W_UV, void* out, int out_bf16, int rows, int S, int H, int dC, int32_t* status, bool chained) {
  // columns that there are partial results for
  const int all = (plan.loose ? std::max(plan.num_items, plan.room_items) : plan.num_items) * S;
  const int n_seqs = rows / S;
  VupParams k;
  k.rows_each = sh.rows_each;
  k.listed = !plan.loose && n_seqs <= kVupListed && plan.num_items < 65536;   // wherever the plan is (list_plan): chunk_off then does not exist
  if (k.listed)
    for (int i = 0; i <= n_seqs; i++) k.first[i] = (uint16_t)plan.first[i];
  k.halves = form == kPartialHalves ? 2 : 1;
  k.n_block = sh.n_block;
  k.n_kb = sh.n_kb;
  k.n_stages = sh.n_stages;
  k.tmem_cols = sh.tmem_cols;
  k.n_blocks = sh.blocks;
  k.room = std::min(sh.blocks * sh.n_block, kVupMaxCols);
  k.all = all;
  const int blk_bytes = k.halves * k.n_block * 128;
  k.part_ml = part_ml;
  k.chunk_off = plan.chunk_off;
  k.out = out;
  k.rows = rows;
  k.S = S;
  k.H = H;
  k.nk = dC / 128;
  k.status = status;
  // W_UV [dC][H * 128]: latent row 32 b + 8 i + 2 q + e at place 32 b + 8 q + 2 i + e (write_partial), or as it is
  const uint64_t ld = (uint64_t)H * kDh, di = natural ? 2 : 8, dq = natural ? 8 : 2, lp = (uint64_t)k.halves * dC;
  const uint64_t w_dims[5] = {ld, 2, 4, 4, (uint64_t)dC / 32}, w_strides[4] = {ld, di * ld, dq * ld, 32 * ld};
  const uint32_t w_box[5] = {64, 2, 4, 4, dC == 128 ? 4u : 8u};
  const uint64_t p_dims[5] = {64, (uint64_t)all, (uint64_t)k.halves, (uint64_t)dC / 64, (uint64_t)H}, p_strides[4] = {H * lp, (uint64_t)dC, 64, lp};
  const uint32_t p_box[5] = {64, (uint32_t)k.n_block, (uint32_t)k.halves, (uint32_t)k.n_kb, 1};
  CUtensorMap tw, tp;
  if (!make_tmap_view(&tw, (void*)W_UV, 5, w_dims, w_strides, w_box) || !make_tmap_view(&tp, (void*)part, 5, p_dims, p_strides, p_box)) {
    set_error("tensor map for w_uv or the partial results could not be encoded");
    return RELUX_ERR_CUDA;
  }
  const size_t smem = (size_t)k.nk * 32768 + (size_t)k.n_stages * k.n_kb * blk_bytes + sizeof(VupShared);
  auto launch = [&](auto kern) -> int32_t {
    if (int32_t rc = allow_smem(dev, kern, smem)) return rc;
    RELUX_CUDA_TRY(launch_chained(chained, kern, dim3(H, sh.groups), dim3(32 * kVupWarps), smem, dev->stream, tw, tp, k));
    count_launch(dev);
    return RELUX_OK;
  };
  if (plan.loose) return out_bf16 ? launch(mla_vup_pieces_kernel<true, true>) : launch(mla_vup_pieces_kernel<false, true>);
  return out_bf16 ? launch(mla_vup_pieces_kernel<true, false>) : launch(mla_vup_pieces_kernel<false, false>);
}

}  // namespace relux
