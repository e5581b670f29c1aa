// Per-warp attention over one 64-token page of a kv head, shared by the GQA decode kernels (gqa_stream.cu: decode and
// verify steps; gqa_decode.cu: prompts as grid slices, and the allocation-free entry point).
//
// The g query heads of a kv head times the S query tokens are the M rows (16 * MT) of mma.sync m16n8k16, bf16 in, float32
// accumulate.  A page is four 8 KB TMA boxes (K dims 0-63, K dims 64-127, V likewise; 128-byte swizzle); each of four
// consumer warps owns 16 of its tokens and a private online-softmax state, so the warps never wait on each other inside
// a piece of work and meet only at its end (gqa_store_state).
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace relux {

constexpr int kGqaPageTok = 64;
constexpr int kGqaD = 128;
constexpr int kGqaStageBytes = 4 * 8192;       // K lo, K hi, V lo, V hi
constexpr int kGqaQStride = kGqaD + 8;         // bf16 elements per Q row in shared memory (272 B, conflict-free ldmatrix)
constexpr int kGqaConsumerWarps = 4;
constexpr int kGqaStateStride = kGqaD + 4;     // float32 per row of a warp's state in shared memory: O, max, sum, padding to 16 bytes

__device__ __forceinline__ float gqa_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int MT>
struct GqaState {
  float o[MT][16][4];
  float m[MT][2], l[MT][2];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
#pragma unroll
      for (int nt = 0; nt < 16; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) o[mt][nt][e] = 0.f;
      m[mt][0] = m[mt][1] = -INFINITY;
      l[mt][0] = l[mt][1] = 0.f;
    }
  }
};

// Q rows [16 * MT][kGqaQStride] in shared memory -> A fragments.
template <int MT>
__device__ __forceinline__ void gqa_load_q(uint32_t (&qa)[MT][8][4], const uint16_t* qs, int lane) {
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int ks = 0; ks < 8; ks++) {
      const int m = lane >> 3;
      const int row = mt * 16 + (m & 1) * 8 + (lane & 7);
      const int col = ks * 16 + (m >> 1) * 8;
      ldmatrix_x4(qa[mt][ks][0], qa[mt][ks][1], qa[mt][ks][2], qa[mt][ks][3], smem_u32(qs + row * kGqaQStride + col));
    }
}

// Adds this warp's 16 tokens (tb .. tb + 15 of the page, logical tokens tok0 ..) to its state.  T: visible tokens; row r
// (counted from row0 of the fragment) belongs to query token r / g of S, which with the causal mask sees tokens up to T - S + r / g.
template <int MT>
__device__ __forceinline__ void gqa_consume_page(GqaState<MT>& st, const uint32_t (&qa)[MT][8][4], uint32_t kt, int tb, int tok0, int T, int S,
                                                 int g, int causal, float scale_log2, int lane, int row0 = 0) {
  const uint32_t vt = kt + 16384;
  // two accumulators per 8-token column block (even and odd K slices): the MMAs of one block depend on each other, and
  // the chain's latency, not the issue rate, is what a page costs a warp
  float sacc[MT][2][4], sodd[MT][2][4];
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) sacc[mt][nt][e] = sodd[mt][nt][e] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 8; ks++) {
    const int m = lane >> 3;
    const uint32_t row = tb + (m >> 1) * 8 + (lane & 7);
    const uint32_t chunk = (ks & 3) * 2 + (m & 1);
    uint32_t b0, b1, b2, b3;
    ldmatrix_x4(b0, b1, b2, b3, kt + (ks >> 2) * 8192 + swz128(row, chunk));
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
      mma_bf16_16816(ks & 1 ? sodd[mt][0] : sacc[mt][0], qa[mt][ks], b0, b1);
      mma_bf16_16816(ks & 1 ? sodd[mt][1] : sacc[mt][1], qa[mt][ks], b2, b3);
    }
  }
  // mask the tail of the sequence and the causal part of the draft
  const bool need_mask = (tok0 + 16 > T - (causal ? S : 0));
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) sacc[mt][nt][e] += sodd[mt][nt][e];
  if (need_mask) {
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int hf = 0; hf < 2; hf++) {
        const int row = row0 + mt * 16 + hf * 8 + (lane >> 2);
        const int limit = causal ? (T - S + row / g) : (T - 1);  // last visible token
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int tok = tok0 + nt * 8 + 2 * (lane & 3) + e;
            if (tok > limit || tok >= T) sacc[mt][nt][hf * 2 + e] = -INFINITY;
          }
      }
  }
  // Running max in the log2 domain; the rescale of sums and outputs is left out on a page where no row of the warp passes
  // its max.  (Not a lazy max with slack: a row's largest probability stays 1, which bf16 holds exactly.)
  float mx[MT][2];
  bool grow = false;
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
      float v = fmaxf(fmaxf(sacc[mt][0][hf * 2], sacc[mt][0][hf * 2 + 1]), fmaxf(sacc[mt][1][hf * 2], sacc[mt][1][hf * 2 + 1]));
      v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
      v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
      mx[mt][hf] = v * scale_log2;
      grow |= mx[mt][hf] > st.m[mt][hf];
    }
  if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int hf = 0; hf < 2; hf++) {
        const float m_new = fmaxf(st.m[mt][hf], mx[mt][hf]);
        const float alpha = (m_new == -INFINITY) ? 0.f : gqa_ex2(st.m[mt][hf] - m_new);
        st.m[mt][hf] = m_new;
        st.l[mt][hf] *= alpha;
#pragma unroll
        for (int nt = 0; nt < 16; nt++) {
          st.o[mt][nt][hf * 2] *= alpha;
          st.o[mt][nt][hf * 2 + 1] *= alpha;
        }
      }
  }
  uint32_t pa[MT][4];
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
      const float neg_m = (st.m[mt][hf] == -INFINITY) ? 0.f : -st.m[mt][hf];
      float ps = 0.f;
#pragma unroll
      for (int nt = 0; nt < 2; nt++) {
        const float p0 = gqa_ex2(fmaf(sacc[mt][nt][hf * 2], scale_log2, neg_m));
        const float p1 = gqa_ex2(fmaf(sacc[mt][nt][hf * 2 + 1], scale_log2, neg_m));
        ps += p0 + p1;
        __nv_bfloat162 b2 = __floats2bfloat162_rn(p0, p1);
        pa[mt][nt * 2 + hf] = *reinterpret_cast<uint32_t*>(&b2);
      }
      st.l[mt][hf] += ps;
    }
  // O += P V
#pragma unroll
  for (int n2 = 0; n2 < 8; n2++) {
    const int m = lane >> 3;
    const uint32_t row = tb + (m & 1) * 8 + (lane & 7);
    const uint32_t chunk = n2 * 2 + (m >> 1);  // 16 chunks of 8 dims
    uint32_t b0, b1, b2, b3;
    ldmatrix_x4_trans(b0, b1, b2, b3, vt + (chunk >> 3) * 8192 + swz128(row, chunk & 7));
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
      mma_bf16_16816(st.o[mt][2 * n2], pa[mt], b0, b1);
      mma_bf16_16816(st.o[mt][2 * n2 + 1], pa[mt], b2, b3);
    }
  }
}

// A warp's state -> its first `rows` rows of kGqaStateStride float32 in shared memory; a warp whose wait ran out
// (alive = false) leaves a neutral state.
template <int MT>
__device__ __forceinline__ void gqa_store_state(const GqaState<MT>& st, float* dst0, int rows, int lane, bool alive) {
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
      float l = st.l[mt][hf];
      l += __shfl_xor_sync(0xffffffffu, l, 1);
      l += __shfl_xor_sync(0xffffffffu, l, 2);
      const int row = mt * 16 + hf * 8 + (lane >> 2);
      if (row >= rows) continue;
      float* dst = dst0 + row * kGqaStateStride;
#pragma unroll
      for (int nt = 0; nt < 16; nt++)
        *reinterpret_cast<float2*>(dst + nt * 8 + 2 * (lane & 3)) = make_float2(st.o[mt][nt][hf * 2], st.o[mt][nt][hf * 2 + 1]);
      if ((lane & 3) == 0) {
        dst[kGqaD] = alive ? st.m[mt][hf] : -INFINITY;
        dst[kGqaD + 1] = alive ? l : 0.f;
      }
    }
}

}  // namespace relux
