// Token selection after a speculative verify pass, on the device: SpeculativeDecoder.acceptPhase and
// resampleRejected (speculative.go:211-295, softmaxAlloc :346-368) and Sampler.Sample without the repetition
// penalties (internal/transformer/sampler.go:73-218).  The uniform draws the reference takes from math/rand are
// arguments, consumed in the reference's order.
//
// FAST: one thread-block cluster per sequence.  The CTAs of a cluster split the vocabulary into contiguous slices;
// every step of the reference's chain (row maximum, sum of exponentials, the top-k threshold, the nucleus cut, the
// inverse-CDF search) is one pass over the row out of L2 with a reduction across the cluster through distributed shared
// memory, so a row is read from HBM once however many passes follow.  Exponentials use the reference's fastexp32 bit
// trick, which makes the distribution the reference's own; what differs is the order of the float32 sums (parallel
// instead of sequential), so a decision can only differ when a draw falls within rounding distance of a boundary.
// REFERENCE: one thread per sequence walks the reference's loops in the reference's order (bit-exact, slow).
#include <cuda_runtime.h>
#include <algorithm>
#include <cooperative_groups.h>
#include <cstdint>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace cg = cooperative_groups;

namespace relux {

int32_t stage_in(Pool* p, GrowBuf& buf, const void* src, size_t bytes, int mem, const void** dptr);   // runtime.cu

namespace {

constexpr int kSelThreads = 512;
constexpr int kSelWarps = kSelThreads / 32;
constexpr int kMaxCluster = 8;
constexpr int kAhead = 32;
constexpr int kStatMax = 32;     // batched statistics: two sums and two maxima for each of up to 8 draft positions

struct SelParams {
  const int32_t* draft_tokens;   // [n][k] or nullptr (plain sampling)
  const float* draft_logits;     // [n][k][V]
  const float* target_logits;    // [n][k+1][V]; plain sampling: [n][V] with k = 0
  const float* draws;            // [n][k+1]
  int32_t* n_accepted;           // [n]
  int32_t* next_token;           // [n]
  int32_t* status;
  int32_t k, vocab;
  float temperature;
  int32_t top_k;
  float top_p, min_p;
  int32_t batched;               // accept loop: the rows of all positions in one stage
  TimeStamp time;
};

// Shared memory of one CTA: exchange slots read by the other CTAs of the cluster.
struct SelShared {
  float red[2][4];            // double-buffered per-CTA partials of a cluster reduction (up to 4 values)
  float warp_part[kSelWarps][4];
  float hist_sum[256];
  uint32_t hist_cnt[256];
  float warp_seg[kSelWarps];  // per-warp segment sums of the search pass
  alignas(16) uint32_t warp_hist[kSelWarps][256];   // radix selection: one histogram per warp (counts, or float sums)
  uint32_t list_count, list_bound;      // candidate list of the small-top-k path (the list itself reuses warp_hist), and its bound
  alignas(16) uint32_t grp_key[kSelThreads];        // keys of the largest element of every thread (or pair of threads)
  float red_n[2][kStatMax];   // cluster_reduce_n: per-CTA partials, double-buffered like red
  float warp_part_n[kSelWarps][kStatMax];
  int32_t tok[kAhead];        // what the accept loop needs of the first positions, fetched at once: draft tokens, their logits in
  float guess[2][kAhead];     // the draft and the target row, and the draws
  float draw[kAhead + 1];
  float stat[kStatMax];       // batched statistics: of draft position i the sums (draft, target) at 4 i, the maxima at 4 i + 2
};

// Keys that order like the values, by their bits alone (-0 below 0) ...
__device__ __forceinline__ uint32_t bit_key(float x) {
  uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// ... and with both zeros equal, as the reference's comparisons have them: what is counted for a threshold.  A threshold at 0 then lets
// the keys by bits of both pass, so that the passes compare these (an addition per element cost 1 % of a nucleus call).
__device__ __forceinline__ uint32_t order_key(float x) { return bit_key(__fadd_rn(x, 0.0f)); }
__device__ __forceinline__ uint32_t with_both_zeros(uint32_t threshold) { return threshold == 0x80000000u ? 0x7fffffffu : threshold; }

// fastexp32 without its upper cut: good up to 88, past which the bits are those of no finite number.  Arguments are differences to a
// row's maximum, or to a guess of it; a sum against a guess is used only where that lies less than 80 below.
__device__ __forceinline__ float fastexp32_below(float x) {
  const float t = __fadd_rn(__fmul_rn(12102203.0f, x), 1064948224.0f);
  return x < -87.0f ? 0.0f : __uint_as_float((uint32_t)__float2int_rz(t));
}

// Everything the passes need to evaluate the reference's probability of one logit on the fly.
struct Dist {
  float temp;        // 1 = untouched
  uint32_t topk_key; // elements whose key is below are masked (0 = nothing masked)
  float m, inv1;     // maximum and 1 / sum of exponentials
  float tau, inv2;   // nucleus: probabilities below tau are dropped, the rest scaled by inv2
  float minp_thr, inv3;
  __device__ __forceinline__ float scaled(float v) const { return temp == 1.0f ? v : __fdiv_rn(v, temp); }
  __device__ __forceinline__ float p1(float v) const {
    float x = scaled(v);
    if (bit_key(x) < topk_key) return 0.0f;
    return __fmul_rn(fastexp32_ref(__fsub_rn(x, m)), inv1);
  }
};

struct Ctx {
  SelShared* sh;
  int rank, csize;     // CTA rank in the cluster, cluster size
  int lo, hi;          // this CTA's slice of the vocabulary
  int wlo, whi;        // this warp's contiguous segment of the slice
  int warp, lane;
  bool vec;            // rows can be read as aligned float4s
  uint32_t round;      // reduction counter (selects the exchange buffer)
};

// Sum or maximum of up to four per-thread values over the whole cluster; every thread of every CTA gets the same result,
// combined in CTA order.  kMode 0: four sums; 1: four maxima; 2: values 0-1 summed, values 2-3 maximised (one barrier
// for the sums of one row pair and the maxima of the next).  One cluster barrier per call: the two exchange buffers
// alternate.
template <int kMode>
__device__ void cluster_reduce4(Ctx& c, float (&v)[4]) {
  cg::cluster_group cl = cg::this_cluster();
  auto is_max = [](int j) { return kMode == 1 || (kMode == 2 && j >= 2); };
#pragma unroll
  for (int j = 0; j < 4; j++) v[j] = is_max(j) ? warp_max(v[j]) : warp_sum(v[j]);
  if (c.lane == 0) {
#pragma unroll
    for (int j = 0; j < 4; j++) c.sh->warp_part[c.warp][j] = v[j];
  }
  __syncthreads();
  const int buf = c.round & 1;
  if (threadIdx.x < 4) {
    const bool mx = is_max((int)threadIdx.x);
    float a = c.sh->warp_part[0][threadIdx.x];
    for (int w = 1; w < kSelWarps; w++) a = mx ? fmaxf(a, c.sh->warp_part[w][threadIdx.x]) : a + c.sh->warp_part[w][threadIdx.x];
    c.sh->red[buf][threadIdx.x] = a;
  }
  cl.sync();
#pragma unroll
  for (int j = 0; j < 4; j++) {
    float a = is_max(j) ? -INFINITY : 0.0f;
    for (int r = 0; r < c.csize; r++) {
      const float* remote = cl.map_shared_rank(&c.sh->red[buf][j], r);
      a = is_max(j) ? fmaxf(a, *remote) : a + *remote;
    }
    v[j] = a;
  }
  c.round++;
}

// The same for `count` <= kStatMax values per thread (acc[]), sums where bit 1 of the index is clear and maxima where it is
// set; the results land in dst[] in this CTA's shared memory.
__device__ void cluster_reduce_n(Ctx& c, const float* acc, int count, float* dst) {
  cg::cluster_group cl = cg::this_cluster();
  for (int j = 0; j < count; j++) {
    const float r = (j & 2) ? warp_max(acc[j]) : warp_sum(acc[j]);
    if (c.lane == 0) c.sh->warp_part_n[c.warp][j] = r;
  }
  __syncthreads();
  const int buf = c.round & 1;
  const bool mx = threadIdx.x & 2;
  if ((int)threadIdx.x < count) {
    float a = c.sh->warp_part_n[0][threadIdx.x];
    for (int w = 1; w < kSelWarps; w++) a = mx ? fmaxf(a, c.sh->warp_part_n[w][threadIdx.x]) : a + c.sh->warp_part_n[w][threadIdx.x];
    c.sh->red_n[buf][threadIdx.x] = a;
  }
  cl.sync();
  if ((int)threadIdx.x < count) {
    float a = mx ? -INFINITY : 0.0f;
    for (int r = 0; r < c.csize; r++) {
      const float x = *cl.map_shared_rank(&c.sh->red_n[buf][threadIdx.x], r);
      a = mx ? fmaxf(a, x) : a + x;
    }
    dst[threadIdx.x] = a;
  }
  __syncthreads();
  c.round++;
}

// Every CTA learns every CTA's value (in rank order), through the same exchange buffers as cluster_reduce4.
__device__ void cluster_gather1(Ctx& c, float mine, float (&all)[kMaxCluster]) {
  cg::cluster_group cl = cg::this_cluster();
  const int buf = c.round & 1;
  if (threadIdx.x == 0) c.sh->red[buf][0] = mine;
  cl.sync();
#pragma unroll
  for (int r = 0; r < kMaxCluster; r++) all[r] = r < c.csize ? *cl.map_shared_rank(&c.sh->red[buf][0], r) : 0.0f;
  c.round++;
}

// Calls f(index, value) for every element of this warp's segment of `row`.  Segments start on multiples of 128
// elements, so when the vocabulary is a multiple of four and the rows are 16-byte aligned (c.vec) every lane reads
// float4s, four in flight; otherwise lanes interleave single floats.
template <class F>
__device__ __forceinline__ void for_segment(const Ctx& c, const float* __restrict__ row, F f) {
  if (c.vec) {
    int i = c.wlo + c.lane * 4;
    for (; i + 896 < c.whi; i += 1024) {   // eight float4 loads in flight per lane
      float4 t[8];
#pragma unroll
      for (int q = 0; q < 8; q++) t[q] = __ldg(reinterpret_cast<const float4*>(row + i + 128 * q));
#pragma unroll
      for (int q = 0; q < 8; q++) { f(i + 128 * q, t[q].x); f(i + 128 * q + 1, t[q].y); f(i + 128 * q + 2, t[q].z); f(i + 128 * q + 3, t[q].w); }
    }
    for (; i + 384 < c.whi; i += 512) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(row + i));
      const float4 b = __ldg(reinterpret_cast<const float4*>(row + i + 128));
      const float4 d = __ldg(reinterpret_cast<const float4*>(row + i + 256));
      const float4 e = __ldg(reinterpret_cast<const float4*>(row + i + 384));
      f(i, a.x); f(i + 1, a.y); f(i + 2, a.z); f(i + 3, a.w);
      f(i + 128, b.x); f(i + 129, b.y); f(i + 130, b.z); f(i + 131, b.w);
      f(i + 256, d.x); f(i + 257, d.y); f(i + 258, d.z); f(i + 259, d.w);
      f(i + 384, e.x); f(i + 385, e.y); f(i + 386, e.z); f(i + 387, e.w);
    }
    for (; i < c.whi; i += 128) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(row + i));
      f(i, a.x); f(i + 1, a.y); f(i + 2, a.z); f(i + 3, a.w);
    }
    return;
  }
  int i = c.wlo + c.lane;
  for (; i + 96 < c.whi; i += 128) {
    float a = __ldg(row + i), b = __ldg(row + i + 32), d = __ldg(row + i + 64), e = __ldg(row + i + 96);
    f(i, a); f(i + 32, b); f(i + 64, d); f(i + 96, e);
  }
  for (; i < c.whi; i += 32) f(i, __ldg(row + i));
}

// The same over two rows at once: f(index, value_a, value_b).
template <class F>
__device__ __forceinline__ void for_segment2(const Ctx& c, const float* __restrict__ ra, const float* __restrict__ rb, F f) {
  if (c.vec) {
    int i = c.wlo + c.lane * 4;
    for (; i + 384 < c.whi; i += 512) {   // four float4 loads per row in flight per lane
      float4 ta[4], tb[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        ta[q] = __ldg(reinterpret_cast<const float4*>(ra + i + 128 * q));
        tb[q] = __ldg(reinterpret_cast<const float4*>(rb + i + 128 * q));
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        f(i + 128 * q, ta[q].x, tb[q].x); f(i + 128 * q + 1, ta[q].y, tb[q].y);
        f(i + 128 * q + 2, ta[q].z, tb[q].z); f(i + 128 * q + 3, ta[q].w, tb[q].w);
      }
    }
    for (; i < c.whi; i += 128) {
      const float4 a0 = __ldg(reinterpret_cast<const float4*>(ra + i)), b0 = __ldg(reinterpret_cast<const float4*>(rb + i));
      f(i, a0.x, b0.x); f(i + 1, a0.y, b0.y); f(i + 2, a0.z, b0.z); f(i + 3, a0.w, b0.w);
    }
    return;
  }
  int i = c.wlo + c.lane;
  for (; i + 32 < c.whi; i += 64) {
    float a0 = __ldg(ra + i), b0 = __ldg(rb + i), a1 = __ldg(ra + i + 32), b1 = __ldg(rb + i + 32);
    f(i, a0, b0); f(i + 32, a1, b1);
  }
  for (; i < c.whi; i += 32) f(i, __ldg(ra + i), __ldg(rb + i));
}

// Radix selection, eight bits a round, over keys that order like the values.  kWeighted = false: the key of the
// `want`-th largest element (Sampler's kthLargest, sampler.go:283-300).  kWeighted = true: keys are probabilities and
// the walk stops at the largest probability tau for which the sum of all probabilities >= tau reaches `want_sum` (the
// nucleus cut of sampler.go:148-160; elements tied with tau are all kept).  Returns false when the total never
// reaches want_sum.
// stop_at (counting walk only): as soon as no more than stop_at elements have a key >= the lower bound of the chosen
// bin, the walk ends early; *key_out is then that lower bound and *n_ge_out the number of elements at or above it (a
// superset of the `want` largest that is small enough to finish on a list).
template <bool kWeighted, class KeyF>
__device__ bool radix_select(Ctx& c, const float* __restrict__ row, KeyF key_weight, uint32_t want, float want_sum, uint32_t* key_out,
                             uint32_t stop_at = 0, uint32_t* n_ge_out = nullptr) {
  const uint32_t want0 = want;
  cg::cluster_group cl = cg::this_cluster();
  uint32_t prefix = 0, mask = 0;
  float above = 0.0f;
  __shared__ uint32_t comb_cnt[256];
  __shared__ float comb_sum[256];
  __shared__ uint32_t pick[3];
  __shared__ float pick_above;
  for (int shift = 24; shift >= 0; shift -= 8) {
    // every warp fills a histogram of its own (no contention between warps); they are added up afterwards
    for (int t = threadIdx.x; t < kSelWarps * 256; t += kSelThreads) (&c.sh->warp_hist[0][0])[t] = 0u;
    __syncthreads();
    uint32_t* my_cnt = c.sh->warp_hist[c.warp];
    float* my_sum = reinterpret_cast<float*>(c.sh->warp_hist[c.warp]);
    // Most keys share their leading bits (the exponent of neighbouring logits or probabilities), so plain atomics
    // would pile onto two or three bins.  Every lane therefore keeps the bin it hit last in a register and only
    // touches shared memory when the bin changes.
    {
      uint32_t cur = 0xffffffffu, cur_n = 0;
      float cur_w = 0.0f;
      for_segment(c, row, [&](int, float v) {
        uint32_t key; float w;
        key_weight(v, key, w);
        if ((key & mask) != prefix) return;
        const uint32_t d = (key >> shift) & 255u;
        if (d != cur) {
          if (cur != 0xffffffffu) {
            if (kWeighted) atomicAdd(&my_sum[cur], cur_w);
            else atomicAdd(&my_cnt[cur], cur_n);
          }
          cur = d; cur_n = 0; cur_w = 0.0f;
        }
        cur_n++;
        cur_w += w;
      });
      if (cur != 0xffffffffu) {
        if (kWeighted) atomicAdd(&my_sum[cur], cur_w);
        else atomicAdd(&my_cnt[cur], cur_n);
      }
    }
    __syncthreads();
    if (threadIdx.x < 256) {
      uint32_t n = 0; float sacc = 0.0f;
      for (int wq = 0; wq < kSelWarps; wq++) {
        if (kWeighted) sacc += reinterpret_cast<const float*>(c.sh->warp_hist[wq])[threadIdx.x];
        else n += c.sh->warp_hist[wq][threadIdx.x];
      }
      c.sh->hist_cnt[threadIdx.x] = n; c.sh->hist_sum[threadIdx.x] = sacc;
    }
    cl.sync();
    if (threadIdx.x < 256) {
      uint32_t n = 0; float s = 0.0f;
      for (int r = 0; r < c.csize; r++) {
        if (kWeighted) s += *cl.map_shared_rank(&c.sh->hist_sum[threadIdx.x], r);
        else n += *cl.map_shared_rank(&c.sh->hist_cnt[threadIdx.x], r);
      }
      comb_cnt[threadIdx.x] = n; comb_sum[threadIdx.x] = s;
    }
    __syncthreads();
    // Walk the bins from the top until the running count (or sum) reaches the target: warp 0, eight bins a lane.
    if (threadIdx.x == 0) { pick[0] = 256; pick_above = above; }
    __syncthreads();
    if (c.warp == 0) {
      const int b_hi = 8 * c.lane + 7;
      if (kWeighted) {
        float mine = 0.0f;
        for (int q = 0; q < 8; q++) mine += comb_sum[b_hi - q];
        float upper = mine;      // inclusive sum over this lane and the lanes above it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          float y = __shfl_down_sync(0xffffffffu, upper, o);
          if (c.lane + o < 32) upper += y;
        }
        const float higher = __shfl_down_sync(0xffffffffu, upper, 1);   // sum over the lanes above this one
        float acc = above + (c.lane < 31 ? higher : 0.0f);
        int hit = -1;
        float acc_hit = acc;
        for (int q = 0; q < 8 && hit < 0; q++) {
          float nxt = acc + comb_sum[b_hi - q];
          if (nxt >= want_sum) { hit = b_hi - q; acc_hit = acc; }
          acc = nxt;
        }
        const uint32_t any = __ballot_sync(0xffffffffu, hit >= 0);
        if (any && c.lane == 31 - __clz(any)) { pick[0] = (uint32_t)hit; pick_above = acc_hit; }
        if (!any && c.lane == 0) pick_above = acc;   // the whole row stays below the target
      } else {
        uint32_t mine = 0;
        for (int q = 0; q < 8; q++) mine += comb_cnt[b_hi - q];
        uint32_t upper = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          uint32_t y = __shfl_down_sync(0xffffffffu, upper, o);
          if (c.lane + o < 32) upper += y;
        }
        uint32_t acc = upper - mine;
        int hit = -1;
        uint32_t acc_hit = 0;
        for (int q = 0; q < 8 && hit < 0; q++) {
          if (acc + comb_cnt[b_hi - q] >= want) { hit = b_hi - q; acc_hit = acc; }
          acc += comb_cnt[b_hi - q];
        }
        const uint32_t any = __ballot_sync(0xffffffffu, hit >= 0);
        if (any && c.lane == 31 - __clz(any)) { pick[0] = (uint32_t)hit; pick[1] = want - acc_hit; pick[2] = comb_cnt[hit]; }
      }
    }
    __syncthreads();
    const uint32_t digit = pick[0];
    if (kWeighted) above = pick_above; else want = pick[1];
    const uint32_t n_ge = kWeighted ? 0u : (want0 - want) + pick[2];   // elements above the bin plus the bin itself
    cl.sync();   // remote readers are done with this round's histograms
    if (digit == 256) return false;
    prefix |= digit << shift;
    mask |= 255u << shift;
    if (n_ge_out) *n_ge_out = n_ge;
    if (!kWeighted && stop_at && n_ge <= stop_at) break;
  }
  *key_out = prefix;
  return true;
}

// Inverse-CDF search: the first index whose running sum of probabilities exceeds r (Sampler.Sample step 8, sampler.go:200-209;
// resampleRejected, speculative.go:271-291), or `dflt` when the sum never does.  Two calls, so that a pass which sums the row
// anyway (for its normalisation) is not made twice: segment_sums() takes this lane's share of the sum over the warp's
// segment, leaves the sums of the warps in shared memory and those of the CTAs in all[], and returns the row's; cdf_search()
// finds the segment that crosses (its sums times `factor`) and walks that one in index order.
__device__ float segment_sums(Ctx& c, float part, float (&all)[kMaxCluster]) {
  part = warp_sum(part);
  if (c.lane == 0) c.sh->warp_seg[c.warp] = part;
  __syncthreads();
  float tot = 0.0f;
  for (int w = 0; w < kSelWarps; w++) tot += c.sh->warp_seg[w];
  cluster_gather1(c, tot, all);
  float sum = 0.0f;
#pragma unroll
  for (int q = 0; q < kMaxCluster; q++)
    if (q < c.csize) sum += all[q];
  return sum;
}
// Four neighbouring elements of a row from index i; what lies at or past hi is 0 (and must not be used).
__device__ __forceinline__ float4 load4(const Ctx& c, const float* __restrict__ row, int i, int hi) {
  if (c.vec) return i < hi ? __ldg(reinterpret_cast<const float4*>(row + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(i < hi ? __ldg(row + i) : 0.f, i + 1 < hi ? __ldg(row + i + 1) : 0.f, i + 2 < hi ? __ldg(row + i + 2) : 0.f,
                     i + 3 < hi ? __ldg(row + i + 3) : 0.f);
}
// prob(value, value of row2 at the same index); row2 may be nullptr.
template <class ProbF>
__device__ void cdf_search(Ctx& c, const float* __restrict__ row, const float* __restrict__ row2, ProbF prob, float r, int dflt, int32_t* out,
                           const float (&all)[kMaxCluster], float factor) {
  float base = 0.0f, run = 0.0f;
  int cross = -1;
#pragma unroll
  for (int q = 0; q < kMaxCluster; q++) {
    if (q >= c.csize) break;
    if (q == c.rank) base = run;
    run += __fmul_rn(all[q], factor);
    if (cross < 0 && run > r) cross = q;
  }
  // No path below leaves early with the cluster's exchange still in use: the caller ends with a cluster barrier.
  if (cross < 0) {
    if (c.rank == 0 && threadIdx.x == 0) *out = dflt;
    return;
  }
  if (cross != c.rank) return;
  // This CTA holds the crossing: pick the warp, then walk its segment in order.  The warps' sums are scaled one by one and round
  // differently from the CTA's: where none of them crosses, it is the last one that carries probability (the warps behind it
  // may have none, or no elements at all).
  int wsel = kSelWarps - 1;
  float acc = base, wbase = base;
  for (int w = 0; w < kSelWarps; w++) {
    const float seg = c.sh->warp_seg[w], nxt = acc + __fmul_rn(seg, factor);
    if (seg > 0.0f) { wsel = w; wbase = acc; }
    if (nxt > r) break;
    acc = nxt;
  }
  if (c.warp != wsel) return;
  // The segment in blocks of 128 elements, four neighbours per lane, four blocks' loads in flight.  The first block in which
  // the running sum crosses is searched lane by lane, and the lane that crosses element by element.  (Lanes that each summed a
  // contiguous chunk of the segment paid for 16 dependent rounds of scattered loads.)
  acc = wbase;
  int hit = -1, last_pos = -1;
  for (int b0 = c.wlo; b0 < c.whi && hit < 0; b0 += 512) {
    float4 p[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int i = b0 + 128 * u + 4 * c.lane;
      const float4 v = load4(c, row, i, c.whi), v2 = row2 ? load4(c, row2, i, c.whi) : v;
      p[u] = v;
      p[u].x = i < c.whi ? prob(v.x, v2.x) : 0.0f;
      p[u].y = i + 1 < c.whi ? prob(v.y, v2.y) : 0.0f;
      p[u].z = i + 2 < c.whi ? prob(v.z, v2.z) : 0.0f;
      p[u].w = i + 3 < c.whi ? prob(v.w, v2.w) : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const float mine = p[u].x + p[u].y + p[u].z + p[u].w;
      float x = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, x, o);
        if (c.lane >= o) x += y;
      }
      const int i = b0 + 128 * u + 4 * c.lane;
      // the last element so far that carries probability: what is taken when rounding puts the crossing past the end
      const int lp = p[u].w > 0.0f ? i + 3 : p[u].z > 0.0f ? i + 2 : p[u].y > 0.0f ? i + 1 : p[u].x > 0.0f ? i : -1;
      // (lanes without probability do not count: their x is a sum in another order, and may lie above the lane's before them)
      const uint32_t pos = __ballot_sync(0xffffffffu, lp >= 0), over = __ballot_sync(0xffffffffu, lp >= 0 && acc + x > r);
      if (hit < 0) {
        if (over) {
          const float before = __shfl_up_sync(0xffffffffu, x, 1);
          float a = acc + (c.lane > 0 ? before : 0.0f);
          int h = -1;
          a += p[u].x; if (h < 0 && a > r && p[u].x > 0.0f) h = i;
          a += p[u].y; if (h < 0 && a > r && p[u].y > 0.0f) h = i + 1;
          a += p[u].z; if (h < 0 && a > r && p[u].z > 0.0f) h = i + 2;
          a += p[u].w; if (h < 0 && a > r && p[u].w > 0.0f) h = i + 3;
          if (h < 0) h = lp;                     // the lane's own sum rounds differently from its four steps
          hit = __shfl_sync(0xffffffffu, h, __ffs(over) - 1);
        }
        if (pos) last_pos = __shfl_sync(0xffffffffu, lp, 31 - __clz(pos));
        acc += __shfl_sync(0xffffffffu, x, 31);
      }
    }
  }
  if (hit < 0) hit = last_pos >= 0 ? last_pos : c.whi > c.wlo ? c.whi - 1 : dflt;
  if (c.lane == 0) *out = min(hit, c.whi - 1);
}

// Sampler.Sample with a small top-k, finished on a list: after top-k only the k largest logits (and their ties) carry
// probability.  Two looks at the row put them on a list.  Every thread keeps the largest element it has read; with m = k / CTAs
// (rounded up), the m-th largest of a CTA's is a bound that at least m of its elements reach, so the smallest of the CTAs'
// bounds is one that at least k of the row's reach, and hardly more do (about 70 of 131072 for k = 50).  The few threads that
// hold one read their elements again.  (A radix walk over the row for the bound took a histogram round or two, each 3-5 us.)
// Rank 0 gathers the lists and walks the rest of the reference's chain (softmax, nucleus, min-p, draw) over what is on them.
// Every float32 sum runs in index order over the kept elements -- the elements the reference adds zeros for are skipped -- so
// this path gives the reference's token bit for bit.  Lists that would not fit (plateaus of ties, tiny rows) are narrowed down
// by the radix walk; returns false (nothing written) when not even that fits, and the caller takes the pass-per-step path.
constexpr int kCandTopK = 128;   // largest top-k that takes this path
constexpr int kCandCap = 512;    // list capacity

__device__ bool sample_row_candidates(Ctx& c, const SelParams& prm, const float* __restrict__ row, const Dist& d, int topk, float r,
                                      int32_t* out) {
  cg::cluster_group cl = cg::this_cluster();
  const int V = prm.vocab;
  SelShared& sh = *c.sh;
  // the lists live in the histogram block: words [0,512) values, [512,1024) indices of this CTA's
  float* l_val = reinterpret_cast<float*>(&sh.warp_hist[0][0]);
  int32_t* l_idx = reinterpret_cast<int32_t*>(&sh.warp_hist[0][0]) + kCandCap;
  // Puts what reaches key_lo of the elements that the threads with `mine` read in for_segment() on the list.  Where a thread has read
  // eight times or more, a warp goes through one such lane's elements together: a trip to L2 and a few instructions each, where the
  // lane by itself, 64 elements unrolled, took 10 us, most of them its own instructions' way into the cache (131072 logits, 64
  // sequences: 109 -> 103.5 us a call).  Fewer reads are one trip for all the lanes (32000 logits: 39.5 us so, 42.5 lane by lane), and
  // so are many lanes of a warp, which ties at the bound bring: a lane's turn costs about what 256 elements of a whole look do (128 of rows
  // that are read one by one).  131072 equal logits, lane by lane -> now: 177 -> 145 us a call of one row, 301 -> 270 of 64; 40 finite ones
  // among -inf 244 -> 199; 700 ties at the top, 16 rows, 159 -> 152.  (Four lanes as the limit: 64 ordinary rows 41.4 -> 42.3.)
  auto collect = [&](uint32_t key_lo, bool mine) {
    auto put = [&](int i, float v) {
      const float x = d.scaled(v);
      if (bit_key(x) >= key_lo) {
        const uint32_t pos = atomicAdd(&sh.list_count, 1u);
        if (pos < (uint32_t)kCandCap) { l_val[pos] = x; l_idx[pos] = i; }
      }
    };
    const int width = c.vec ? 4 : 1;
    uint32_t lanes = __ballot_sync(0xffffffffu, mine);
    if (c.whi - c.wlo < 8 * 32 * width || __popc(lanes) * (c.vec ? 256 : 128) > c.whi - c.wlo) {
      if (mine) for_segment(c, row, put);
      return;
    }
#pragma unroll 1
    for (; lanes; lanes &= lanes - 1) {
#pragma unroll 1
      for (int i = c.wlo + (__ffs(lanes) - 1 + 32 * c.lane) * width; i < c.whi; i += 1024 * width) {
        const float4 v = load4(c, row, i, c.whi);
#pragma unroll 1
        for (int e = 0; e < width; e++) put(i + e, e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w);
      }
    }
  };
  // The largest element per thread, as a key (the division by the temperature keeps the order, so it is made once, behind the
  // pass).  Of long slices, pairs of threads: half as many keys to rank.
  uint32_t key = 0;
  for_segment(c, row, [&](int, float v) { key = max(key, bit_key(v)); });
  if (key) {
    const uint32_t u = (key & 0x80000000u) ? (key & 0x7fffffffu) : ~key;
    key = bit_key(d.scaled(__uint_as_float(u)));
  }
  const bool pairs = c.hi - c.lo > 8 * kSelThreads;
  const int m = (topk + c.csize - 1) / c.csize;
  const int n_grp = pairs ? kSelThreads / 2 : kSelThreads;
  uint32_t grp = key;
  if (pairs) grp = max(grp, __shfl_xor_sync(0xffffffffu, grp, 1));
  if (!pairs) sh.grp_key[threadIdx.x] = grp;
  else if (!(c.lane & 1)) sh.grp_key[threadIdx.x >> 1] = grp;
  if (threadIdx.x == 0) sh.list_count = 0;
  __syncthreads();
  if ((int)threadIdx.x < n_grp) {
    const uint32_t mine = sh.grp_key[threadIdx.x];
    int gt = 0, ge = 0;
#pragma unroll 4
    for (int j = 0; j < n_grp; j += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(&sh.grp_key[j]);
      gt += (q.x > mine) + (q.y > mine) + (q.z > mine) + (q.w > mine);
      ge += (q.x >= mine) + (q.y >= mine) + (q.z >= mine) + (q.w >= mine);
    }
    if (gt < m && m <= ge) sh.list_bound = mine;   // several threads with the same key write the same value
  }
  __syncthreads();
  cl.sync();
  uint32_t bound = 0xffffffffu;
  for (int q = 0; q < c.csize; q++) bound = min(bound, *cl.map_shared_rank(&sh.list_bound, q));
  bound = with_both_zeros(bound);
  collect(bound, key >= bound);
  __syncthreads();
  cl.sync();
  uint32_t total = 0;
  for (int q = 0; q < c.csize; q++) total += *cl.map_shared_rank(&sh.list_count, q);
  if (total > (uint32_t)kCandCap) {   // uniform over the cluster
    cl.sync();                        // everyone has read the counts
    uint32_t key_lo = 0, n_ge = 0;
    radix_select<false>(c, row, [&](float v, uint32_t& k, float& w) { k = order_key(d.scaled(v)); w = 0.0f; }, (uint32_t)topk, 0.0f, &key_lo,
                        (uint32_t)kCandCap, &n_ge);
    if (n_ge > (uint32_t)kCandCap) return false;     // more ties at the threshold than the list holds
    if (threadIdx.x == 0) sh.list_count = 0;
    __syncthreads();
    collect(with_both_zeros(key_lo), true);
    __syncthreads();
    cl.sync();
  }
  if (c.rank == 0) {
    float* a_val = l_val + 2 * kCandCap;            // all candidates, then the kept ones by index and their probabilities
    int32_t* a_idx = l_idx + 2 * kCandCap;
    float* k_p = l_val + 4 * kCandCap;
    int32_t* k_idx = l_idx + 4 * kCandCap;
    int32_t* k_ord = l_idx + 6 * kCandCap;
    __shared__ int s_n, s_c, s_cut;
    __shared__ float s_thr, s_scale, s_max;
    if (threadIdx.x == 0) { s_n = 0; s_c = 0; }
    __syncthreads();
    {   // gather: the warps share the lists out among them
      const int q = c.warp % c.csize, per = kSelWarps / c.csize;
      const int cnt = (int)*cl.map_shared_rank(&sh.list_count, q);
      const float* rv = cl.map_shared_rank(l_val, q);
      const int32_t* ri = cl.map_shared_rank(l_idx, q);
      for (int t = (c.warp / c.csize) * 32 + c.lane; t < cnt; t += per * 32) {
        const float v = rv[t];
        const int32_t i = ri[t];
        const int pos = atomicAdd(&s_c, 1);
        a_val[pos] = v;
        a_idx[pos] = i;
      }
    }
    __syncthreads();
    const int n_c = s_c;
    // kthLargest (sampler.go:283-300): the value with fewer than topk elements above it and at least topk at or above
    for (int t = threadIdx.x; t < n_c; t += kSelThreads) {
      const float v = a_val[t];
      int gt = 0, ge = 0;
#pragma unroll 4
      for (int j = 0; j < n_c; j++) { gt += a_val[j] > v; ge += a_val[j] >= v; }
      if (gt < topk && topk <= ge) s_thr = v;
      if (gt == 0) s_max = v;
    }
    __syncthreads();
    const float thr = s_thr, maxV = s_max;
    // keep what the mask leaves (not below the threshold), in index order, with its exponential (sampler.go:118-137)
    for (int t = threadIdx.x; t < n_c; t += kSelThreads) {
      const float v = a_val[t];
      if (v < thr) continue;
      const int i = a_idx[t];
      int pos = 0;
#pragma unroll 4
      for (int j = 0; j < n_c; j++) pos += (!(a_val[j] < thr)) && a_idx[j] < i;
      k_idx[pos] = i;
      k_p[pos] = fastexp32_ref(__fsub_rn(v, maxV));
      atomicAdd(&s_n, 1);
    }
    __syncthreads();
    const int n_k = s_n;
    // sums in index order: one thread, four elements a load (what is padded adds zeros)
    auto sum_in_order = [&]() {
      if (threadIdx.x == 0) {
        for (int j = n_k; j < ((n_k + 3) & ~3); j++) k_p[j] = 0.0f;
        float sum = 0.0f;
#pragma unroll 4
        for (int j = 0; j < n_k; j += 4) {
          const float4 q = *reinterpret_cast<const float4*>(k_p + j);
          sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, q.x), q.y), q.z), q.w);
        }
        s_scale = sum > 0.0f ? __fdiv_rn(1.0f, sum) : 1.0f;
      }
      __syncthreads();
    };
    auto rescale = [&]() {
      for (int t = threadIdx.x; t < n_k; t += kSelThreads) k_p[t] = __fmul_rn(k_p[t], s_scale);
      __syncthreads();
    };
    sum_in_order();
    rescale();
    float topP = prm.top_p;
    if (topP <= 0.0f || topP > 1.0f) topP = 1.0f;
    if (topP < 1.0f) {
      // The reference sorts by probability (argsortDescF32, sampler.go:268-281) and cuts where the running sum reaches topP.
      // Which of equal probabilities comes first does not change the sums, so any order by rank gives the cut; only when it
      // falls between equals does it matter which of them are kept, and then the sort is followed step by step (below).
      float* ranked = a_val;
      for (int t = threadIdx.x; t < n_k; t += kSelThreads) {
        const float v = k_p[t];
        int rank = 0;
#pragma unroll 4
        for (int j = 0; j < n_k; j++) rank += k_p[j] > v || (k_p[j] == v && j < t);
        ranked[rank] = v;
        k_ord[t] = rank;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        float cum = 0.0f;
        int cut = n_k;
        for (int j = 0; j < n_k; j += 4) {   // four sums a load: what lies past the end follows the last sum that counts
          const float4 q = *reinterpret_cast<const float4*>(ranked + j);
          const float c0 = __fadd_rn(cum, q.x), c1 = __fadd_rn(c0, q.y), c2 = __fadd_rn(c1, q.z);
          cum = __fadd_rn(c2, q.w);
          const int at = c0 >= topP ? j : c1 >= topP ? j + 1 : c2 >= topP ? j + 2 : cum >= topP ? j + 3 : n_k;
          if (at < n_k) { cut = at + 1; break; }
        }
        s_cut = cut < n_k && ranked[cut] == ranked[cut - 1] ? -1 : cut;
      }
      __syncthreads();
      const int cut = s_cut;
      if (cut >= 0) {
        for (int t = threadIdx.x; t < n_k; t += kSelThreads)
          if (k_ord[t] >= cut) k_p[t] = 0.0f;
        __syncthreads();
      } else {
        // argsortDescF32 followed as far as the cut: a selection sort over all indices whose step i swaps the first largest
        // remaining entry with whatever sits at position i.  Entries without probability are interchangeable, so only the
        // positions of the kept elements are tracked (k_ord: position in the reference's index array, -2 once selected);
        // which of two equal probabilities comes first follows from the swaps, exactly as in the reference.
        for (int t = threadIdx.x; t < n_k; t += kSelThreads) k_ord[t] = k_idx[t];
        __syncthreads();
        if (c.warp == 0) {   // one warp: the search of every step is spread over its lanes, the running sum stays sequential
          float cum = 0.0f;
          bool done = false;
          for (int step = 0; step < n_k && !done; step++) {
            float bp = -1.0f;
            int bpos = 0x7fffffff, bj = -1, at_i = -1;
            for (int j = c.lane; j < n_k; j += 32) {
              const int pj = k_ord[j];
              if (pj < 0) continue;
              if (pj == step) at_i = j;
              const float pv = k_p[j];
              if (pv > bp || (pv == bp && pj < bpos)) { bp = pv; bpos = pj; bj = j; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              const float op = __shfl_xor_sync(0xffffffffu, bp, o);
              const int opos = __shfl_xor_sync(0xffffffffu, bpos, o), oj = __shfl_xor_sync(0xffffffffu, bj, o);
              at_i = max(at_i, __shfl_xor_sync(0xffffffffu, at_i, o));
              if (op > bp || (op == bp && opos < bpos)) { bp = op; bpos = opos; bj = oj; }
            }
            if (bj < 0 || !(bp > 0.0f)) break;      // only zeros are left: the running sum stays below top-p
            if (c.lane == 0) {
              if (at_i >= 0 && at_i != bj) k_ord[at_i] = bpos;   // what sat at position `step` moves to the winner's place
              k_ord[bj] = -2;
            }
            __syncwarp();
            cum = __fadd_rn(cum, bp);
            if (cum >= topP) done = true;
          }
          if (c.lane == 0) s_cut = done ? 1 : 0;
        }
        __syncthreads();
        if (s_cut)
          for (int t = threadIdx.x; t < n_k; t += kSelThreads)
            if (k_ord[t] != -2) k_p[t] = 0.0f;
        __syncthreads();
      }
      sum_in_order();
      rescale();
    }
    if (prm.min_p > 0.0f) {
      if (threadIdx.x == 0) {
        float maxProb = 0.0f;
        for (int j = 0; j < n_k; j++) if (k_p[j] > maxProb) maxProb = k_p[j];
        s_thr = __fmul_rn(maxProb, prm.min_p);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < n_k; t += kSelThreads)
        if (k_p[t] < s_thr) k_p[t] = 0.0f;
      __syncthreads();
      sum_in_order();
      rescale();
    }
    if (threadIdx.x == 0) {
      float cum = 0.0f;
      int tok = V - 1;
      for (int j = 0; j < n_k; j += 4) {
        const float4 q = *reinterpret_cast<const float4*>(k_p + j);
        const float c0 = __fadd_rn(cum, q.x), c1 = __fadd_rn(c0, q.y), c2 = __fadd_rn(c1, q.z);
        cum = __fadd_rn(c2, q.w);
        const int at = r < c0 ? j : r < c1 ? j + 1 : r < c2 ? j + 2 : r < cum ? j + 3 : n_k;
        if (at < n_k) { tok = k_idx[at]; break; }
      }
      *out = tok;
    }
  }
  return true;
}

// Sampler.Sample on one row (sampler.go:73-218, steps 3-8; no repetition penalties), one cluster per row.
__device__ void sample_row(Ctx& c, const SelParams& prm, const float* __restrict__ row, float r, int32_t* out) {
  const int V = prm.vocab;
  Dist d;
  d.temp = prm.temperature <= 0.0f ? 1e-5f : prm.temperature;
  d.topk_key = 0; d.tau = 0.0f; d.inv2 = 1.0f; d.minp_thr = 0.0f; d.inv3 = 1.0f;
  bool nucleus = false, minp = false;
  int topk = prm.top_k;
  if (topk < 0 || topk >= V) topk = 0;
  d.m = 0.0f; d.inv1 = 1.0f;
  if (topk > 0 && topk <= kCandTopK && sample_row_candidates(c, prm, row, d, topk, r, out)) return;
  if (topk > 0) {
    uint32_t key = 0;
    radix_select<false>(c, row, [&](float v, uint32_t& k, float& w) { k = order_key(d.scaled(v)); w = 0.0f; }, (uint32_t)topk, 0.0f, &key);
    d.topk_key = with_both_zeros(key);
  }
  float v4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for_segment(c, row, [&](int, float v) { v4[0] = fmaxf(v4[0], v); });
  cluster_reduce4<1>(c, v4);
  d.m = d.scaled(v4[0]);   // the division keeps the order: one of it instead of one an element
  d.inv1 = 1.0f;
  float all[kMaxCluster], part = 0.0f;
  for_segment(c, row, [&](int, float v) { part += d.p1(v); });
  const float sum = segment_sums(c, part, all);
  if (sum > 0.0f) d.inv1 = __fdiv_rn(1.0f, sum);
  float topP = prm.top_p;
  if (topP <= 0.0f || topP > 1.0f) topP = 1.0f;
  if (topP < 1.0f) {
    nucleus = true;
    uint32_t key = 0;
    bool cut = radix_select<true>(c, row, [&](float v, uint32_t& k, float& w) { w = d.p1(v); k = __float_as_uint(w); }, 0u, topP, &key);
    const float tau = cut ? __uint_as_float(key) : 0.0f;
    part = 0.0f;
    for_segment(c, row, [&](int, float v) { float p = d.p1(v); if (p >= tau) part += p; });
    const float kept = segment_sums(c, part, all);
    d.tau = tau;
    d.inv2 = kept > 0.0f ? __fdiv_rn(1.0f, kept) : 1.0f;
  }
  // Dist::p2 drops below tau only when tau > 0; the renormalisation applies whenever the nucleus step ran
  auto p2 = [&](float v) { float p = d.p1(v); if (nucleus) p = p < d.tau ? 0.0f : __fmul_rn(p, d.inv2); return p; };
  if (prm.min_p > 0.0f) {
    minp = true;
    // the largest probability belongs to the row maximum, which no filter removes
    v4[0] = v4[1] = v4[2] = v4[3] = 0.0f;
    for_segment(c, row, [&](int, float v) { v4[0] = fmaxf(v4[0], p2(v)); });
    cluster_reduce4<1>(c, v4);
    const float thr = __fmul_rn(v4[0], prm.min_p);
    v4[0] = v4[1] = v4[2] = v4[3] = 0.0f;
    for_segment(c, row, [&](int, float v) { float p = p2(v); if (!(p < thr)) v4[0] += p; });
    cluster_reduce4<0>(c, v4);
    d.minp_thr = thr;
    d.inv3 = v4[0] > 0.0f ? __fdiv_rn(1.0f, v4[0]) : 1.0f;
  }
  auto p3 = [&](float v, float) { float p = p2(v); if (minp) p = p < d.minp_thr ? 0.0f : __fmul_rn(p, d.inv3); return p; };
  float factor = nucleus ? d.inv2 : d.inv1;   // the segments of the last normalisation are the search's
  if (minp) {
    factor = 1.0f;
    part = 0.0f;
    for_segment(c, row, [&](int, float v) { part += p3(v, 0.0f); });
    segment_sums(c, part, all);
  }
  cdf_search(c, row, nullptr, p3, r, V - 1, out, all, factor);
}

__global__ void __launch_bounds__(kSelThreads, 2) spec_accept_kernel(SelParams prm) {
  cg::cluster_group cl = cg::this_cluster();
  __shared__ SelShared sh;
  Ctx c;
  c.sh = &sh;
  c.csize = (int)cl.num_blocks();
  c.rank = (int)cl.block_rank();
  c.warp = threadIdx.x >> 5;
  c.lane = threadIdx.x & 31;
  c.round = 0;
  const int V = prm.vocab, k = prm.k;
  const int per = ((V + c.csize - 1) / c.csize + 127) & ~127;
  c.lo = min(V, c.rank * per);
  c.hi = min(V, c.lo + per);
  const int wper = ((c.hi - c.lo + kSelWarps - 1) / kSelWarps + 127) & ~127;
  c.vec = (V & 3) == 0 && (((uintptr_t)prm.target_logits | (uintptr_t)prm.draft_logits) & 15) == 0;
  c.wlo = min(c.hi, c.lo + c.warp * wper);
  c.whi = min(c.hi, c.wlo + wper);
  const int b = blockIdx.x / c.csize;
  if (threadIdx.x == 0) stamp_begin(prm.time);
  const float* draws = prm.draws + (size_t)b * (k + 1);
  int32_t* out_tok = prm.next_token + b;
  const bool writer = c.rank == 0 && threadIdx.x == 0;
  int used = 0;
  int n_acc = k;
  bool done = false;
  // Maximum and sum of exponentials of a draft and a target row in ONE pass: the sum needs the maximum first (fastexp32 is not
  // multiplicative), so it is taken against a guess, the logit of the draft token -- the draft's largest where the draft model
  // decodes greedily, and the target's where the two agree -- and made again, out of L2, for a row whose maximum turns out to
  // be another.
  auto drow_of = [&](int i) { return prm.draft_logits + ((size_t)b * k + i) * V; };
  auto trow_of = [&](int i) { return prm.target_logits + ((size_t)b * (k + 1) + i) * V; };
  auto fetch = [&](int i, int32_t& tok, float& gd, float& gt) {   // tok as it is, possibly outside the vocabulary
    if (i < kAhead) {
      tok = sh.tok[i];
      gd = sh.guess[0][i];
      gt = sh.guess[1][i];
    } else {
      tok = prm.draft_tokens[(size_t)b * k + i];
      const int j = min(max(tok, 0), V - 1);
      gd = __ldg(drow_of(i) + j);
      gt = __ldg(trow_of(i) + j);
    }
  };
  if ((int)threadIdx.x < min(k, kAhead)) {
    const int i = threadIdx.x, tok = prm.draft_tokens[(size_t)b * k + i], j = min(max(tok, 0), V - 1);
    sh.tok[i] = tok;
    sh.guess[0][i] = __ldg(drow_of(i) + j);
    sh.guess[1][i] = __ldg(trow_of(i) + j);
  } else if (threadIdx.x >= 64 && (int)threadIdx.x - 64 <= min(k, kAhead)) {
    sh.draw[threadIdx.x - 64] = draws[threadIdx.x - 64];
  }
  __syncthreads();
  auto next_draw = [&]() {
    const int j = used++;
    return j <= kAhead ? sh.draw[j] : draws[j];
  };
  auto pair_pass = [&](int i, float& sd, float& st, float& md, float& mt) {
    int32_t tok;
    float gd, gt;
    fetch(i, tok, gd, gt);
    float a = 0.0f, t = 0.0f, ma = -INFINITY, mb = -INFINITY;
    for_segment2(c, drow_of(i), trow_of(i), [&](int, float dv, float tv) {
      ma = fmaxf(ma, dv);
      mb = fmaxf(mb, tv);
      a += fastexp32_below(__fsub_rn(dv, gd));
      t += fastexp32_below(__fsub_rn(tv, gt));
    });
    sd = a; st = t; md = ma; mt = mb;
  };
  // the sums again where the guess was not the maximum; which they are (bit 0: draft, bit 1: target)
  auto pair_again = [&](int i, float md, float mt, float& sd, float& st) {
    int32_t tok;
    float gd, gt;
    fetch(i, tok, gd, gt);
    const int bad = (gd != md ? 1 : 0) | (gt != mt ? 2 : 0);
    float a = 0.0f, t = 0.0f;
    if (bad == 3)
      for_segment2(c, drow_of(i), trow_of(i), [&](int, float dv, float tv) { a += fastexp32_below(__fsub_rn(dv, md)); t += fastexp32_below(__fsub_rn(tv, mt)); });
    else if (bad == 1)
      for_segment(c, drow_of(i), [&](int, float dv) { a += fastexp32_below(__fsub_rn(dv, md)); });
    else if (bad == 2)
      for_segment(c, trow_of(i), [&](int, float tv) { t += fastexp32_below(__fsub_rn(tv, mt)); });
    sd = a; st = t;
    return bad;
  };
  // Few sequences: the chain's length is what costs, not the bytes.  The rows of ALL draft positions are read in one stage, so
  // the accept loop below runs without a pass of its own per position (rows after a rejection are read in vain).
  const bool batched = prm.batched && k >= 2 && 4 * k <= kStatMax;
  if (batched) {
    float acc[kStatMax];
    for (int i = 0; i < k; i++) pair_pass(i, acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]);
    cluster_reduce_n(c, acc, 4 * k, c.sh->stat);
  }
  for (int i = 0; i < k && !done; i++) {
    const float* drow = drow_of(i);
    const float* trow = trow_of(i);
    int32_t tok;
    float tok_d, tok_t;   // the token's logits
    fetch(i, tok, tok_d, tok_t);
    if (tok < 0 || tok >= V) {   // uniform over the cluster: every thread reads the same token
      if (writer) { set_status(prm.status, RELUX_ERR_INVALID_ARG); *out_tok = -1; }
      n_acc = -1;
      done = true;
      break;
    }
    float v4[4], md, mt;
    if (batched) {
      v4[0] = c.sh->stat[4 * i];
      v4[1] = c.sh->stat[4 * i + 1];
      md = c.sh->stat[4 * i + 2];
      mt = c.sh->stat[4 * i + 3];
    } else {
      pair_pass(i, v4[0], v4[1], v4[2], v4[3]);
      cluster_reduce4<2>(c, v4);
      md = v4[2];
      mt = v4[3];
    }
    const float u = next_draw();
    if (tok_d != md || tok_t != mt) {
      // A sum against a guess says most of what the one against the maximum would: fastexp32 is e^x but for a factor between
      // 0.967 and 1.027, so the two differ from e^(guess - maximum) by a factor below 1.062.  A draw that is accepted with that
      // much to spare needs no second pass (the usual case); everything else gets the sums as the reference has them.
      constexpr float kSpare = 1.07f;
      const float est_d = v4[0] * expf(tok_d - md), est_t = v4[1] * expf(tok_t - mt);
      const float dP = fastexp32_ref(__fsub_rn(tok_d, md)) / est_d * (tok_d != md ? kSpare : 1.0001f);
      const float tP = fastexp32_ref(__fsub_rn(tok_t, mt)) / est_t / (tok_t != mt ? kSpare : 1.0001f);
      const bool sound = md - tok_d < 80.0f && mt - tok_t < 80.0f && v4[0] < 1e38f && v4[1] < 1e38f;   // false for NaN too
      if (sound && u < fminf(tP / fmaxf(dP, 1e-10f), 1.0f)) continue;
      float w4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      const int bad = pair_again(i, md, mt, w4[0], w4[1]);
      cluster_reduce4<0>(c, w4);
      if (bad & 1) v4[0] = w4[0];
      if (bad & 2) v4[1] = w4[1];
    }
    const float invd = v4[0] > 0.0f ? __fdiv_rn(1.0f, v4[0]) : 1.0f;
    const float invt = v4[1] > 0.0f ? __fdiv_rn(1.0f, v4[1]) : 1.0f;
    const float dP = __fmul_rn(fastexp32_ref(__fsub_rn(tok_d, md)), invd);
    const float tP = __fmul_rn(fastexp32_ref(__fsub_rn(tok_t, mt)), invt);
    float ap = __fdiv_rn(tP, dP > 1e-10f ? dP : 1e-10f);
    if (ap > 1.0f) ap = 1.0f;
    if (u < ap) continue;
    // rejected at i: resample from norm(max(0, p_target - p_draft))   speculative.go:256-295
    auto adj = [&](float tv, float dv) {
      float tp = __fmul_rn(fastexp32_ref(__fsub_rn(tv, mt)), invt);
      float dp = __fmul_rn(fastexp32_ref(__fsub_rn(dv, md)), invd);
      float diff = __fsub_rn(tp, dp);
      return diff < 0.0f ? 0.0f : diff;
    };
    float all[kMaxCluster], part = 0.0f;
    for_segment2(c, drow, trow, [&](int, float dv, float tv) { part += adj(tv, dv); });
    const float sum = segment_sums(c, part, all);
    const float r = next_draw();
    if (sum > 0.0f) {
      const float inv = __fdiv_rn(1.0f, sum);
      cdf_search(c, trow, drow, [&](float tv, float dv) { return __fmul_rn(adj(tv, dv), inv); }, r, 0, out_tok, all, inv);
    } else {
      auto tprob = [&](float tv, float) { return __fmul_rn(fastexp32_ref(__fsub_rn(tv, mt)), invt); };
      part = 0.0f;
      for_segment(c, trow, [&](int, float tv) { part += tprob(tv, 0.0f); });
      segment_sums(c, part, all);
      cdf_search(c, trow, nullptr, tprob, r, 0, out_tok, all, 1.0f);
    }
    n_acc = i;
    done = true;
  }
  if (!done) sample_row(c, prm, prm.target_logits + ((size_t)b * (k + 1) + k) * V, next_draw(), out_tok);
  if (writer && prm.n_accepted) prm.n_accepted[b] = n_acc;
  cl.sync();   // no CTA leaves while another may still read its exchange buffers
  if (threadIdx.x == 0) stamp_end(prm.time);
}

// ---- REFERENCE: one thread per sequence, the reference's loops in the reference's order ------------------------
__device__ void ref_softmax_alloc(const float* logits, int n, float* probs) {   // speculative.go:346-368
  float maxV = logits[0];
  for (int i = 1; i < n; i++)
    if (logits[i] > maxV) maxV = logits[i];
  float sum = 0.0f;
  for (int i = 0; i < n; i++) {
    probs[i] = fastexp32_ref(__fsub_rn(logits[i], maxV));
    sum = __fadd_rn(sum, probs[i]);
  }
  if (sum > 0.0f) {
    const float inv = __fdiv_rn(1.0f, sum);
    for (int i = 0; i < n; i++) probs[i] = __fmul_rn(probs[i], inv);
  }
}

__device__ void ref_renormalise(float* probs, int n) {
  float s = 0.0f;
  for (int i = 0; i < n; i++) s = __fadd_rn(s, probs[i]);
  if (s > 0.0f) {
    const float inv = __fdiv_rn(1.0f, s);
    for (int i = 0; i < n; i++) probs[i] = __fmul_rn(probs[i], inv);
  }
}

// Sampler.Sample steps 3-8 (sampler.go:89-209).  scratch, probs: [n] floats; idx: [n] ints.
__device__ int ref_sample(const SelParams& prm, const float* logits, int n, float r, float* scratch, float* probs, int32_t* idx) {
  float temp = prm.temperature <= 0.0f ? 1e-5f : prm.temperature;
  for (int i = 0; i < n; i++) scratch[i] = temp != 1.0f ? __fdiv_rn(logits[i], temp) : logits[i];
  int topK = prm.top_k;
  if (topK < 0 || topK >= n) topK = 0;
  if (topK > 0) {
    // value of the topK-th largest element, duplicates counted (kthLargest, sampler.go:283-300)
    float bound = INFINITY;
    int seen = 0;
    float threshold = scratch[0];
    while (true) {
      float best = -INFINITY;
      int cnt = 0;
      for (int i = 0; i < n; i++) {
        const float v = scratch[i];
        if (v < bound) {
          if (v > best) { best = v; cnt = 1; }
          else if (v == best) cnt++;
        }
      }
      if (cnt == 0) break;
      seen += cnt;
      threshold = best;
      if (seen >= topK) break;
      bound = best;
    }
    for (int i = 0; i < n; i++)
      if (scratch[i] < threshold) scratch[i] = -INFINITY;
  }
  float maxV = scratch[0];
  for (int i = 1; i < n; i++)
    if (scratch[i] > maxV) maxV = scratch[i];
  float sum = 0.0f;
  for (int i = 0; i < n; i++) {
    if (scratch[i] == -INFINITY) probs[i] = 0.0f;
    else { probs[i] = fastexp32_ref(__fsub_rn(scratch[i], maxV)); sum = __fadd_rn(sum, probs[i]); }
  }
  if (sum > 0.0f) {
    const float inv = __fdiv_rn(1.0f, sum);
    for (int i = 0; i < n; i++) probs[i] = __fmul_rn(probs[i], inv);
  }
  float topP = prm.top_p;
  if (topP <= 0.0f || topP > 1.0f) topP = 1.0f;
  if (topP < 1.0f) {
    // argsortDescF32's selection sort (sampler.go:268-281), stopped at the cut-off: later positions are all zeroed
    for (int i = 0; i < n; i++) idx[i] = i;
    float cum = 0.0f;
    int cutoff = n;
    for (int i = 0; i < n; i++) {
      int maxJ = i;
      for (int j = i + 1; j < n; j++)
        if (probs[idx[j]] > probs[idx[maxJ]]) maxJ = j;
      const int t = idx[i]; idx[i] = idx[maxJ]; idx[maxJ] = t;
      cum = __fadd_rn(cum, probs[idx[i]]);
      if (cum >= topP) { cutoff = i + 1; break; }
    }
    for (int j = cutoff; j < n; j++) probs[idx[j]] = 0.0f;
    ref_renormalise(probs, n);
  }
  if (prm.min_p > 0.0f) {
    float maxProb = 0.0f;
    for (int i = 0; i < n; i++)
      if (probs[i] > maxProb) maxProb = probs[i];
    const float threshold = __fmul_rn(maxProb, prm.min_p);
    for (int i = 0; i < n; i++)
      if (probs[i] < threshold) probs[i] = 0.0f;
    ref_renormalise(probs, n);
  }
  float cum = 0.0f;
  for (int i = 0; i < n; i++) {
    cum = __fadd_rn(cum, probs[i]);
    if (r < cum) return i;
  }
  return n - 1;
}

__global__ void spec_accept_reference_kernel(SelParams prm, int n_seqs, float* fscratch, int32_t* iscratch) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n_seqs) return;
  const int V = prm.vocab, k = prm.k;
  float* dp = fscratch + (size_t)b * 2 * V;
  float* tp = dp + V;
  int32_t* idx = iscratch + (size_t)b * V;
  const float* draws = prm.draws + (size_t)b * (k + 1);
  int used = 0;
  for (int i = 0; i < k; i++) {
    const int tok = prm.draft_tokens[(size_t)b * k + i];
    if (tok < 0 || tok >= V) {
      set_status(prm.status, RELUX_ERR_INVALID_ARG);
      prm.next_token[b] = -1;
      if (prm.n_accepted) prm.n_accepted[b] = -1;
      return;
    }
    ref_softmax_alloc(prm.draft_logits + ((size_t)b * k + i) * V, V, dp);
    ref_softmax_alloc(prm.target_logits + ((size_t)b * (k + 1) + i) * V, V, tp);
    const float dP = dp[tok], tP = tp[tok];
    float ap = __fdiv_rn(tP, dP > 1e-10f ? dP : 1e-10f);
    if (ap > 1.0f) ap = 1.0f;
    if (draws[used++] < ap) continue;
    // resampleRejected (speculative.go:256-295); the adjusted row overwrites dp
    float sum = 0.0f;
    for (int j = 0; j < V; j++) {
      float diff = __fsub_rn(tp[j], dp[j]);
      if (diff < 0.0f) diff = 0.0f;
      dp[j] = diff;
      sum = __fadd_rn(sum, diff);
    }
    const float r = draws[used++];
    int result = 0;
    float cum = 0.0f;
    if (sum > 0.0f) {
      const float inv = __fdiv_rn(1.0f, sum);
      for (int j = 0; j < V; j++) {
        cum = __fadd_rn(cum, __fmul_rn(dp[j], inv));
        if (r < cum) { result = j; break; }
      }
    } else {
      for (int j = 0; j < V; j++) {
        cum = __fadd_rn(cum, tp[j]);
        if (r < cum) { result = j; break; }
      }
    }
    prm.next_token[b] = result;
    if (prm.n_accepted) prm.n_accepted[b] = i;
    return;
  }
  prm.next_token[b] = ref_sample(prm, prm.target_logits + ((size_t)b * (k + 1) + k) * V, V, draws[used++], dp, tp, idx);
  if (prm.n_accepted) prm.n_accepted[b] = k;
}


// Sampler.applyRepetitionPenalties (sampler.go:221-266): copies every row to `dst` and rewrites the logits of the tokens
// in the row's window of previous tokens -- repeat penalty (divide a positive logit, multiply a negative one), then
// frequency penalty times the token's count in the window, then presence penalty, each applied once per distinct
// token, in float32 like the reference.  One block per row; win_off [n + 1] delimits the rows' windows in win_tok.
__global__ void repetition_penalty_kernel(const float* __restrict__ src, float* __restrict__ dst, int vocab,
                                          const int32_t* __restrict__ win_tok, const int32_t* __restrict__ win_off,
                                          float rp, float fp, float pp) {
  const int b = blockIdx.x;
  const float* s = src + (size_t)b * vocab;
  float* d = dst + (size_t)b * vocab;
  if ((vocab & 3) == 0 && ((((uintptr_t)src) | ((uintptr_t)dst)) & 15) == 0) {
    for (int i = threadIdx.x * 4; i < vocab; i += blockDim.x * 4)
      *reinterpret_cast<float4*>(d + i) = __ldg(reinterpret_cast<const float4*>(s + i));
  } else {
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) d[i] = s[i];
  }
  __syncthreads();
  const int w0 = win_off[b], w1 = win_off[b + 1];
  for (int j = w0 + threadIdx.x; j < w1; j += blockDim.x) {
    const int tok = win_tok[j];
    if (tok < 0 || tok >= vocab) continue;
    bool first = true;
    int freq = 0;
    for (int q = w0; q < w1; q++) {
      if (win_tok[q] == tok) { freq++; if (q < j) first = false; }
    }
    if (!first) continue;     // one thread per distinct token: the first occurrence owns the update
    float x = d[tok];
    if (rp != 1.0f && rp != 0.0f) x = x > 0.0f ? __fdiv_rn(x, rp) : __fmul_rn(x, rp);
    if (fp != 0.0f) x = __fsub_rn(x, __fmul_rn(fp, (float)freq));
    if (pp != 0.0f) x = __fsub_rn(x, pp);
    d[tok] = x;
  }
}

// Launches the selection kernel on device-resident inputs (prm holds the input pointers, k and vocab) and synchronises the
// stream.  *host: the 2 n result words (accepted counts, then tokens), which the kernel writes to page-locked host memory
// itself (one word each per row, nothing reads them back), and it stamps its own time: the copy, two event records and a
// memset around it took 12 us of a 200 us call.
static int32_t launch_selection(Pool* p, SelParams& prm, int n, const relux_sampler_params& sp, int mode, const int32_t** host) {
  Device* dev = p->dev;
  const int V = prm.vocab;
  int32_t rc;
  if (p->sel_words < 2 * (size_t)n) {
    if (p->sel_host) {
      RELUX_CUDA_TRY(cudaStreamSynchronize(dev->stream));   // an earlier call that failed may have left its kernel running
      int32_t* old = p->sel_host;
      p->sel_host = nullptr;
      p->sel_words = 0;
      RELUX_CUDA_TRY(cudaFreeHost(old));
    }
    const size_t words = std::max<size_t>(512, 2 * (size_t)n);
    RELUX_CUDA_TRY(cudaMallocHost((void**)&p->sel_host, words * sizeof(int32_t)));
    p->sel_words = words;
  }
  prm.n_accepted = p->sel_host;
  prm.next_token = prm.n_accepted + n;
  prm.status = p->d_status;
  prm.temperature = sp.temperature;
  prm.top_k = sp.top_k;
  prm.top_p = sp.top_p;
  prm.min_p = sp.min_p;
  prm.batched = n <= 24 ? 1 : 0;
  if (p->tune.get(RELUX_TUNE_SEL_BATCHED) >= 0) prm.batched = p->tune.get(RELUX_TUNE_SEL_BATCHED) ? 1 : 0;       // tuning knob
  if (mode == RELUX_ATTN_REFERENCE) {
    // One thread per sequence repeats the reference's selection sorts: quadratic in the vocabulary for the nucleus cut,
    // top_k x vocabulary for kthLargest.  Refuse sizes that would keep the device busy for many seconds.
    const bool nucleus = sp.top_p > 0.0f && sp.top_p < 1.0f;
    const bool topk = sp.top_k > 0 && sp.top_k < V;
    if ((nucleus && V > 32768) || (topk && (double)sp.top_k * V > 1e9)) {
      set_error("RELUX_ATTN_REFERENCE repeats the reference's O(vocab^2) sorts on one thread per sequence: vocab %d with these "
                "filters is outside what it is meant for (parity checks); use RELUX_ATTN_FAST", V);
      return RELUX_ERR_UNSUPPORTED;
    }
    rc = grow(dev, p->part_o, sizeof(float) * 2 * (size_t)n * V);
    if (rc) return rc;
    rc = grow(dev, p->part_ml, sizeof(int32_t) * (size_t)n * V);
    if (rc) return rc;
  }
  // device time of the selection kernel, readable through relux_pool_kernel_ms_mean like the attention kernels'
  if (mode == RELUX_ATTN_REFERENCE) {
    if (int32_t rct = time_events_begin(p, p->attn_times)) return rct;
    spec_accept_reference_kernel<<<(n + 31) / 32, 32, 0, dev->stream>>>(prm, n, (float*)p->part_o.p, (int32_t*)p->part_ml.p);
    RELUX_CUDA_TRY(cudaGetLastError());
    if (int32_t rct = time_events_end(p, p->attn_times)) return rct;
  } else {
    prm.time = time_stamp_next(p, p->attn_times);
    // Cluster size: slices should stay long enough to keep 512 threads busy, and all sequences should be resident at
    // once -- a second wave of clusters doubles the latency of the whole chain, which costs more than longer slices.
    const int by_vocab = V >= 32768 ? 8 : V >= 8192 ? 4 : V >= 2048 ? 2 : 1;
    static int resident[64][4] = {};   // [device][log2 cluster size]: clusters the device holds at once, 0 = not asked yet
    int csize = 1;
    double best = 1e30;
    for (int lg = 3; lg >= 0; lg--) {
      const int cs = 1 << lg;
      if (cs > by_vocab) continue;
      int& have = resident[dev->index & 63][lg];
      if (have == 0) {
        cudaLaunchConfig_t q{};
        q.gridDim = dim3((unsigned)(cs * 64));
        q.blockDim = dim3(kSelThreads);
        cudaLaunchAttribute qa{};
        qa.id = cudaLaunchAttributeClusterDimension;
        qa.val.clusterDim.x = (unsigned)cs;
        qa.val.clusterDim.y = qa.val.clusterDim.z = 1;
        q.attrs = &qa;
        q.numAttrs = 1;
        int nc = 0;
        if (cudaOccupancyMaxActiveClusters(&nc, spec_accept_kernel, &q) != cudaSuccess || nc <= 0) { cudaGetLastError(); nc = 1; }
        have = nc;
      }
      const double cost = (double)((n + have - 1) / have) / cs;   // waves x slice length
      if (cost <= best) { best = cost; csize = cs; }   // on a tie the smaller cluster: fewer waves, fewer remote reads
    }
    {   // tuning knob: 1, 2, 4 or 8
      const int v = p->tune.get(RELUX_TUNE_SEL_CLUSTER);
      if (v == 1 || v == 2 || v == 4 || v == 8) csize = v;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(n * csize));
    cfg.blockDim = dim3(kSelThreads);
    cfg.stream = dev->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)csize;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    RELUX_CUDA_TRY(cudaLaunchKernelEx(&cfg, spec_accept_kernel, prm));
    time_stamp_done(p->attn_times, prm.time);
  }
  count_launch(dev);
  RELUX_CUDA_TRY(cudaStreamSynchronize(dev->stream));
  *host = p->sel_host;
  return RELUX_OK;
}

}  // namespace

int32_t do_spec_accept(Pool* p, const relux_spec_accept_args* a) {
  if (!a) { set_error("nil argument struct"); return RELUX_ERR_INVALID_ARG; }
  const int n = a->n_seqs, k = a->k, V = a->vocab;
  if (n <= 0 || k < 0 || V <= 0 || !a->target_logits || !a->draws || !a->next_token ||
      (k > 0 && (!a->draft_tokens || !a->draft_logits || !a->n_accepted)) ||
      (a->mem != RELUX_MEM_HOST && a->mem != RELUX_MEM_DEVICE) ||
      (a->mode != RELUX_ATTN_FAST && a->mode != RELUX_ATTN_REFERENCE)) {
    set_error("spec_accept: bad arguments");
    return RELUX_ERR_INVALID_ARG;
  }
  if (a->commit) {
    // checked before anything is launched, so that a commit is all or nothing: every sequence live and named once, and
    // room on every layer for the longest possible result (k + 1 rows)
    if (n > p->prm.max_seqs) { set_error("spec_accept: more sequences than the pool holds"); return RELUX_ERR_INVALID_ARG; }
    SeqBatch chk;
    int32_t rc0 = stage_batch(p, n, a->seq_ids, nullptr, 1, &chk);
    if (rc0) return rc0;
    for (int l = 0; l < p->prm.num_layers; l++)
      for (int i = 0; i < n; i++) {
        const int s = chk.seq[i];
        const int len = p->h_len[(size_t)l * p->prm.max_seqs + s], cap = p->seq_pages[s] * p->prm.page_tokens;
        if (len + k + 1 > cap) {
          set_error("spec_accept: committing up to %d rows would pass the capacity %d of sequence %d on layer %d (length %d)", k + 1, cap, s, l, len);
          return RELUX_ERR_OVERFLOW;
        }
      }
  }
  if (a->mem == RELUX_MEM_HOST)
    for (size_t i = 0; i < (size_t)n * k; i++)
      if (a->draft_tokens[i] < 0 || a->draft_tokens[i] >= V) {
        set_error("spec_accept: draft token %d outside the vocabulary of %d", a->draft_tokens[i], V);
        return RELUX_ERR_INVALID_ARG;
      }
  SelParams prm{};
  const void* d = nullptr;
  int32_t rc;
  if (k > 0) {
    rc = stage_in(p, p->in_a, a->draft_logits, sizeof(float) * (size_t)n * k * V, a->mem, &d);
    if (rc) return rc;
    prm.draft_logits = (const float*)d;
    rc = stage_in(p, p->q_conv, a->draft_tokens, sizeof(int32_t) * (size_t)n * k, a->mem, &d);
    if (rc) return rc;
    prm.draft_tokens = (const int32_t*)d;
  }
  rc = stage_in(p, p->in_b, a->target_logits, sizeof(float) * (size_t)n * (k + 1) * V, a->mem, &d);
  if (rc) return rc;
  prm.target_logits = (const float*)d;
  rc = stage_in(p, p->o_lat, a->draws, sizeof(float) * (size_t)n * (k + 1), a->mem, &d);
  if (rc) return rc;
  prm.draws = (const float*)d;
  prm.k = k;
  prm.vocab = V;
  const int32_t* host = nullptr;
  rc = launch_selection(p, prm, n, a->sampler, a->mode, &host);
  if (rc) return rc;
  for (int i = 0; i < n; i++) {
    if (a->n_accepted) a->n_accepted[i] = host[i];
    a->next_token[i] = host[(size_t)n + i];
    if (host[(size_t)n + i] < 0 || (k > 0 && host[i] < 0)) {
      set_error("spec_accept: a draft token of sequence %d lies outside the vocabulary of %d", i, V);
      return RELUX_ERR_INVALID_ARG;
    }
  }
  if (a->commit) {
    std::vector<int32_t> new_len((size_t)n);
    for (int l = 0; l < p->prm.num_layers; l++) {
      for (int i = 0; i < n; i++) {
        const int s = a->seq_ids ? a->seq_ids[i] : i;
        if (s < 0 || s >= p->prm.max_seqs) { set_error("spec_accept: bad sequence id %d", s); return RELUX_ERR_INVALID_ARG; }
        new_len[i] = p->h_len[(size_t)l * p->prm.max_seqs + s] + (k > 0 ? host[i] : 0) + 1;
      }
      rc = seq_set_len(p, l, n, a->seq_ids, new_len.data());
      if (rc) return rc;
    }
  }
  return RELUX_OK;
}

int32_t do_sample(Pool* p, const relux_sample_args* a) {
  if (!a) { set_error("nil argument struct"); return RELUX_ERR_INVALID_ARG; }
  const int n = a->n_rows, V = a->vocab;
  if (n <= 0 || V <= 0 || !a->logits || !a->draws || !a->tokens || (a->mem != RELUX_MEM_HOST && a->mem != RELUX_MEM_DEVICE) ||
      (a->mode != RELUX_ATTN_FAST && a->mode != RELUX_ATTN_REFERENCE) || (a->prev_tokens && (!a->prev_len || a->prev_stride < 0))) {
    set_error("sampler_sample: bad arguments");
    return RELUX_ERR_INVALID_ARG;
  }
  Device* dev = p->dev;
  SelParams prm{};
  const void* d = nullptr;
  int32_t rc = stage_in(p, p->in_b, a->logits, sizeof(float) * (size_t)n * V, a->mem, &d);
  if (rc) return rc;
  prm.target_logits = (const float*)d;
  rc = stage_in(p, p->o_lat, a->draws, sizeof(float) * (size_t)n, a->mem, &d);
  if (rc) return rc;
  prm.draws = (const float*)d;
  const bool penalties = a->prev_tokens && ((a->repeat_penalty != 1.0f && a->repeat_penalty != 0.0f) || a->frequency_penalty != 0.0f ||
                                            a->presence_penalty != 0.0f);
  if (penalties) {
    // the window of every row (sampler.go:225-228), flattened: offsets [n + 1] then tokens
    std::vector<int32_t> flat((size_t)n + 1, 0);
    for (int i = 0; i < n; i++) {
      int len = a->prev_len[i];
      if (len < 0 || len > a->prev_stride) { set_error("sampler_sample: prev_len[%d] = %d outside [0, %d]", i, len, a->prev_stride); return RELUX_ERR_INVALID_ARG; }
      int w0 = (a->repeat_window > 0 && len > a->repeat_window) ? len - a->repeat_window : 0;
      const int32_t* row = a->prev_tokens + (size_t)i * a->prev_stride;
      flat.insert(flat.end(), row + w0, row + len);
      flat[i + 1] = (int32_t)(flat.size() - (size_t)n - 1);
    }
    if (flat.size() > (size_t)n + 1) {
      rc = grow(dev, p->q_conv, sizeof(int32_t) * flat.size());
      if (rc) return rc;
      rc = grow(dev, p->layer_buf, sizeof(float) * (size_t)n * V);
      if (rc) return rc;
      // pageable source: the copy has left the vector when the call returns
      RELUX_CUDA_TRY(cudaMemcpyAsync(p->q_conv.p, flat.data(), sizeof(int32_t) * flat.size(), cudaMemcpyHostToDevice, dev->stream));
      const int32_t* d_off = (const int32_t*)p->q_conv.p;
      repetition_penalty_kernel<<<n, 256, 0, dev->stream>>>(prm.target_logits, (float*)p->layer_buf.p, V, d_off + n + 1, d_off,
                                                            a->repeat_penalty, a->frequency_penalty, a->presence_penalty);
      RELUX_CUDA_TRY(cudaGetLastError());
      count_launch(dev);
      prm.target_logits = (const float*)p->layer_buf.p;
    }
  }
  prm.k = 0;
  prm.vocab = V;
  const int32_t* host = nullptr;
  rc = launch_selection(p, prm, n, a->sampler, a->mode, &host);
  if (rc) return rc;
  for (int i = 0; i < n; i++) a->tokens[i] = host[(size_t)n + i];
  return RELUX_OK;
}

}  // namespace relux
