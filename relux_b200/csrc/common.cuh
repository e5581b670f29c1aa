// Shared device/host helpers for librelux_cuda (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "relux_cuda.h"

namespace relux {

// ---------------------------------------------------------------------------------------------
// bf16 <-> f32 with the reference's exact bit rule (internal/transformer/dtype_convert.go:15-24):
// u += 0x7FFF + ((u >> 16) & 1); u >>= 16.  No NaN special case, so results match the reference
// bit for bit on every input, unlike __float2bfloat16_rn which canonicalises NaN.
// ---------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint16_t bf16_bits_from_f32(float x) {
#ifdef __CUDA_ARCH__
  uint32_t u = __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
#endif
  u += 0x7FFFu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}
__device__ __forceinline__ float f32_from_bf16_bits(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  return (uint32_t)bf16_bits_from_f32(lo) | ((uint32_t)bf16_bits_from_f32(hi) << 16);
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ uint32_t round_bf16x2(float lo, float hi) {   // to nearest, by the conversion instruction (pack_bf16x2: the reference's rule)
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&b);
}

// fastexp32 of internal/transformer/mha.go:823-833 with its operations kept unfused.
__device__ __forceinline__ float fastexp32_ref(float x) {
  if (x < -87.0f) return 0.0f;
  if (x > 87.0f) return __uint_as_float(0x7F800000u);
  float t = __fmul_rn(12102203.0f, x);
  t = __fadd_rn(t, 1064948224.0f);
  return __uint_as_float((uint32_t)__float2int_rz(t));
}

// ---------------------------------------------------------------------------------------------
// Device status word: kernels record the first problem they meet and carry on without faulting.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void set_status(int32_t* status, int32_t code) {
  if (status) atomicCAS(status, 0, code);
}

// Resolves (sequence, token position) to the element offset of the row's page inside one layer.
// Returns false (and records RELUX_ERR_BAD_PAGE) when the table holds an id outside the pool.
__device__ __forceinline__ bool page_of(const int32_t* __restrict__ table, int32_t table_stride, int32_t seq,
                                        int32_t page_slot, int32_t num_pages, int32_t* status, int32_t* page_out) {
  int32_t pg = table[(size_t)seq * table_stride + page_slot];
  if (pg < 0 || pg >= num_pages) {
    set_status(status, RELUX_ERR_BAD_PAGE);
    return false;
  }
  *page_out = pg;
  return true;
}

// Element offset of (token-in-page, column) inside one MLA page.
//   blocked (page_tokens = 64 and row width a multiple of 64): the page is stored as
//     [row_width / 64 column blocks][64 tokens][64 columns], so each 64 x 64 tile a TMA box fetches is one
//     contiguous 8 KB run of HBM instead of 64 pieces of 128 bytes 1152 bytes apart;
//   otherwise token-major [page_tokens][row_width].
// A vector of 8 consecutive columns starting at a multiple of 8 never straddles a block.
__device__ __forceinline__ size_t mla_page_off(bool blocked, int page_tokens, int row_width, int tok, int col) {
  return blocked ? ((size_t)(col >> 6) * page_tokens + tok) * 64 + (col & 63) : (size_t)tok * row_width + col;
}

// ---------------------------------------------------------------------------------------------
// PTX wrappers: shared-memory addresses, mbarrier with bounded waits, TMA, ldmatrix, mma.sync.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Every wait is bounded: after kSpinLimit failed polls the caller gets `false`, records
// RELUX_ERR_TIMEOUT and leaves its loop, so a protocol bug cannot hang the GPU.
constexpr uint32_t kSpinLimit = 4u * 1000u * 1000u;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kSpinLimit; i++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (i > 64) __nanosleep(32);
  }
  return false;
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 2-D tiled TMA load global -> shared (no multicast), completion on an mbarrier of this CTA.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int32_t x, int32_t y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// The same with an L2 eviction priority: evict_first for what is read once and streams past everything else.
__device__ __forceinline__ void tma_load_2d_hint(void* smem_dst, const CUtensorMap* map, int32_t x, int32_t y, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t make_evict_first_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t make_evict_normal_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// A box of a 5-D map (a reordered view of a matrix).
__device__ __forceinline__ void tma_load_5d(void* smem_dst, const CUtensorMap* map, int32_t x, int32_t y, int32_t z, int32_t u, int32_t w, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(
          smem_u32(smem_dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(u), "r"(w)
      : "memory");
}
// 2-D tiled TMA store shared -> global of one box (bulk async-group completion).  The shared tile must have been made
// visible to the async proxy (fence_proxy_async) by the threads that wrote it.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int32_t x, int32_t y, const void* smem_src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, int32_t x, int32_t y, int32_t z, int32_t w, const void* smem_src) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(smem_u32(smem_src)), "r"(x),
               "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// All committed stores of this thread have finished READING their shared tiles (the tiles may be written again).
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// All committed stores of this thread are complete.
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Programmatic dependent launch.  A kernel launched with the stream-serialization attribute may be scheduled while the
// kernel before it in the stream still runs; chain_wait() returns once that kernel has completed and its writes are
// visible.  chain_release() lets the kernel after this one be scheduled.  Both are no-ops in a plain launch.  The rules of a
// chain (who writes these launches, who may read before the wait) stand at launch_chained in internal.h.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Device time of a launch without event records between it and its neighbours (two records cost the stream 2-4 us per
// call and keep a chained launch from starting early): every block stamps its first and last moment into the call's slot.
// `begin_inv` holds the complement, so that both words are maxima over zero-filled memory; the first block clears the
// slot of the call after this one (whose stamps come after its chain_wait()).
struct TimeSlot {
  unsigned long long begin_inv, end;
};
struct TimeStamp {
  TimeSlot* slot;    // nullptr: this call is not timed
  TimeSlot* clear;
};
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// By one thread per block, after chain_wait().
__device__ __forceinline__ void stamp_begin(const TimeStamp& ts) {
  if (!ts.slot) return;
  atomicMax(&ts.slot->begin_inv, ~global_ns());
  if ((blockIdx.x | blockIdx.y | blockIdx.z) == 0) ts.clear->begin_inv = ts.clear->end = 0ull;
}
__device__ __forceinline__ void stamp_end(const TimeStamp& ts) {
  if (ts.slot) atomicMax(&ts.slot->end, global_ns());
}

// By every thread that wrote with ordinary stores what a later launch of the chain reads by TMA (cached rows, bf16 activations,
// queries), behind its last store: TMA reads through the async proxy, and it is nowhere stated that chain_wait() alone orders that
// proxy after another launch's generic writes, as the end of a plain launch does.  On this side because nothing is in flight
// here; behind the readers' wait the same fence waited for their weights (67.0 -> 69.4 us of a GQA layer step).
__device__ __forceinline__ void fence_chained_writes() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// What the launch before this one may have written after this launch began (lengths, plans, activations, partial results): read
// from L2, so that a line which another block of this SM brought into L1 meanwhile is not taken for it.  Never by __ldg, nor
// through a const __restrict__ pointer without this: such loads may become ld.global.nc, which wants data that nobody writes
// while the kernel exists, and which the compiler may move ahead of chain_wait().
template <typename T>
__device__ __forceinline__ T load_chained(const T* p) { return __ldcg(p); }

// Stores with an L2 eviction priority: evict_last for what a later launch reads while other data streams through L2.
__device__ __forceinline__ uint64_t make_evict_last_policy() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void store_hint(void* p, const uint4& v, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.v4.b32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(__cvta_generic_to_global(p)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w),
               "l"(policy)
               : "memory");
}
// A store by a predicate, not behind a branch.
__device__ __forceinline__ void store_if(float* p, float v, bool there) {
  asm volatile("{\n\t.reg .pred t;\n\tsetp.ne.s32 t, %2, 0;\n\t@t st.global.f32 [%0], %1;\n\t}" ::"l"(__cvta_generic_to_global(p)), "f"(v), "r"((int)there) : "memory");
}
__device__ __forceinline__ void store_if(uint16_t* p, uint16_t v, bool there) {
  asm volatile("{\n\t.reg .pred t;\n\tsetp.ne.s32 t, %2, 0;\n\t@t st.global.u16 [%0], %1;\n\t}" ::"l"(__cvta_generic_to_global(p)), "h"(v), "r"((int)there) : "memory");
}
__device__ __forceinline__ void store_hint(float* p, float v, uint64_t policy) {
  asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(__cvta_generic_to_global(p)), "f"(v), "l"(policy) : "memory");
}

// Brings [p, p + bytes) into L2 (both multiples of 16).
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// D(16x8,f32) += A(16x16,bf16,row) * B(16x8,bf16,col)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Byte offset of element (row, col16B chunk) inside a tile whose rows are 128 bytes and which was
// written by TMA with CU_TENSOR_MAP_SWIZZLE_128B: the 16-byte chunk index is XORed with (row & 7).
__device__ __forceinline__ uint32_t swz128(uint32_t row, uint32_t chunk16) { return row * 128u + ((chunk16 ^ (row & 7u)) << 4); }
// The same for rows of 64 bytes and CU_TENSOR_MAP_SWIZZLE_64B.
__device__ __forceinline__ uint32_t swz64(uint32_t row, uint32_t chunk16) { return row * 64u + ((chunk16 ^ ((row >> 1) & 3u)) << 4); }

}  // namespace relux
