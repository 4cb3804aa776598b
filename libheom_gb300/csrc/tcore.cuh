// PTX wrappers of the 16-bit tensor-core kernels (the learned closure's and its
// GEMMs, BF16; k_rhs_split, FP16): descriptors and issue of tcgen05.mma
// (kind::f16, FP32 accumulators in tensor memory), tensor-memory loads, bulk
// copies and bounded mbarrier waits.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace heomgb {

__device__ __forceinline__ uint32_t s_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// One lane of a converged warp.  The MMAs of a loop belong in a branch on it:
// the compiler then knows that a single thread issues them and keeps their
// descriptors in uniform registers (measured: 48 cycles per MMA of 128 x 64 x
// 16, the rate of the operand reads; 115-160 behind `threadIdx.x == 0`).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n .reg .pred P;\n elect.sync _|P, 0xffffffff;\n selp.b32 %0, 1, 0, P;\n}\n" : "=r"(e));
  return e != 0;
}

// shared-memory matrix descriptor without swizzle (8-row x 16-byte core
// matrices).  K-major operand: lbo = the K-adjacent core matrix, sbo = the
// next 8 rows.  MN-major operand (8 k x 16 bytes of M or N): sbo = the next 8
// of M or N, lbo = the next 8 k.
__device__ __forceinline__ uint64_t g_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return static_cast<uint64_t>((saddr >> 4) & 0x3FFF) | (static_cast<uint64_t>((lbo >> 4) & 0x3FFF) << 16) |
         (static_cast<uint64_t>((sbo >> 4) & 0x3FFF) << 32) | (static_cast<uint64_t>(1) << 46);
}

// instruction descriptor: D FP32, A and B BF16, M = 128, N = n; a_mn, b_mn = 1: that operand is MN-major
__device__ __forceinline__ uint32_t g_idesc(int n, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_mn) << 15) | (static_cast<uint32_t>(b_mn) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (8u << 24);
}

__device__ __forceinline__ void g_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, int acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void g_commit(uint64_t* mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(s_addr(mbar)));
}

// bounded wait for phase `parity` of an mbarrier; 1 when it completed
__device__ __forceinline__ uint32_t g_wait(uint64_t* mbar, uint32_t parity) {
  uint32_t done = 0;
  for (int it = 0; it < (1 << 24) && !done; ++it) {
    asm volatile(
        "{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n selp.b32 %0, 1, 0, q;\n}\n"
        : "=r"(done)
        : "r"(s_addr(mbar)), "r"(parity)
        : "memory");
  }
  return done;
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(s_addr(mbar)) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ void expect_bytes(uint64_t* mbar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(s_addr(mbar)), "r"(bytes) : "memory");
}
// `bytes` (a multiple of 16, both addresses 16-byte aligned) from global to
// shared memory, counted on mbar
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   s_addr(dst)),
               "l"(src), "r"(bytes), "r"(s_addr(mbar))
               : "memory");
}

__device__ __forceinline__ void g_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}

// 16 columns
__device__ __forceinline__ void g_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(s_addr(slot)), "r"(cols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(cols));
}

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

// ------------------------------------------------------------------ packed operands
// The closure kernels compute transposed products D^T = W act^T: the outputs
// run along the tensor-memory lanes (M, tiles of 128) and the rows of a CTA's
// tile along the columns (N, any multiple of 16), so a tile can be as small
// as the number of SMs asks for.
//
// W: BF16, `rows` outputs (padded to 128) by k inputs (padded to 32, zeros), K
// in chunks of 32: a chunk = [rows / 8][4][8 rows][8 k] core matrices (K-major,
// lbo 128, sbo 512), contiguous, so one bulk copy brings it in.
//
// act: [columns / 8][rows of the tile / 8][8 columns][8 rows]: the MN-major
// operand of the product over columns (sbo 128, lbo = 16 x rows bytes) and the
// K-major operand of the product over rows (the weight gradients).
constexpr int kChunkK = 32;
__host__ __device__ __forceinline__ int pack_rows(int r) { return (r + 127) / 128 * 128; }
__host__ __device__ __forceinline__ int pack_k(int k) { return (k + kChunkK - 1) / kChunkK * kChunkK; }
__host__ __device__ __forceinline__ size_t pack_index(int rows_pad, int r, int k) {
  return ((static_cast<size_t>(k >> 5) * (rows_pad >> 3) + (r >> 3)) * 4 + ((k >> 3) & 3)) * 64 + (r & 7) * 8 + (k & 7);
}

// The weight chunks that a CTA consumes, in order: up to six operands one
// after another through a ring of 16 KB slots.  One thread of a warp of its own
// (the producer) copies them as slots come free; the thread that issues the
// MMAs waits for a chunk, issues, and hands the slot back with a commit.  Every
// wait is bounded: one that runs out ends the thread's part, and the CTA
// reports it (the producer lets its copies in flight land before it leaves).
template <int SLOTS>
struct WeightRing {
  static_assert((SLOTS & (SLOTS - 1)) == 0, "a power of two");
  unsigned char* ring;
  uint64_t* full;   // SLOTS: the copy has landed
  uint64_t* empty;  // SLOTS: the MMAs that read it have completed
  __device__ __forceinline__ WeightRing(unsigned char* r, uint64_t* bars) : ring(r), full(bars), empty(bars + SLOTS) {}
  __device__ __forceinline__ void init() const {
    for (int i = 0; i < 2 * SLOTS; ++i) mbar_init(full + i);
  }
  // producer: all chunks of one operand; `n` counts the chunks copied so far
  __device__ __forceinline__ bool copy(const void* w, int rows_pad, int k_pad, int& n) const {
    const uint32_t bytes = static_cast<uint32_t>(rows_pad) * kChunkK * 2;
    const unsigned char* src = static_cast<const unsigned char*>(w);
    for (int c = 0; c < k_pad / kChunkK; ++c, ++n, src += bytes) {
      const int s = n & (SLOTS - 1);
      if (n >= SLOTS && !g_wait(empty + s, static_cast<uint32_t>(n / SLOTS - 1) & 1u)) return false;
      expect_bytes(full + s, bytes);
      bulk_load(ring + s * 16384, src, bytes, full + s);
    }
    return true;
  }
  __device__ __forceinline__ void drain(int n) const {
    for (int c = n > SLOTS ? n - SLOTS : 0; c < n; ++c)
      g_wait(full + (c & (SLOTS - 1)), static_cast<uint32_t>(c / SLOTS) & 1u);
  }
  // D^T (m_tiles x 128 lanes, n columns each, tensor memory) = the next operand
  // (n_chunks chunks) x act^T; `taken` chunks were consumed before
  __device__ __forceinline__ bool layer(uint32_t act, int n, int m_tiles, int n_chunks, uint32_t tmem,
                                        int taken) const {
    const uint32_t idesc = g_idesc(n, 0, 1), kg = static_cast<uint32_t>(n) * 16u;
    const uint64_t da = g_desc(s_addr(ring), 128, 512);  // + (bytes >> 4) moves its start
    uint64_t db = g_desc(act, kg, 128);
    for (int c = 0; c < n_chunks; ++c, ++taken) {
      const int s = taken & (SLOTS - 1);
      if (!g_wait(full + s, static_cast<uint32_t>(taken / SLOTS) & 1u)) return false;
      const uint64_t w = da + static_cast<uint64_t>(s * (16384 >> 4));
      for (int m = 0; m < m_tiles; ++m) {
        g_mma(tmem + m * n, w + m * (8192 >> 4), db, idesc, c > 0 ? 1 : 0);
        g_mma(tmem + m * n, w + (m * 8192 + 256) / 16, db + (2 * kg >> 4), idesc, 1);
      }
      g_commit(empty + s);
      db += 4 * kg >> 4;
    }
    return true;
  }
};

}  // namespace heomgb
