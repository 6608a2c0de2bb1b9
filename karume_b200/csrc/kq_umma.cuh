// Helpers shared by the tcgen05 GEMM kernels (kq_qgemm_i4.cu, kq_qgemm_exact.cu): mbarriers with
// bounded waits, shared-memory matrix descriptors for the K-major 128-byte-swizzled layout, the
// kind::f16 MMA with bf16 operands, and the swizzled tile addressing.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace kq {
namespace umma {

constexpr uint32_t kWaitLimit = 1u << 24;

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}

// Bounded wait.  Returns false (at once, if another thread already gave up) when the
// barrier did not flip in time; the caller keeps going without blocking.
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                             int code) {
  for (uint32_t spins = 0; spins < kWaitLimit; ++spins) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spins & 1023u) == 1023u && *abort_flag) return false;
  }
  *abort_flag = 1;
  *reinterpret_cast<volatile int*>(status) = code;
  return false;
}

// K-major, 128-byte swizzle: rows are 128 B, groups of 8 rows are 1024 B apart (SBO),
// descriptor version 1 (Blackwell), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
         (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
         (static_cast<uint64_t>(2) << 61);
}

// kind::f16 instruction descriptor: f32 accumulate, bf16 A and B, both K-major, M x N.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t mma_m, uint32_t mma_n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((mma_n >> 3) << 17) | ((mma_m >> 4) << 24);
}

// ---- CTA pairs (cta_group::2): one MMA spans the two CTAs of a cluster -------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the address of this CTA's shared-memory location `addr` as seen in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Arrives on a barrier of either CTA of the pair.  What such an arrival hands over is read by the
// tensor core (a tile behind fence.proxy.async, an accumulator behind tcgen05.fence), never by a
// load of the other CTA's threads, so the default CTA-scope release is enough; a cluster-scope one
// waits for the thread's whole memory traffic (500 - 1500 clocks per arrival beside running copies).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// One lane of a warp, the same one every time.  What a single thread has to do below is a predicated
// instruction of a converged warp, never a branch: in a divergent lane-0 region the barrier tests and
// MMA issues took two to three times as long (700 - 850 clocks a k-step whatever its width).
__device__ __forceinline__ uint32_t elect_lane() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
// Descriptors by their low words (address, leading offset); the high word is the layout's constant.
constexpr uint32_t kDescHigh = (1024u >> 4) | (1u << 14) | (2u << 29);
// bf16, M 128 x N in one CTA; or M 256 (128 rows per CTA) x N: A and D are each CTA's own rows, B is read half from each.
template <bool kAccumulate>
__device__ __forceinline__ void umma_bf16_single(uint32_t leader, uint32_t tmem_d, uint32_t desc_a, uint32_t desc_b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(desc_a), "r"(desc_b), "r"(idesc), "n"(kAccumulate ? 1 : 0), "r"(kDescHigh), "r"(leader) : "memory");
}
template <bool kAccumulate>
__device__ __forceinline__ void umma_bf16_pair(uint32_t leader, uint32_t tmem_d, uint32_t desc_a, uint32_t desc_b, uint32_t idesc) {
  asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}"
               ::"r"(tmem_d), "r"(desc_a), "r"(desc_b), "r"(idesc), "n"(kAccumulate ? 1 : 0), "r"(kDescHigh), "r"(leader) : "memory");
}
// arrives on the barrier at this address in BOTH CTAs of the pair (bits of `ctas`: their cluster ranks) once the MMAs issued so far are done
__device__ __forceinline__ void commit_both(uint32_t leader, uint32_t bar, uint32_t ctas = 3u) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
               "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
               ::"r"(bar), "h"(static_cast<uint16_t>(ctas)), "r"(leader) : "memory");
}
__device__ __forceinline__ void commit_one(uint32_t leader, uint32_t bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
               ::"r"(bar), "r"(leader) : "memory");
}

// 8 nibbles of one 32-bit word -> 8 bf16 (16 bytes, k ascending), each
// RNE_bf16(fround((u - 8) * s)).  (word & (0xF << 4e)) | 0x4B000000 is the float
// 2^23 + u * 16^e exactly; subtracting 2^23 + 8 * 16^e leaves (u - 8) * 16^e exactly, and
// the power of sixteen is taken out of the scale (exact), so the one rounding of the
// multiply is the reference's.
__device__ __forceinline__ uint4 dequant8_bf16(uint32_t word, float s) {
  const float s1 = s * 0.0625f, s2 = s * 0.00390625f, s3 = s * 0.000244140625f;
  const uint32_t hi = word >> 16;
  float v[8];
  v[0] = (__uint_as_float((word & 0x000Fu) | 0x4B000000u) - 8388616.0f) * s;
  v[1] = (__uint_as_float((word & 0x00F0u) | 0x4B000000u) - 8388736.0f) * s1;
  v[2] = (__uint_as_float((word & 0x0F00u) | 0x4B000000u) - 8390656.0f) * s2;
  v[3] = (__uint_as_float((word & 0xF000u) | 0x4B000000u) - 8421376.0f) * s3;
  v[4] = (__uint_as_float((hi & 0x000Fu) | 0x4B000000u) - 8388616.0f) * s;
  v[5] = (__uint_as_float((hi & 0x00F0u) | 0x4B000000u) - 8388736.0f) * s1;
  v[6] = (__uint_as_float((hi & 0x0F00u) | 0x4B000000u) - 8390656.0f) * s2;
  v[7] = (__uint_as_float((hi & 0xF000u) | 0x4B000000u) - 8421376.0f) * s3;
  uint4 out;
  __nv_bfloat162 p;
  p = __floats2bfloat162_rn(v[0], v[1]); out.x = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(v[2], v[3]); out.y = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(v[4], v[5]); out.z = *reinterpret_cast<uint32_t*>(&p);
  p = __floats2bfloat162_rn(v[6], v[7]); out.w = *reinterpret_cast<uint32_t*>(&p);
  return out;
}

__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// byte offset of 16-byte piece c (0..7) of tile row r in the swizzled K-major layout
__device__ __forceinline__ uint32_t swz(uint32_t r, uint32_t c) { return r * 128u + ((c ^ (r & 7u)) << 4); }

}  // namespace umma
}  // namespace kq
