// qgemm_exact — the linear for many activation rows (m > 16) whose weights enter the tensor
// core as EXACT small integers:  out[m, n] = x[m, k] . W[n, k]^T + bias.
//
// Replaces the reference's large-M linear variants that compute in f32
// (linear:v2:f32:reg64x32r4x4w8 and reg128x128r8x8w16 —
// packages/runtime/src/kernels/gemm-geometry.ts:243-267) for every packed storage, and its
// integer-dot GEMMs (packages/runtime/src/kernels/linear-i8a8.ts:21-72).
//
// A stored int4 / int8 weight is an integer q of at most 8 bits, exact in binary16 and in bf16, so
// nothing has to be rounded and nothing has to be multiplied by a scale on its way to the tensor core:
//     y[m, n] = sum_groups s[n, g] * ( sum_{k in g} x[m, k] * q[n, k] )
// The inner sum is a short MMA chain into a tensor-memory accumulator; every group the "drain"
// warps read that accumulator and add it, times the group's scale, to f32 sums they keep in
// registers.  An activation is carried exactly: a binary16 or bf16 one as it is, an int8 one of the
// integer-dot form as binary16, an f32 one as three bf16 parts (3 x 8 = 24 bits, each with f32's
// exponents).  Only f32 ones on tiled int8 weights are two binary16 parts of the row's power-of-two
// pre-scaled values, as in the int8 GEMV: 22 bits, down to 2^-37 of the row's largest value.  So
//   * binary16 and bf16 activations cost ONE product, f32 ones three or two, where splitting both
//     operands costs three for 16 bits.  (Two binary16 parts everywhere would lose what an f32
//     multiply-add keeps: a small value of a row, on a channel without weight at the large ones.
//     The third part costs 333 x 1536 -> 8960 int4 32.6 us against 32.1, 1024 x 4096 -> 6144 129
//     against 118; 257 x 1536 -> 8960 int8 29 against 25.)
//   * an accumulator chain is at most one group long, and at most 64 to 256 k (chain_of), so the tensor
//     core's f32 accumulation, which truncates, never gets the chance to drift;
//   * the integer-dot form of int4 weights is the same kernel: its per-group sums are integers
//     below 2^24, exact in the f32 accumulator, and the contract's one fma per group in
//     ascending order IS the drain (bit-identical).  Int8 weights with int8 activations run on
//     kind::i8 with an int32 accumulator over the whole of k.
//
// The weights are the M side (256 output channels per CTA pair, 128 per CTA), the activation
// rows the N side (NT <= 256 of them), so a lane of the accumulator is one output channel: its
// scale and bias are per-lane scalars and a store instruction writes 32 consecutive outputs.
//
//   warps 0-7    drain: tcgen05.ld, one fma per sum, then the epilogue (K slices of one tile that form a cluster
//                add their sums over its shared memory first, in slice order)
//   warps 8-11   producers: raw packed weights (shared memory) -> integers in the K-major,
//                128-byte-swizzled tile the MMA reads.  Shared memory to shared memory only: a
//                global load still in flight when a thread runs its proxy fence would hold the
//                fence, and with it the stage, for a trip to memory.
//   warp 12      starts every copy: the activation tile (tensor map), the raw weights (bulk)
//   warp 13      tensor memory; in the first CTA of the pair one thread issues the MMAs
//                (cta_group::2: the pair shares the activation tile, half from each CTA)
//   warps 14-15  the group scales, a few chains ahead, as f32 into shared memory
//
// A gate and its up projection share a tile (64 channels of each per CTA), so that silu(gate) * up is the epilogue:
// 333 rows of 1536 -> 2 x 8960, norm included, 66.7 us with the gate in a kernel of its own, 61.4 so.
// Register split (setmaxnreg): 2 x 128 x 184 + 2 x 128 x 72 = 512 x 128.
//
// Every mbarrier wait is bounded; a wait that gives up sets a status word and a CTA-wide abort
// flag that makes all later waits return at once, so tensor memory is always released.  Copies and
// producers whose wait gave up leave their stage alone: an arrival on a barrier whose phase has all
// its arrivals and still waits for bytes is undefined.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "kq_common.cuh"
#include "kq_exact_geometry.h"
#include "kq_gemv_core.cuh"
#include "kq_internal.h"
#include "kq_umma.cuh"

namespace kq {
namespace {

using namespace umma;
using namespace exact;

enum WeightKind : int { kI4Tiled = 0, kI4Rows = 1, kI8Tiled = 2, kI8Rows = 3 };
template <int kMath>
constexpr bool kIsBf = kMath == kBf1 || kMath == kBf3;

constexpr int kDrainWarps = 8, kProdWarps = 4, kCopyWarp = 12, kMmaWarp = 13, kScaleWarp = 14, kExThreads = 512;
constexpr uint32_t kRows = 128;                 // output channels per CTA
constexpr uint32_t kATile = kRows * 128;        // 16 KB: 128 rows x 128 bytes of k
constexpr uint32_t kMaxStages = 8;
constexpr uint32_t kSmemLimit = 227 * 1024;
constexpr uint32_t kScaleBatch = 8;             // accumulator chains per slot of the scale ring (two slots)
constexpr uint32_t kOutCols = 8;                // columns a drain warp hands to its epilogue at a time
constexpr uint32_t kTailScales = 320, kTailRows = kTailScales + 2 * kScaleBatch * kRows * 4;
// Barriers, the scale ring, the row factors; where a pair takes several tiles each drain warp has row factors of its own
// (the warps of a column half may be in different tiles), and finished sums on their way out.  (A copy for each warp in
// every form cost binary16 tiles of 256 rows one of six stages: 1225 x 2816 -> 7424 group 128 69.7 us, 65.1 without.)
__host__ __device__ constexpr uint32_t tail_out(uint32_t nt) { return kTailRows + kDrainWarps * nt / 2 * 4; }
__host__ __device__ constexpr uint32_t smem_tail(bool multi, uint32_t nt) { return multi ? tail_out(nt) + kDrainWarps * kOutCols * 128 : kTailRows + nt * 4; }
constexpr uint32_t kMaxChain = 1024;            // k per accumulator chain: whole groups of the integer-dot form

struct ExTarget {
  const uint8_t* w;
  const void* scale;      // rows layouts: [n, k / group]; int8: [n]; tiled int4: inside the chunks
  const float* bias;
  float* out;
  const float* residual;  // null, or [m, n] added after the bias (may alias out)
  uint32_t n;
  uint32_t pair0;         // first column pair (256 channels) of this weight
};

struct ExParams {
  ExTarget t[kMaxMulti];
  uint32_t count;
  uint32_t pairs, m_tiles; // column pairs of all weights, row tiles
  uint32_t multi, resident; // more tiles than pairs the device holds: each of `resident` takes several
  uint32_t swiglu;         // one output, silu(gate) * up: t[0] is the gate, t[1] up, and a CTA's 128 rows are 64 channels of each
  uint32_t m, k;
  uint32_t ksteps;         // k-steps of 128 bytes (64 binary16 or 128 int8 values)
  uint32_t nt;             // activation rows per tile, a multiple of 32
  uint32_t drain16;        // k16 slices per accumulator chain
  uint32_t drains_per_group_shift;  // accumulator chains per scale group, log2 (groups longer than a chain)
  uint32_t groups;         // scale groups per row
  uint32_t scale_f16;
  uint32_t stages, stage_bytes, raw_off, raw_bytes, raw_box;
  const float* row_scale;  // [m]: undoes the pre-scale (2^-e), or the activation scale of the integer-dot form; null: 1
  uint32_t splits, ksteps_per_split;
  uint32_t cluster_splits; // 1, or = splits: the K slices of a tile are one cluster and add their sums over its shared memory
  float* partial;          // [splits][m][n of all weights] raw sums when splits > 1
  uint32_t n_total;
  int* status;
};

__device__ __forceinline__ float load_scale_dyn(const void* base, size_t index, uint32_t f16) {
  return f16 ? __half2float(reinterpret_cast<const __half*>(base)[index]) : reinterpret_cast<const float*>(base)[index];
}

// ---- integers -> binary16 or bf16 ------------------------------------------------------------
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) { return (a & mask) | bits; }

// 8 nibbles u (k ascending) -> 8 binary16 values u - 8, exact.
__device__ __forceinline__ uint4 nibbles_to_half(uint32_t w) {
  __half2 h[4];
  nibble_pairs(w, h);
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) r[i] = *reinterpret_cast<const uint32_t*>(&h[i]);
  return make_uint4(__byte_perm(r[0], r[1], 0x5410), __byte_perm(r[2], r[3], 0x5410), __byte_perm(r[0], r[1], 0x7632),
                    __byte_perm(r[2], r[3], 0x7632));
}
// ... -> 8 bf16 values u - 8, exact.  bf16 has seven bits behind the exponent of 128: 128 + u holds a
// nibble in its lowest place only, so all four pairs are shifted there.
__device__ __forceinline__ uint4 nibbles_to_bf16(uint32_t w) {
  const __nv_bfloat162 k136 = __bfloat162bfloat162(__ushort_as_bfloat16(0x4308));
  uint32_t r[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t v = and_or(w >> (4 * i), 0x000F000Fu, 0x43004300u);
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&v), k136);
    r[i] = *reinterpret_cast<const uint32_t*>(&d);
  }
  return make_uint4(__byte_perm(r[0], r[1], 0x5410), __byte_perm(r[2], r[3], 0x5410), __byte_perm(r[0], r[1], 0x7632),
                    __byte_perm(r[2], r[3], 0x7632));
}
template <int kMath>
__device__ __forceinline__ uint4 nibbles_to_operand(uint32_t w) {
  if constexpr (kIsBf<kMath>) return nibbles_to_bf16(w);
  else return nibbles_to_half(w);
}

// 4 bytes q + 128 -> 4 binary16 values q, exact.
__device__ __forceinline__ uint2 bytes_to_half(uint32_t w) {
  __half2 h[2];
  byte_pairs(w, h);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&h[0]), *reinterpret_cast<const uint32_t*>(&h[1]));
}
// ... -> 4 bf16 values q, exact.  With b = q + 128 under the exponent of 128 the seven low bits of b read as
// 128 + (b & 127); the top bit, which would reach into the exponent, is taken out and says what to subtract:
// 128 where it is set (q = b & 127), 256 = the bits of 128 with that one flipped where it is not.
__device__ __forceinline__ uint2 bytes_to_bf16(uint32_t w) {
  uint32_t r[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t t = __byte_perm(w, 0x43434343u, i ? 0x4342 : 0x4140);
    const uint32_t low = t & 0xFF7FFF7Fu, off = (t & 0xFF80FF80u) ^ 0x00800080u;
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&low), *reinterpret_cast<const __nv_bfloat162*>(&off));
    r[i] = *reinterpret_cast<const uint32_t*>(&d);
  }
  return make_uint2(r[0], r[1]);
}
template <int kMath>
__device__ __forceinline__ uint2 bytes_to_operand(uint32_t w) {
  if constexpr (kIsBf<kMath>) return bytes_to_bf16(w);
  else return bytes_to_half(w);
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
// of another CTA of the cluster (an address of map_to_cta)
__device__ __forceinline__ uint32_t lds32_cluster(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts64(uint32_t addr, uint2 v) {
  asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// ---- tensor memory ---------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld16_begin(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Registers of a finished load: nothing that uses them may be scheduled in front of the wait.
__device__ __forceinline__ void tmem_ld16_done(uint32_t (&v)[16]) {
  asm volatile("" : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                    "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  tmem_ld16_begin(taddr, v);
  tmem_ld_wait();
  tmem_ld16_done(v);
}

// kind::f16 with binary16 or bf16 operands / kind::i8 with signed operands; f32 / s32 accumulate, M 256
template <int kMath>
__host__ __device__ constexpr uint32_t exact_idesc(uint32_t nt) {
  return kIsBf<kMath> ? umma_idesc(256, nt)
                      : (kMath == kInt8 ? ((2u << 4) | (1u << 7) | (1u << 10)) : (1u << 4)) | ((nt >> 3) << 17) | ((256u >> 4) << 24);
}
template <int kMath, bool kAccumulate>
__device__ __forceinline__ void mma_pair(uint32_t leader, uint32_t tmem_d, uint32_t desc_a, uint32_t desc_b, uint32_t idesc) {
  if constexpr (kMath == kInt8)
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
                 "@q tcgen05.mma.cta_group::2.kind::i8 [%0], a, b, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(desc_a), "r"(desc_b), "r"(idesc), "n"(kAccumulate ? 1 : 0), "r"(kDescHigh), "r"(leader) : "memory");
  else
    asm volatile("{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
                 "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(desc_a), "r"(desc_b), "r"(idesc), "n"(kAccumulate ? 1 : 0), "r"(kDescHigh), "r"(leader) : "memory");
}
__device__ __forceinline__ void arrive_if(uint32_t leader, uint32_t cluster_bar) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q mbarrier.arrive.shared::cluster.b64 _, [%0];\n\t}"
               ::"r"(cluster_bar), "r"(leader) : "memory");
}

// ---- copies ---------------------------------------------------------------------------------
__device__ __forceinline__ void expect_tx(uint32_t leader, uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
               ::"r"(bar), "r"(bytes), "r"(leader) : "memory");
}
// reports to a barrier of either CTA of the pair
__device__ __forceinline__ void copy_tile_3d(uint32_t leader, uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t z, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n\t}"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar), "r"(leader) : "memory");
}
__device__ __forceinline__ void copy_tile_2d(uint32_t leader, uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}"
      ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar), "r"(leader) : "memory");
}

// Bytes of raw weights one 16-row block (tiled layouts) or one row (rows layouts) brings per k-step.
template <int kW, int kMath>
__host__ __device__ constexpr uint32_t raw_unit_bytes(uint32_t scale_f16) {
  return kW == kI4Tiled ? kChunkWeightBytes + (scale_f16 ? 64u : 128u)
         : kW == kI4Rows ? 32u
         : kW == kI8Tiled ? (kMath == kInt8 ? 2048u : 1024u)
                          : (kMath == kInt8 ? 128u : 64u);
}

// Producer warps that convert a stage's weight tile together (each of them arrives on the stage's barrier).
template <int kMath>
__device__ __forceinline__ uint32_t stage_warps(uint32_t stages) {
  return parts_of(kMath) == 3 && stages < kProdWarps ? kProdWarps : 1u;
}

// What a launch does: a tile to a pair; K slices of a tile to a cluster; either, or a tile of a gate and its up projection;
// several tiles to a pair.  (Code that a launch does not run still costs it, in instructions fetched cold around those that
// it does: with the slices' in the plain form 24 x 9472 -> 4096 binary16 20.5 us, 20.0 without, 39 x 4736 -> 1920 bf16 14.4, 13.9.)
enum ExForm : int { kPlain, kSliced, kGate, kSeveral };

template <int kW, int kMath, int kForm>
__global__ void __launch_bounds__(kExThreads, 1)
qgemm_exact_kernel(const ExParams p, const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map0,
                   const __grid_constant__ CUtensorMap w_map1, const __grid_constant__ CUtensorMap w_map2,
                   const __grid_constant__ CUtensorMap w_map3) {
  constexpr bool kTiled = kW == kI4Tiled || kW == kI8Tiled;
  constexpr bool kGroupScales = kW == kI4Tiled || kW == kI4Rows;
  constexpr uint32_t kParts = parts_of(kMath);
  constexpr bool kMulti = kForm == kSeveral, kMayGate = kForm == kGate, kMaySlice = kForm == kSliced || kForm == kGate;
  static_assert(!kMulti || kMath == kInt8, "only sums that stay in tensor memory leave the drain warps time for another tile");
  const bool gated = kMayGate && p.swiglu != 0;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t raw_base = static_cast<uint32_t>(__cvta_generic_to_shared(smem_raw));
  const uint32_t tiles = (raw_base + 1023u) & ~1023u;
  const uint32_t bars = tiles + p.stages * p.stage_bytes;
  uint8_t* tail = smem_raw + (tiles - raw_base) + p.stages * p.stage_bytes;
  const uint32_t full = bars, empty = bars + kMaxStages * 8, rawfull = empty + kMaxStages * 8, dfull = rawfull + kMaxStages * 8,
                 dempty = dfull + 16, sfull = dempty + 16, sempty = sfull + 16;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(tail + 296);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 304);
  float* scale_ring = reinterpret_cast<float*>(tail + kTailScales);
  // a cluster is one pair, or the pairs of all K slices of a tile: ranks 2z and 2z + 1 are slice z
  const uint32_t cluster_rank = cluster_ctarank(), cta_rank = cluster_rank & 1u, pair_rank0 = cluster_rank & ~1u;
  // Tensor memory holds two sets of accumulators, the MMAs fill one while the drain reads the other.  A set is as
  // many chains as fit half of the 512 columns (one of 256 columns, two of 128, four of 64, eight of 32): a
  // hand-over costs about 390 clocks whatever it hands over (24 x 4096 -> 9472: 33 us with one chain of 32 columns each).
  const uint32_t acc_cols = p.nt <= 32 ? 32u : p.nt <= 64 ? 64u : p.nt <= 128 ? 128u : 256u, per_set = 256u / acc_cols;

  // kMulti (int8 x int8): a cluster of one pair takes tiles (column pair, row tile) in turn, and while the drain warps store
  // a tile's outputs, copies, producers and MMAs are at work on the next (4096 x 2048 -> 8192, 512 tiles on 74 pairs: 111 us
  // with a cluster per tile, 76 so).  Elsewhere a cluster has one tile: with sums in the drain warps' registers there is
  // nobody to drain the next one meanwhile (333 x 1536 -> 17920 f32 60 | 66, 1948 x 11264 -> 3088 binary16 group 16 475 | 553).
  const uint32_t tiles_all = p.pairs * p.m_tiles, tile0 = blockIdx.x >> 1, tile_step = gridDim.x >> 1;  // (kMulti)
  // (a weight's pointers are read from the parameters where they are used: kept in registers they would spill beside
  // the drain warps' sums)
  struct Tile { uint32_t wi, n0, m0, z, ks_begin, ks_count; };  // weight, this CTA's first output channel, first row, K slice and its k-steps
  auto tile_at = [&](uint32_t t) {
    Tile r;
    const uint32_t mt = kMulti ? t / p.pairs : blockIdx.y, pair = kMulti ? t - mt * p.pairs : blockIdx.x >> 1;
    r.z = kMulti ? 0u : blockIdx.z;
    r.wi = 0;
    if (gated) {
      r.n0 = pair * kRows + cta_rank * (kRows / 2);
    } else {
#pragma unroll
      for (int i = 1; i < kMaxMulti; ++i)
        if (i < static_cast<int>(p.count) && pair >= p.t[i].pair0) r.wi = i;
      r.n0 = (pair - p.t[r.wi].pair0) * (2 * kRows) + cta_rank * kRows;
    }
    r.m0 = mt * p.nt;
    r.ks_begin = r.z * p.ksteps_per_split;
    r.ks_count = min(r.ks_begin + p.ksteps_per_split, p.ksteps) - r.ks_begin;
    return r;
  };

  const Tile tile_first = tile_at(tile0);  // (looked up here, in front of the wait for the launch before)

  if (warp == kMmaWarp) {
    if (lane == 0) {
      for (uint32_t s = 0; s < p.stages; ++s) {
        mbar_init(full + s * 8, 2 * stage_warps<kMath>(p.stages) + 1);  // the producer warps of each CTA; + the activation tiles' bytes
        mbar_init(empty + s * 8, 1);                  // one tcgen05.commit
        mbar_init(rawfull + s * 8, 1);                // the raw weights' bytes
      }
      for (uint32_t b = 0; b < 2; ++b) {
        mbar_init(dfull + b * 8, 1);
        mbar_init(dempty + b * 8, 2 * kDrainWarps);
        mbar_init(sfull + b * 8, 2);
        mbar_init(sempty + b * 8, kDrainWarps);
      }
      *abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bars + 296), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait_prior_grid();  // the converted activations come from the launch before
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync_all();  // barriers of both CTAs are initialised
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot_ptr;
  pdl_launch_dependents();

  const uint32_t leader = elect_lane();

  if (warp < kDrainWarps) {
    // ---------------- drain ----------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    const uint32_t quarter = warp & 3u, half = warp >> 2;
    const uint32_t cols = p.nt / 2, col0 = half * cols;  // this warp's share of the tile's activation rows
    const uint32_t taddr = tmem + ((quarter * 32u) << 16) + col0;
    // Finished sums leave through shared memory: the stores to `out` are then a short loop, where 128 unrolled copies
    // of them are 24 KB of instructions that every CTA fetches cold (13 us instead of 3 for 256 x 18944 outputs).  A
    // CTA's last tile parks them all in the stages, which are free then; before that, eight columns of a warp at a time.
    const uint32_t out_at = bars + tail_out(p.nt) + warp * (kOutCols * 128u) + lane * 4u;
    const uint32_t park = tiles + warp * (cols * 128u) + lane * 4u;
    float* row_factor = reinterpret_cast<float*>(tail + kTailRows) + (kMulti ? warp * cols : col0);
    // the factors of activation rows c, c + step, .. of this warp's columns
    auto row_factors = [&](uint32_t first_row, uint32_t c, uint32_t step) {
      for (; c < cols; c += step) row_factor[c] = p.row_scale != nullptr && first_row + c < p.m ? p.row_scale[first_row + c] : 1.0f;
    };
    if constexpr (!kMulti) {  // one tile: the four warps of a column half share them
      row_factors(blockIdx.y * p.nt + col0, quarter * 32u + lane, 128u);
      asm volatile("bar.sync %0, 128;" ::"r"(1u + half) : "memory");
    }
    uint32_t set = 0;  // accumulator sets so far, over all tiles
    uint32_t tile = tile0;
    do {
    const Tile at_tile = kMulti ? tile_at(tile) : tile_first;
    const uint32_t m0 = at_tile.m0, ks_count = at_tile.ks_count;
    // ---- a tile's columns [8 h, 8 h + 8) of this warp, at `from` in shared memory, to where they go: emit_gate, emit_tile ----
    // (what belongs to this thread's channel, or to its channel of the gate and of up, is read once a tile)
    struct Channel { float bias, up_bias, ws, up_ws; };
    auto channel = [&]() {
      Channel c = {0.0f, 0.0f, 1.0f, 1.0f};
      const ExTarget& tg = p.t[at_tile.wi];
      const uint32_t row = at_tile.n0 + (gated ? quarter & 1u : quarter) * 32u + lane;
      if (row < tg.n && p.splits == 1) {
        c.bias = tg.bias[row];
        if constexpr (!kGroupScales) c.ws = load_scale_dyn(tg.scale, row, p.scale_f16);
        if (gated) {
          c.up_bias = p.t[1].bias[row];
          if constexpr (!kGroupScales) c.up_ws = load_scale_dyn(p.t[1].scale, row, p.scale_f16);
        }
      }
      return c;
    };
    auto finished = [](uint32_t v, float rs, float ws, float bias) {
      if constexpr (kMath == kInt8) return fmaf(__int2float_rn(static_cast<int>(v)), __fmul_rn(rs, ws), bias);
      else if constexpr (kGroupScales) return fmaf(__uint_as_float(v), rs, bias);
      else return fmaf(__uint_as_float(v) * ws, rs, bias);
    };
    // silu(gate) * up of parked sums: warps 0 and 1 of a column half hold gate rows, 2 and 3 the same rows of up; each takes
    // half of the columns
    auto emit_gate = [&](uint32_t h, const Channel& ch, uint32_t from, uint32_t warp_bytes) {
      const uint32_t c0 = h * kOutCols, mm0 = m0 + col0 + c0;
      const uint32_t row = at_tile.n0 + (quarter & 1u) * 32u + lane, first = (quarter >> 1) * (kOutCols / 2);
      const uint32_t gate_at = from - (quarter >> 1) * 2u * warp_bytes, up_at = gate_at + 2u * warp_bytes;
      const bool live = row < p.t[0].n;
      float* dst = p.t[0].out + static_cast<size_t>(mm0 + first) * p.t[0].n + row;
      float gate[kOutCols / 2], up[kOutCols / 2];
#pragma unroll
      for (uint32_t i = 0; i < kOutCols / 2; ++i) {
        gate[i] = __uint_as_float(lds32(gate_at + (first + i) * 128u));
        up[i] = __uint_as_float(lds32(up_at + (first + i) * 128u));
      }
#pragma unroll
      for (uint32_t i = 0; i < kOutCols / 2; ++i) {
        const float rs = row_factor[c0 + first + i];
        if constexpr (!kGroupScales) {
          gate[i] *= ch.ws;
          up[i] *= ch.up_ws;
        }
        gate[i] = silu_mul(fmaf(gate[i], rs, ch.bias), fmaf(up[i], rs, ch.up_bias));
      }
#pragma unroll
      for (uint32_t i = 0; i < kOutCols / 2; ++i, dst += p.t[0].n)
        if (live && mm0 + first + i < p.m) *dst = gate[i];
    };
    // (kMulti: the loads of all columns first, one column at a time is one trip to shared memory after the other)
    auto emit_tile = [&](uint32_t h, const Channel& ch, uint32_t from) {
      const uint32_t c0 = h * kOutCols, mm0 = m0 + col0 + c0;
      const ExTarget& tg = p.t[at_tile.wi];
      const uint32_t row = at_tile.n0 + quarter * 32u + lane;  // this lane's output channel
      const bool row_live = row < tg.n;
      uint32_t v[kOutCols];
#pragma unroll
      for (uint32_t j = 0; j < kOutCols; ++j) v[j] = lds32(from + j * 128u);
      float* dst = tg.out + static_cast<size_t>(mm0) * tg.n + row;
#pragma unroll
      for (uint32_t j = 0; j < kOutCols; ++j, dst += tg.n)
        if (row_live && mm0 + j < p.m) *dst = finished(v[j], row_factor[c0 + j], ch.ws, ch.bias);
    };
    if constexpr (kMulti) {
      row_factors(m0 + col0, lane, 32u);
      __syncwarp();
    }
    const bool last_tile = !kMulti || tile + tile_step >= tiles_all;
    // parked sums: the same, all columns (without a gate column by column: 2 us less for 333 x 1536 -> 17920)
    auto emit_parked = [&]() {
      const Channel ch = channel();
      if constexpr (kMulti) {
#pragma unroll 1
        for (uint32_t h = 0; h * kOutCols < cols; ++h) emit_tile(h, ch, park + h * (kOutCols * 128u));
        return;
      }
      if (gated) {
        asm volatile("bar.sync %0, 128;" ::"r"(1u + half) : "memory");  // all warps of the column half have parked
#pragma unroll 1
        for (uint32_t h = 0; h * kOutCols < cols; ++h) emit_gate(h, ch, park + h * (kOutCols * 128u), cols * 128u);
        return;
      }
      const ExTarget& tg = p.t[at_tile.wi];
      const uint32_t row = at_tile.n0 + quarter * 32u + lane, mm0 = m0 + col0;
      const uint32_t live_cols = row < tg.n && mm0 < p.m ? min(cols, p.m - mm0) : 0u, n = tg.n;
      if (p.splits == 1) {
        float* dst = tg.out + static_cast<size_t>(mm0) * n + row;
        const float* res = tg.residual != nullptr ? tg.residual + static_cast<size_t>(mm0) * n + row : nullptr;
#pragma unroll 4
        for (uint32_t c = 0; c < live_cols; ++c) {
          float o = finished(lds32(park + c * 128u), row_factor[c], ch.ws, ch.bias);
          if (res != nullptr) {
            o = __fadd_rn(o, *res);
            res += n;
          }
          *dst = o;
          dst += n;
        }
      } else {
        uint32_t before = 0;
#pragma unroll
        for (int i = 0; i < kMaxMulti; ++i)
          if (static_cast<uint32_t>(i) < at_tile.wi) before += p.t[i].n;
        uint32_t* dst = reinterpret_cast<uint32_t*>(p.partial) + (static_cast<size_t>(at_tile.z) * p.m + mm0) * p.n_total + before + row;
#pragma unroll 4
        for (uint32_t c = 0; c < live_cols; ++c) {
          *dst = lds32(park + c * 128u);
          dst += p.n_total;
        }
      }
    };
    if constexpr (kMath == kInt8) {
      wait_bounded(dfull + (set & 1u) * 8, (set >> 1) & 1u, abort_flag, p.status, 23);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t at = taddr + (set & 1u) * kMaxNT;
      if (kMulti && !last_tile) {
        const Channel ch = channel();
#pragma unroll 1
        for (uint32_t b = 0; b * 16u < cols; ++b) {
          uint32_t v[16];
          tmem_ld16(at + b * 16u, v);
#pragma unroll
          for (uint32_t hh = 0; hh < 2; ++hh) {
#pragma unroll
            for (uint32_t j = 0; j < kOutCols; ++j) sts32(out_at + j * 128u, v[hh * kOutCols + j]);
            emit_tile(2 * b + hh, ch, out_at);
          }
        }
      } else {
#pragma unroll 1
        for (uint32_t b = 0; b * 16u < cols; ++b) {
          uint32_t v[16];
          tmem_ld16(at + b * 16u, v);
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) sts32(park + (b * 16u + j) * 128u, v[j]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      arrive_if(leader, map_to_cta(dempty, pair_rank0) + (set & 1u) * 8);
      ++set;
    } else {
      const uint32_t drains = (ks_count * 4 + p.drain16 - 1) / p.drain16;
      const uint32_t dempty_0 = map_to_cta(dempty, pair_rank0);
      const float* my_scale = scale_ring + quarter * 32u + lane;
      // kBatches x 16 columns per warp, a constant.  A chain of 256 columns takes 883 clocks from one to the next,
      // hand-over included (group 32, binary16: two of them are the k-step of 1,765; 690 at 192 columns, 504 at
      // 128); with a branch around every batch (a runtime width) it is 1,130, 1,043 and 728.
      auto drain_all = [&](auto batches) {
        constexpr int kBatches = decltype(batches)::value;
        float acc[kBatches][16];
#pragma unroll
        for (int b = 0; b < kBatches; ++b)
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[b][j] = 0.0f;
#pragma unroll 1
        for (uint32_t d0 = 0; d0 < drains; d0 += per_set, ++set) {
          const uint32_t batch = d0 / kScaleBatch, d_end = min(d0 + per_set, drains);  // a set lies inside a batch of scales
          if constexpr (kGroupScales) {
            if (d0 % kScaleBatch == 0) wait_bounded(sfull + (batch & 1u) * 8, (batch >> 1) & 1u, abort_flag, p.status, 25);
          }
          wait_bounded(dfull + (set & 1u) * 8, (set >> 1) & 1u, abort_flag, p.status, 23);
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          uint32_t at = taddr + (set & 1u) * kMaxNT;
#pragma unroll 1
          for (uint32_t d = d0; d < d_end; ++d, at += acc_cols) {
            [[maybe_unused]] float s = 1.0f;
            if constexpr (kGroupScales) s = my_scale[((batch & 1u) * kScaleBatch + d % kScaleBatch) * kRows];
            // scalar fused multiply-adds: the packed form (fma.rn.f32x2) wants register pairs, which the
            // allocator does not find beside 128 sums without spills (k-steps of 1,777 and 1,426 clocks at 256 and
            // 192 columns against 1,765 and 1,380; narrower tiles, with sums to spare, gain 5 to 9 %)
            auto add = [&](float (&sums)[16], const uint32_t (&v)[16]) {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                if constexpr (kGroupScales) sums[j] = fmaf(__uint_as_float(v[j]), s, sums[j]);
                else sums[j] += __uint_as_float(v[j]);
              }
            };
            if constexpr (kBatches <= 4) {  // the chain's columns in flight at once, one wait
              uint32_t v[kBatches][16];
#pragma unroll
              for (int b = 0; b < kBatches; ++b) tmem_ld16_begin(at + b * 16u, v[b]);
              tmem_ld_wait();
#pragma unroll
              for (int b = 0; b < kBatches; ++b) {
                tmem_ld16_done(v[b]);
                add(acc[b], v[b]);
              }
            } else {
#pragma unroll
              for (int b = 0; b < kBatches; ++b) {
                uint32_t v[16];
                tmem_ld16(at + b * 16u, v);
                add(acc[b], v);
              }
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          arrive_if(leader, dempty_0 + (set & 1u) * 8);
          if (kGroupScales) arrive_if(d_end % kScaleBatch == 0 ? leader : 0u, sempty + (batch & 1u) * 8);
        }
#pragma unroll
        for (int b = 0; b < kBatches; ++b)
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) sts32(park + (b * 16u + j) * 128u, __float_as_uint(acc[b][j]));
      };
      switch (p.nt / 32) {
        case 1: drain_all(std::integral_constant<int, 1>{}); break;
        case 2: drain_all(std::integral_constant<int, 2>{}); break;
        case 3: drain_all(std::integral_constant<int, 3>{}); break;
        case 4: drain_all(std::integral_constant<int, 4>{}); break;
        case 5: drain_all(std::integral_constant<int, 5>{}); break;
        case 6: drain_all(std::integral_constant<int, 6>{}); break;
        case 7: drain_all(std::integral_constant<int, 7>{}); break;
        default: drain_all(std::integral_constant<int, 8>{}); break;
      }
    }
    if (last_tile && (!kMaySlice || p.cluster_splits == 1)) emit_parked();
    if (kMaySlice && p.cluster_splits > 1) {
      // ---------------- K slices of a cluster: they meet in slice order, each finishing its share of the columns ----------------
      const ExTarget tg = p.t[at_tile.wi];
      const uint32_t slices = p.cluster_splits, share0 = cols * at_tile.z / slices, share1 = cols * (at_tile.z + 1) / slices;
      const uint32_t row = at_tile.n0 + quarter * 32u + lane, mm0 = m0 + col0;
      const bool row_live = row < tg.n;
      const uint32_t live_cols = row_live && mm0 < p.m ? min(cols, p.m - mm0) : 0u, last = min(share1, live_cols);
      cluster_sync_all();  // everybody has parked
      const float bias = row_live ? tg.bias[row] : 0.0f;
      [[maybe_unused]] float ws = 1.0f;
      if constexpr (!kGroupScales) ws = row_live ? load_scale_dyn(tg.scale, row, p.scale_f16) : 0.0f;
      float* dst = tg.out + static_cast<size_t>(mm0 + share0) * tg.n + row;
      const float* res = tg.residual != nullptr ? tg.residual + static_cast<size_t>(mm0 + share0) * tg.n + row : nullptr;
      uint32_t from[kMaxClusterSplits];
#pragma unroll
      for (uint32_t z = 0; z < kMaxClusterSplits; ++z) from[z] = map_to_cta(park, 2u * min(z, slices - 1u) + cta_rank);
      auto finish = [&](auto count, uint32_t c) {
        uint32_t sum = 0, v[decltype(count)::value];
#pragma unroll
        for (uint32_t z = 0; z < decltype(count)::value; ++z) v[z] = lds32_cluster(from[z] + c * 128u);
        const float rs = row_factor[c];
#pragma unroll
        for (uint32_t z = 0; z < decltype(count)::value; ++z)
          sum = z == 0 ? v[0] : kMath == kInt8 ? sum + v[z] : __float_as_uint(__uint_as_float(sum) + __uint_as_float(v[z]));
        float o = finished(sum, rs, ws, bias);
        if (res != nullptr) {
          o = __fadd_rn(o, *res);
          res += tg.n;
        }
        *dst = o;
        dst += tg.n;
      };
      if (slices == 2) {
#pragma unroll 8
        for (uint32_t c = share0; c < last; ++c) finish(std::integral_constant<uint32_t, 2>{}, c);
      } else {
#pragma unroll 4
        for (uint32_t c = share0; c < last; ++c) finish(std::integral_constant<uint32_t, kMaxClusterSplits>{}, c);
      }
    }
    } while (kMulti && (tile += tile_step) < tiles_all);
  } else if (warp < kDrainWarps + kProdWarps) {
    // ---------------- producers ----------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    // With four stages or more one warp converts the whole weight tile of a k-step, and the four warps take
    // stages in turn: what a k-step costs in latency (wait, loads, fence, arrival) then overlaps other
    // k-steps.  A stage belongs to ONE warp: it waits for that barrier's phases one after the other, so a
    // parity can never be mistaken for the one two phases away (copies of different stages finish in any
    // order).  Wide tiles of three-part activations leave three stages: a tile's conversion is then part of
    // every third k-step's trip, and the four warps share it.
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t unit = raw_unit_bytes<kW, kMath>(p.scale_f16), full_0 = map_to_cta(full, pair_rank0);
    constexpr int kUnroll = kParts == 3 ? 2 : 4;
    const bool shared_stage = stage_warps<kMath>(p.stages) != 1;
    const uint32_t rb0 = shared_stage ? 2u * (warp - kDrainWarps) : 0u, rb1 = shared_stage ? rb0 + 2u : 8u;  // this warp's 16-row blocks
    uint32_t s = 0, phase = 0;
    uint32_t tile = tile0;
    do {
    const uint32_t ks_count = kMulti ? tile_at(tile).ks_count : tile_first.ks_count;
#pragma unroll 1
    for (uint32_t ks = 0; ks < ks_count; ++ks, s = s + 1 == p.stages ? 0u : s + 1u, phase ^= s == 0 ? 1u : 0u) {
      if (!shared_stage && (s & (kProdWarps - 1u)) != warp - kDrainWarps) continue;
      const uint32_t ready = wait_bounded(rawfull + s * 8, phase, abort_flag, p.status, 21) ? leader : 0u;
      const uint32_t a_tile = tiles + s * p.stage_bytes, raw = a_tile + p.raw_off;
      if constexpr (kW == kI4Tiled) {
        // words: row g group 0 | row g+8 group 0 | row g group 1 | row g+8 group 1, each k 8t..8t+7 of
        // the group: 16-byte piece t / 4 + t of the tile row.  Odd g stores group 1 first, so the 8
        // lanes of a shared-memory phase hit 8 different pieces of the swizzled rows.
        const bool odd = (g & 1u) != 0;
        const uint32_t p0 = odd ? 4u + t : t, p1 = odd ? t : 4u + t;
        uint4 q = lds128(raw + rb0 * unit + lane * 16u);
#pragma unroll kUnroll
        for (uint32_t c = rb0; c < rb1; ++c) {
          const uint4 now = q;
          if (c + 1u < rb1) q = lds128(raw + (c + 1u) * unit + lane * 16u);
          const uint32_t r_a = c * 16u + g, r_b = r_a + 8u;
          sts128(a_tile + swz(r_a, p0), nibbles_to_operand<kMath>(odd ? now.z : now.x));
          sts128(a_tile + swz(r_a, p1), nibbles_to_operand<kMath>(odd ? now.x : now.z));
          sts128(a_tile + swz(r_b, p0), nibbles_to_operand<kMath>(odd ? now.w : now.y));
          sts128(a_tile + swz(r_b, p1), nibbles_to_operand<kMath>(odd ? now.y : now.w));
        }
      } else if constexpr (kW == kI4Rows) {
        // a row's k-step is 32 bytes: lane = (row, half), 16 bytes = 32 k = four pieces
#pragma unroll kUnroll
        for (uint32_t c = rb0; c < rb1; ++c) {
          const uint32_t r = c * 16u + (lane >> 1), h = lane & 1u;
          const uint4 q = lds128(raw + r * 32u + h * 16u);
          sts128(a_tile + swz(r, h * 4u + 0u), nibbles_to_operand<kMath>(q.x));
          sts128(a_tile + swz(r, h * 4u + 1u), nibbles_to_operand<kMath>(q.y));
          sts128(a_tile + swz(r, h * 4u + 2u), nibbles_to_operand<kMath>(q.z));
          sts128(a_tile + swz(r, h * 4u + 3u), nibbles_to_operand<kMath>(q.w));
        }
      } else if constexpr (kW == kI8Tiled && kMath != kInt8) {
        // chunk j, words: row g k 4t.. | row g+8 same k | row g k 16+4t.. | row g+8: four weights = 8
        // bytes = half (t & 1) of piece 4j + 2h + (t >> 1).  The order in which a lane walks its four
        // (j, h) pairs is XORed with a value that differs where the rows' swizzle term does not, so
        // the 16 lanes of a phase hit 8 different pieces.
#pragma unroll 2
        for (uint32_t rb = rb0; rb < rb1; ++rb) {
          const uint32_t r_a = rb * 16u + g, r_b = r_a + 8u;
          const uint32_t flip = (g & 1u) * 2u, sub = t >> 1, byte = (t & 1u) * 8u;
          uint4 q[2];
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j) q[j] = lds128(raw + rb * unit + (j ^ (flip >> 1)) * 512u + lane * 16u);
#pragma unroll
          for (uint32_t j = 0; j < 2; ++j) {
            const uint32_t o = (2u * j) ^ flip;
            sts64(a_tile + swz(r_a, o * 2u + sub) + byte, bytes_to_operand<kMath>(q[j].x));
            sts64(a_tile + swz(r_b, o * 2u + sub) + byte, bytes_to_operand<kMath>(q[j].y));
            sts64(a_tile + swz(r_a, (o + 1u) * 2u + sub) + byte, bytes_to_operand<kMath>(q[j].z));
            sts64(a_tile + swz(r_b, (o + 1u) * 2u + sub) + byte, bytes_to_operand<kMath>(q[j].w));
          }
        }
      } else if constexpr (kW == kI8Rows && kMath != kInt8) {
        // a row's k-step is 64 bytes: lane = (row, quarter), 16 bytes = 16 k = two pieces
#pragma unroll 4
        for (uint32_t c = 2u * rb0; c < 2u * rb1; ++c) {
          const uint32_t r = c * 8u + (lane >> 2), qd = lane & 3u;
          const uint4 q = lds128(raw + r * 64u + qd * 16u);
          const uint2 a = bytes_to_operand<kMath>(q.x ^ 0x80808080u), b = bytes_to_operand<kMath>(q.y ^ 0x80808080u);
          const uint2 d = bytes_to_operand<kMath>(q.z ^ 0x80808080u), e = bytes_to_operand<kMath>(q.w ^ 0x80808080u);
          sts128(a_tile + swz(r, qd * 2u), make_uint4(a.x, a.y, b.x, b.y));
          sts128(a_tile + swz(r, qd * 2u + 1u), make_uint4(d.x, d.y, e.x, e.y));
        }
      } else if constexpr (kW == kI8Tiled) {
        // int8 tile: four chunks (32 k each) of a row block; a word is 4 bytes of piece 2j + h, the sign
        // bit flipped back.  Eight rows x four words hit 32 different banks.
#pragma unroll 2
        for (uint32_t rb = rb0; rb < rb1; ++rb) {
          const uint32_t r_a = rb * 16u + g, r_b = r_a + 8u;
          uint4 qs[4];
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) qs[j] = lds128(raw + rb * unit + j * 512u + lane * 16u);
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j) {
            const uint4 q = qs[j];
            sts32(a_tile + swz(r_a, 2u * j) + 4u * t, q.x ^ 0x80808080u);
            sts32(a_tile + swz(r_b, 2u * j) + 4u * t, q.y ^ 0x80808080u);
            sts32(a_tile + swz(r_a, 2u * j + 1u) + 4u * t, q.z ^ 0x80808080u);
            sts32(a_tile + swz(r_b, 2u * j + 1u) + 4u * t, q.w ^ 0x80808080u);
          }
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // -> visible to the tensor core
      __syncwarp();
      arrive_if(ready, full_0 + s * 8);  // the issuing CTA's barrier
    }
    } while (kMulti && (tile += tile_step) < tiles_all);
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == kCopyWarp) {
      // ---------------- copies ----------------
      // One thread, two tensor copies per k-step (all activation parts come with one): a copy takes it about
      // 100 clocks, and a bulk copy per 16-row block, eight of them, 700 - 1000: more than the k-step's MMAs.
      {
        const uint32_t half_rows = p.nt / 2, b_bytes = half_rows * 128u, raw_bytes = p.raw_bytes;
        const uint32_t full_0 = map_to_cta(full, pair_rank0), raw_off = kW == kI8Rows && kMath == kInt8 ? 0u : p.raw_off;
        uint32_t s = 0, phase = 0;
        uint32_t tile = tile0;
        do {
        const Tile at = kMulti ? tile_at(tile) : tile_first;
        const CUtensorMap* w_map = at.wi == 0 ? &w_map0 : at.wi == 1 ? &w_map1 : at.wi == 2 ? &w_map2 : &w_map3;
        const uint32_t w_row = kTiled ? at.n0 / 16u : at.n0, w_step = p.raw_box;  // tensor-map rows and columns of the raw weights
#pragma unroll 1
        for (uint32_t ks = 0; ks < at.ks_count; ++ks) {
          const uint32_t free = wait_bounded(empty + s * 8, phase ^ 1u, abort_flag, p.status, 20) ? leader : 0u;
          const uint32_t a_tile = tiles + s * p.stage_bytes, kstep = at.ks_begin + ks;
          expect_tx(cta_rank == 0 ? free : 0u, full + s * 8, kParts * 2u * b_bytes);
          expect_tx(free, rawfull + s * 8, raw_bytes);
          copy_tile_2d(free, a_tile + raw_off, w_map, kstep * w_step, w_row, rawfull + s * 8);
          if (gated) copy_tile_2d(free, a_tile + raw_off + raw_bytes / 2, &w_map1, kstep * w_step, w_row, rawfull + s * 8);
          copy_tile_3d(free, a_tile + kATile, &x_map, kstep * (kMath == kInt8 ? 128u : 64u), at.m0 + cta_rank * half_rows, 0, full_0 + s * 8);
          if (++s == p.stages) { s = 0; phase ^= 1u; }
        }
        } while (kMulti && (tile += tile_step) < tiles_all);
      }
      __syncwarp();
    } else if (warp == kMmaWarp && cta_rank == 0) {
      // ---------------- MMA issuer: one thread, nothing converges in its loop ----------------
      {
        const uint32_t idesc = exact_idesc<kMath>(p.nt);
        const uint32_t pair_mask = 3u << pair_rank0;
        const uint32_t b_step = (p.nt / 2 * 128u) >> 4, stage_step = p.stage_bytes >> 4;
        const uint32_t desc_a0 = static_cast<uint32_t>(umma_desc(tiles)), desc_b0 = static_cast<uint32_t>(umma_desc(tiles + kATile));
        // kSlices: k16 slices per accumulator chain when chains end inside a k-step or with it; 0: longer
        // chains, of p.drain16 slices
        auto issue = [&](auto slices) {
          constexpr uint32_t kSlices = decltype(slices)::value;
          uint32_t s = 0, phase = 0, set = 0, in_set = 0, in_chain = 0;
          auto chain_begins = [&]() {
            if (in_set == 0 && set >= 2) {  // both CTAs have read the set's previous sums
              wait_bounded(dempty + (set & 1u) * 8, ((set >> 1) - 1u) & 1u, abort_flag, p.status, 24);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
          };
          auto chain_ends = [&](bool last) {
            if (++in_set == per_set || last) {
              commit_both(leader, dfull + (set & 1u) * 8, pair_mask);
              ++set;
              in_set = 0;
            }
          };
          uint32_t tile = tile0;
          do {
          const uint32_t ks_count = kMulti ? tile_at(tile).ks_count : tile_first.ks_count;
#pragma unroll 1
          for (uint32_t ks = 0; ks < ks_count; ++ks) {
            wait_bounded(full + s * 8, phase, abort_flag, p.status, 22);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t desc_a = desc_a0 + s * stage_step, desc_b = desc_b0 + s * stage_step, this_empty = empty + s * 8;
            if (++s == p.stages) { s = 0; phase ^= 1u; }
            // Low parts first: an accumulation truncates to the accumulator's size, so the fewer follow once the
            // high parts are in, the better (289 rows through four layers of a decoder: 1.8e-7 from f64 against
            // 3.9e-7 with the high parts first).
            constexpr uint32_t kRun = kSlices == 0 ? 4u : kSlices;  // slices of a chain in this k-step
#pragma unroll
            for (uint32_t run = 0; run < 4; run += kRun) {
              const bool starts = kSlices != 0 || in_chain == 0;
              if (starts) chain_begins();
              const uint32_t dst = tmem + (set & 1u) * kMaxNT + in_set * acc_cols;
#pragma unroll
              for (uint32_t back = 1; back <= kParts; ++back) {
                const uint32_t part = kParts - back;
#pragma unroll
                for (uint32_t kk = run; kk < run + kRun; ++kk) {
                  const uint32_t a = desc_a + kk * 2u, b = desc_b + part * b_step + kk * 2u;
                  if (back == 1 && kk == run && starts) mma_pair<kMath, false>(leader, dst, a, b, idesc);
                  else mma_pair<kMath, true>(leader, dst, a, b, idesc);
                }
              }
              if constexpr (kMath != kInt8 && kSlices != 0) chain_ends(run + kRun == 4 && ks + 1 == ks_count);
            }
            if constexpr (kSlices == 0) {
              in_chain += 4;
              if ((kMath != kInt8 && in_chain == p.drain16) || ks + 1 == ks_count) {  // the last chain may be short
                chain_ends(ks + 1 == ks_count);
                in_chain = 0;
              }
            }
            commit_both(leader, this_empty, pair_mask);  // the stage is free, in both CTAs, once these MMAs have read it
          }
          } while (kMulti && (tile += tile_step) < tiles_all);
        };
        if (kGroupScales && p.drain16 == 1) issue(std::integral_constant<uint32_t, 1>{});
        else if (kGroupScales && p.drain16 == 2) issue(std::integral_constant<uint32_t, 2>{});
        else if (kGroupScales && p.drain16 == 4) issue(std::integral_constant<uint32_t, 4>{});
        else issue(std::integral_constant<uint32_t, 0>{});
      }
      __syncwarp();
    } else if (kGroupScales && warp >= kScaleWarp) {
      // ---------------- scales: global memory -> f32 ring, eight accumulator chains at a time ----------------
      // Each of the 64 lanes serves two rows.  A batch is fetched into registers as soon as the one before it has
      // been stored: fetched only once its slot was free, a batch cost two trips to memory and the drain waited
      // for it (4,600 clocks per eight chains; 24 x 4096 -> 9472: 30 us).
      const uint32_t wl = (warp - kScaleWarp) * 32u + lane;
      uint32_t batch = 0;
      const Tile at_tile = tile_first;  // (kMulti has no group scales)
      const uint32_t drains = (at_tile.ks_count * 4 + p.drain16 - 1) / p.drain16, drain0 = at_tile.ks_begin * 4 / p.drain16;
      if constexpr (kW == kI4Tiled) {
        // rows 16 (wl / 8) + wl % 8 and + 8: a chunk holds their scales of two groups side by side
        const uint32_t unit = raw_unit_bytes<kW, kMath>(p.scale_f16), r = (wl >> 3) * 16u + (wl & 7u);
        const ExTarget& tg = p.t[gated ? r / (kRows / 2) : at_tile.wi];
        const uint32_t row = at_tile.n0 + (gated ? r % (kRows / 2) : r);
        const uint8_t* base = tg.w + static_cast<size_t>(row >> 4) * (p.k / kChunkK) * unit + kChunkWeightBytes + (wl & 7u) * (p.scale_f16 ? 8u : 16u);
        float4 v[kScaleBatch / 2];  // {row, group 0 | row + 8, group 0 | row, group 1 | row + 8, group 1}
        auto load = [&](uint32_t d0) {
#pragma unroll
          for (uint32_t i = 0; i < kScaleBatch / 2; ++i) {
            const uint32_t chunk = (drain0 + d0) / 2 + i;
            v[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < tg.n && d0 + 2 * i < drains && chunk < p.k / kChunkK) {
              const uint8_t* at = base + static_cast<size_t>(chunk) * unit;
              if (p.scale_f16) {
                const uint2 raw = __ldg(reinterpret_cast<const uint2*>(at));
                const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
                v[i] = make_float4(lo.x, lo.y, hi.x, hi.y);
              } else {
                v[i] = __ldg(reinterpret_cast<const float4*>(at));
              }
            }
          }
        };
        load(0);
        for (uint32_t d0 = 0; d0 < drains; d0 += kScaleBatch, ++batch) {
          if (batch >= 2) wait_bounded(sempty + (batch & 1u) * 8, ((batch >> 1) - 1u) & 1u, abort_flag, p.status, 26);
          float* ring = scale_ring + (batch & 1u) * (kScaleBatch * kRows) + r;
#pragma unroll
          for (uint32_t i = 0; i < kScaleBatch / 2; ++i) {
            ring[2 * i * kRows] = v[i].x;
            ring[2 * i * kRows + 8] = v[i].y;
            ring[(2 * i + 1) * kRows] = v[i].z;
            ring[(2 * i + 1) * kRows + 8] = v[i].w;
          }
          __syncwarp();
          arrive_if(leader, sfull + (batch & 1u) * 8);
          load(d0 + kScaleBatch);
        }
      } else {
        const uint32_t each = p.scale_f16 ? 2u : 4u;
        float v[2][kScaleBatch];
        auto load = [&](uint32_t d0) {
#pragma unroll
          for (uint32_t rr = 0; rr < 2; ++rr) {
            const ExTarget& tg = p.t[gated ? rr : at_tile.wi];
            const uint32_t row = at_tile.n0 + wl + (gated ? 0u : rr * 64u);
            const uint8_t* base = static_cast<const uint8_t*>(tg.scale) + static_cast<size_t>(row) * p.groups * each;
#pragma unroll
            for (uint32_t i = 0; i < kScaleBatch; ++i) {
              const uint32_t grp = (drain0 + d0 + i) >> p.drains_per_group_shift;
              v[rr][i] = 0.0f;
              if (row < tg.n && grp < p.groups && d0 + i < drains) {
                const uint8_t* at = base + static_cast<size_t>(grp) * each;
                v[rr][i] = p.scale_f16 ? __half2float(*reinterpret_cast<const __half*>(at)) : *reinterpret_cast<const float*>(at);
              }
            }
          }
        };
        load(0);
        for (uint32_t d0 = 0; d0 < drains; d0 += kScaleBatch, ++batch) {
          if (batch >= 2) wait_bounded(sempty + (batch & 1u) * 8, ((batch >> 1) - 1u) & 1u, abort_flag, p.status, 26);
#pragma unroll
          for (uint32_t rr = 0; rr < 2; ++rr)
#pragma unroll
            for (uint32_t i = 0; i < kScaleBatch; ++i) scale_ring[((batch & 1u) * kScaleBatch + i) * kRows + wl + rr * 64u] = v[rr][i];
          __syncwarp();
          arrive_if(leader, sfull + (batch & 1u) * 8);
          load(d0 + kScaleBatch);
        }
      }
    }
  }

  if (kMaySlice && p.cluster_splits > 1 && warp >= kDrainWarps) cluster_sync_all();  // (the drain warps' barrier in front of their epilogue)
  if (*abort_flag)  // a wait gave up: copies may still be in flight towards this CTA's shared memory
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  cluster_sync_all();  // neither CTA leaves, or frees tensor memory, while the other still works
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- f32 and bf16 activations -> parts ----------------------------------------------------------
// One CTA per row.  [rms_norm ->] a power of two over the whole row -> parts that add up to the value: three
// bf16 ones of an f32 value, the one of a bf16 value, or two binary16 ones (pow2_prescale); inv[row] = 2^-e
// undoes the power in the epilogue.
//
// bf16 parts have f32's exponents, so their power of two is only there to keep the sums of up to 1024 products
// with integers, and those times a group scale, away from both ends of the range: the row's largest value goes
// to [2^40, 2^41).  A value then keeps all its bits down to 2^-150 of that one (a part of less than 2^-133
// vanishes).  A row of zeros, or one whose largest value is not finite, keeps its values.
__device__ __forceinline__ Pow2 pow2_row(float amax) {
  const uint32_t bits = __float_as_uint(amax) & 0x7fffffffu;
  int e = 0;
  if (bits != 0u && bits < 0x7f800000u) e = min(126, 40 + 127 - static_cast<int>(bits >> 23));  // -87 .. 126
  Pow2 r;
  r.scale = __uint_as_float(static_cast<uint32_t>(e + 127) << 23);
  r.inv = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
  return r;
}
// kHold: a row of up to 2,048 values a unit stays in the threads' registers between the passes; 0: it is read again for
// each.  (Bound by trips to memory one after the other: three of them were one too many or two.  125 x 11904 -> 5984 78.7 us
// before, 74.3 now; 257 x 1536 -> 8960 23.3, 22.5; four layers of 333 rows 665, 653.)
template <typename XT, int kMath, int kHold>
__global__ void __launch_bounds__(256)
split_kernel(const XT* __restrict__ x, uint32_t m, uint32_t k, uint16_t* __restrict__ parts, float* __restrict__ inv,
             const float* __restrict__ norm_weight, float norm_eps) {
  constexpr uint32_t kParts = parts_of(kMath);
  const uint32_t row = blockIdx.x;
  const XT* xr = x + static_cast<size_t>(row) * k;
  __shared__ float part[8];
  pdl_wait_prior_grid();
  float r_inv = 1.0f;
  float held[kHold > 0 ? kHold : 1][8];
  if constexpr (kHold > 0) {
#pragma unroll
    for (int h = 0; h < kHold; ++h) {
      const uint32_t i = threadIdx.x * 8 + h * 2048u;
#pragma unroll
      for (int e = 0; e < 8; ++e) held[h][e] = 0.0f;
      if (i < k) load_x8<XT>(xr + i, held[h]);
    }
  }
  if (norm_weight != nullptr) {
    // sum of squares in a fixed order: thread-strided, shuffle tree, warps in order
    float sq = 0.0f;
    if constexpr (kHold > 0) {
#pragma unroll
      for (int h = 0; h < kHold; ++h)
#pragma unroll
        for (int e = 0; e < 8; ++e) sq = fmaf(held[h][e], held[h][e], sq);
    } else {
      for (uint32_t i = threadIdx.x * 8; i < k; i += 2048) {
        float v[8];
        load_x8<XT>(xr + i, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) sq = fmaf(v[e], v[e], sq);
      }
    }
    sq = warp_sum(sq);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = sq;
    __syncthreads();
    float total = 0.0f;
    for (int w = 0; w < 8; ++w) total += part[w];
    r_inv = rsqrtf(total * (1.0f / static_cast<float>(k)) + norm_eps);
    __syncthreads();
  }
  auto scaled = [&](uint32_t i, float (&v)[8]) {
    if (norm_weight != nullptr) {
      const float4 w0 = __ldg(reinterpret_cast<const float4*>(norm_weight + i)), w1 = __ldg(reinterpret_cast<const float4*>(norm_weight + i + 4));
      const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = __fmul_rn(__fmul_rn(v[e], r_inv), wv[e]);
    }
  };
  float amax = 0.0f;
  if constexpr (kHold > 0) {
#pragma unroll
    for (int h = 0; h < kHold; ++h) {
      const uint32_t i = threadIdx.x * 8 + h * 2048u;
      if (i < k) {
        scaled(i, held[h]);
        amax = fmaxf(amax, absmax8(held[h]));
      }
    }
  } else {
    for (uint32_t i = threadIdx.x * 8; i < k; i += 2048) {  // k is a multiple of 16
      float v[8];
      load_x8<XT>(xr + i, v);
      scaled(i, v);
      amax = fmaxf(amax, absmax8(v));
    }
  }
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, offset));
  if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = part[0];
  for (int w = 1; w < 8; ++w) amax = fmaxf(amax, part[w]);
  const Pow2 ps = kIsBf<kMath> ? pow2_row(amax) : pow2_prescale(amax);
  if (threadIdx.x == 0) inv[row] = ps.inv;
  auto store = [&](uint32_t i, float (&v)[8]) {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= ps.scale;
#pragma unroll
    for (uint32_t part = 0; part < kParts; ++part) {
      uint4 o;
      uint32_t* po = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f;
        if constexpr (kIsBf<kMath>) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
          po[j] = *reinterpret_cast<const uint32_t*>(&h);
          f = __bfloat1622float2(h);
        } else {
          const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
          po[j] = *reinterpret_cast<const uint32_t*>(&h);
          f = __half22float2(h);
        }
        // the rest is exact; an infinite value has none (Inf - Inf is a NaN)
        v[2 * j] = isinf(f.x) ? 0.0f : v[2 * j] - f.x;
        v[2 * j + 1] = isinf(f.y) ? 0.0f : v[2 * j + 1] - f.y;
      }
      *reinterpret_cast<uint4*>(parts + (static_cast<size_t>(part) * m + row) * k + i) = o;
    }
  };
  if constexpr (kHold > 0) {
#pragma unroll
    for (int h = 0; h < kHold; ++h) {
      const uint32_t i = threadIdx.x * 8 + h * 2048u;
      if (i < k) store(i, held[h]);
    }
  } else {
    for (uint32_t i = threadIdx.x * 8; i < k; i += 2048) {
      float v[8];
      load_x8<XT>(xr + i, v);
      scaled(i, v);
      store(i, v);
    }
  }
  pdl_launch_dependents();
}

// int8 activations -> binary16 (exact), 16 values per thread
__global__ void __launch_bounds__(256)
bytes_to_half_kernel(const int8_t* __restrict__ q, uint64_t sixteens, __half* __restrict__ out) {
  pdl_wait_prior_grid();
  for (uint64_t i = blockIdx.x * 256ull + threadIdx.x; i < sixteens; i += static_cast<uint64_t>(gridDim.x) * 256ull) {
    const uint4 v = reinterpret_cast<const uint4*>(q)[i];
    const uint2 a = bytes_to_half(v.x ^ 0x80808080u), b = bytes_to_half(v.y ^ 0x80808080u);
    const uint2 c = bytes_to_half(v.z ^ 0x80808080u), d = bytes_to_half(v.w ^ 0x80808080u);
    reinterpret_cast<uint4*>(out)[2 * i] = make_uint4(a.x, a.y, b.x, b.y);
    reinterpret_cast<uint4*>(out)[2 * i + 1] = make_uint4(c.x, c.y, d.x, d.y);
  }
  pdl_launch_dependents();
}

// The K slices of a split launch, added in ascending order, then the epilogue.
struct ExReduceParams {
  ExTarget t[kMaxMulti];
  uint32_t count, m, n_total, splits, scale_f16, per_channel;
  const float* row_scale;
  const void* partial;
};
template <bool kInt8Sums>
__global__ void __launch_bounds__(256) exact_reduce_kernel(const ExReduceParams p) {
  pdl_wait_prior_grid();
  pdl_launch_dependents();
  const size_t slice = static_cast<size_t>(p.m) * p.n_total;
  for (size_t i = blockIdx.x * static_cast<size_t>(256) + threadIdx.x; i < slice; i += static_cast<size_t>(gridDim.x) * 256) {
    const uint32_t mm = static_cast<uint32_t>(i / p.n_total);
    uint32_t col = static_cast<uint32_t>(i - static_cast<size_t>(mm) * p.n_total);
    uint32_t wi = 0;
#pragma unroll
    for (int j = 1; j < kMaxMulti; ++j)
      if (j < static_cast<int>(p.count) && wi + 1 == static_cast<uint32_t>(j) && col >= p.t[j - 1].n) { col -= p.t[j - 1].n; wi = j; }
    const ExTarget& tg = p.t[wi];
    const float rs = p.row_scale != nullptr ? p.row_scale[mm] : 1.0f;
    float o;
    if constexpr (kInt8Sums) {
      const int* src = static_cast<const int*>(p.partial) + i;
      int acc = 0;
      for (uint32_t z = 0; z < p.splits; ++z) acc += src[z * slice];
      o = fmaf(__int2float_rn(acc), __fmul_rn(rs, load_scale_dyn(tg.scale, col, p.scale_f16)), tg.bias[col]);
    } else {
      const float* src = static_cast<const float*>(p.partial) + i;
      float acc = 0.0f;
      for (uint32_t z = 0; z < p.splits; ++z) acc += src[z * slice];
      if (p.per_channel) acc *= load_scale_dyn(tg.scale, col, p.scale_f16);
      o = fmaf(acc, rs, tg.bias[col]);
    }
    const size_t at = static_cast<size_t>(mm) * tg.n + col;
    if (tg.residual != nullptr) o = __fadd_rn(o, tg.residual[at]);
    tg.out[at] = o;
  }
}

// ---- host ---------------------------------------------------------------------------------------
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled tensor_map_encoder() {
  static EncodeTiled encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<EncodeTiled>(fn);
  }();
  return encode;
}

// Activations [parts][m][k] (binary16, bf16 or int8), box 128 bytes x `rows` rows of every part, 128-byte swizzle; what
// lies past k or m reads as zero.
cudaError_t encode_x_map(const void* x, bool int8, uint32_t m, uint32_t k, uint32_t parts, uint32_t rows, CUtensorMap* map) {
  EncodeTiled encode = tensor_map_encoder();
  if (encode == nullptr) return cudaErrorNotSupported;
  const cuuint64_t each = int8 ? 1 : 2;
  const cuuint64_t dims[3] = {k, m, parts}, strides[2] = {k * each, static_cast<cuuint64_t>(m) * k * each};
  const cuuint32_t box[3] = {int8 ? 128u : 64u, rows, parts}, ones[3] = {1, 1, 1};
  const CUresult r = encode(map, int8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void*>(x), dims,
                            strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
// The packed weights as rows of bytes, one copy per k-step and CTA: rows layouts [n][row_bytes], box
// `bytes` x 128 rows (128-byte swizzled when it is the MMA's tile itself); tiled layouts [n / 16][row_bytes]
// of 16-row blocks, box `bytes` x 8.  `elem` bytes per element keep the box within 256 elements.
cudaError_t encode_w_map(const void* w, uint32_t rows, uint64_t row_bytes, uint32_t bytes, uint32_t elem, uint32_t box_rows, bool swizzle,
                         CUtensorMap* map) {
  EncodeTiled encode = tensor_map_encoder();
  if (encode == nullptr) return cudaErrorNotSupported;
  const cuuint64_t dims[2] = {row_bytes / elem, rows}, strides[1] = {row_bytes};
  const cuuint32_t box[2] = {bytes / elem, box_rows}, ones[2] = {1, 1};
  const CUtensorMapDataType type = elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT64;
  const CUresult r = encode(map, type, 2, const_cast<void*>(w), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <typename Kernel, typename... Args>
cudaError_t launch_dependent(Kernel kernel, dim3 grid, uint32_t threads, size_t smem, dim3 cluster, const LaunchEnv& env, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = env.stream;
  cudaLaunchAttribute attr[2];
  unsigned int na = 0;
  if (env.overlap) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (cluster.x > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = cluster.x;
    attr[na].val.clusterDim.y = cluster.y;
    attr[na].val.clusterDim.z = cluster.z;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

WeightKind kind_of(const Weight& w) {
  if (w.layout == kLayoutTiledI4) return kI4Tiled;
  if (w.layout == kLayoutTiledI8) return kI8Tiled;
  return w.storage == KQ_STORAGE_I4 ? kI4Rows : kI8Rows;
}
int math_of(int x_dtype, const Weight& w) { return x_dtype == KQ_F16 ? kHalf1 : x_dtype == KQ_BF16 ? kBf1 : kind_of(w) == kI8Tiled ? kHalf2 : kBf3; }
// The packed rows of the untiled layouts are read through a tensor map: 16-byte row strides.
bool kind_ok(const Weight& w) {
  switch (kind_of(w)) {
    case kI4Tiled: return true;
    case kI8Tiled: return w.k % 16 == 0;
    case kI4Rows: return w.k % 32 == 0;
    default: return w.k % 16 == 0;
  }
}

template <int kW, int kMath, int kForm>
cudaError_t launch_form(const LaunchEnv& env, const ExParams& p, const CUtensorMap& xm, const CUtensorMap (&wm)[kMaxMulti]) {
  auto kernel = qgemm_exact_kernel<kW, kMath, kForm>;
  static OncePerDevice configured;
  const cudaError_t ready = configured.run([&]() -> cudaError_t {
    // the register split adds up to 512 x 128: refuse to run a build whose launch holds fewer
    cudaFuncAttributes fa;
    const cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    if (fa.numRegs < 128) return cudaErrorInvalidKernelImage;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit));
  });
  if (ready != cudaSuccess) return ready;
  const size_t smem = 1024 + static_cast<size_t>(p.stages) * p.stage_bytes + smem_tail(kForm == kSeveral, p.nt);
  const dim3 grid = kForm == kSeveral ? dim3(p.resident * 2) : dim3(p.pairs * 2, p.m_tiles, p.splits);
  return launch_dependent(kernel, grid, kExThreads, smem, dim3(2, 1, p.cluster_splits), env, p, xm, wm[0], wm[1], wm[2], wm[3]);
}
template <int kW, int kMath>
cudaError_t launch_main(const LaunchEnv& env, const ExParams& p, const CUtensorMap& xm, const CUtensorMap (&wm)[kMaxMulti]) {
  if constexpr (kMath == kInt8) {
    return p.multi ? launch_form<kW, kMath, kSeveral>(env, p, xm, wm)
           : p.cluster_splits > 1 ? launch_form<kW, kMath, kSliced>(env, p, xm, wm) : launch_form<kW, kMath, kPlain>(env, p, xm, wm);
  } else {
    // (a decoder's prompt takes one kernel for all its matmuls: two that take turns cost it 6 us a layer in instructions
    // fetched again, 692 | 667 us for four layers of 333 rows.  Up to 512 channels are none of a decoder's: 20 x 64 -> 256 7.9
    // us in the prompt's form, 7.2 in the plain one, 64 x 6144 -> 128 16.0, 15.3)
    constexpr bool kPrompt = kW == kI4Tiled && parts_of(kMath) == 3;
    if (p.swiglu || (kPrompt && p.pairs > 2)) return launch_form<kW, kMath, kGate>(env, p, xm, wm);
    return p.cluster_splits > 1 ? launch_form<kW, kMath, kSliced>(env, p, xm, wm) : launch_form<kW, kMath, kPlain>(env, p, xm, wm);
  }
}

// Pairs (slots[1]) and clusters of two or four pairs that the device holds at once; 0 where it cannot say.  Every form of
// the kernel fills an SM, so one of them stands for all.
cudaError_t resident_pairs(const LaunchEnv& env, uint32_t (&slots)[kMaxClusterSplits + 1]) {
  struct Held { uint32_t clusters[kMaxClusterSplits + 1]; };
  static PerDevice<Held> held_on;
  const Held* held = nullptr;
  const cudaError_t known = held_on.get([](Held& h) -> cudaError_t {
    auto kernel = qgemm_exact_kernel<kI4Tiled, kHalf1, kSliced>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit));
    if (e != cudaSuccess) return e;
    for (uint32_t z = 2; z <= kMaxClusterSplits; z *= 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2, 1, z);
      cfg.blockDim = dim3(kExThreads);
      cfg.dynamicSmemBytes = kSmemLimit;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 2;
      attr.val.clusterDim.y = 1;
      attr.val.clusterDim.z = z;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 0) {
        (void)cudaGetLastError();
        n = 0;
      }
      h.clusters[z] = static_cast<uint32_t>(n);
    }
    return cudaSuccess;
  }, &held);
  if (known != cudaSuccess) return known;
  for (uint32_t z = 0; z <= kMaxClusterSplits; ++z) slots[z] = held->clusters[z];
  slots[1] = static_cast<uint32_t>(std::max(1, env.sm_count / 2));
  return cudaSuccess;
}

template <int kW>
cudaError_t launch_math(int math, const LaunchEnv& env, const ExParams& p, const CUtensorMap& xm, const CUtensorMap (&wm)[kMaxMulti]) {
  if (math == kHalf1) return launch_main<kW, kHalf1>(env, p, xm, wm);
  if (math == kBf1) return launch_main<kW, kBf1>(env, p, xm, wm);
  constexpr int kF32 = kW == kI8Tiled ? kHalf2 : kBf3;
  if (math == kF32) return launch_main<kW, kF32>(env, p, xm, wm);
  if constexpr (kW == kI8Tiled || kW == kI8Rows) return launch_main<kW, kInt8>(env, p, xm, wm);
  return cudaErrorInvalidValue;
}

// x: binary16 (kHalf1), parts already split (kHalf2 / kBf1 / kBf3) or int8 (kInt8).
cudaError_t run_exact(const LaunchEnv& env, int count, const LinearTarget* targets, const float* residual, const void* x, int math,
                      uint32_t m, uint32_t max_chain, const float* row_scale, void* scratch, uint64_t scratch_bytes, bool may_split, bool swiglu, int* launches) {
  const Weight& w0 = *targets[0].w;
  const WeightKind kind = kind_of(w0);
  ExParams p = {};
  ExReduceParams rp = {};
  CUtensorMap xm, wm[kMaxMulti] = {};
  const bool int8 = math == kInt8;
  uint32_t pairs = 0, n_total = 0;
  uint32_t used = 0;
  const uint32_t unit = kind == kI4Tiled ? raw_unit_bytes<kI4Tiled, kHalf1>(w0.scale_dtype == KQ_F16)
                        : kind == kI4Rows ? 32u
                        : kind == kI8Tiled ? (int8 ? 2048u : 1024u) : (int8 ? 128u : 64u);
  const bool tiled = kind == kI4Tiled || kind == kI8Tiled;
  const uint32_t elem = !tiled ? 1u : unit > 1024 ? 8u : 4u;
  for (int i = 0; i < count; ++i) {
    const Weight& w = *targets[i].w;
    if (w.n == 0) continue;
    p.t[used] = ExTarget{static_cast<const uint8_t*>(w.data), w.scale, targets[i].bias, targets[i].out, residual, w.n, pairs};
    const uint64_t row_bytes = kind == kI4Tiled ? static_cast<uint64_t>(w.k / kChunkK) * unit
                               : kind == kI8Tiled ? static_cast<uint64_t>(w.k) * 16 : kind == kI4Rows ? w.k / 2 : w.k;
    cudaError_t e = tiled ? encode_w_map(w.data, w.n / 16, row_bytes, unit, elem, swiglu ? 4 : 8, false, &wm[used])
                          : encode_w_map(w.data, w.n, row_bytes, unit, elem, swiglu ? kRows / 2 : kRows, kind == kI8Rows && int8, &wm[used]);
    if (e != cudaSuccess) return e;
    if (!swiglu || used == 0) {
      const uint32_t wide = swiglu ? kRows : 2 * kRows;  // channels of a pair
      pairs += (w.n + wide - 1) / wide;
      n_total += w.n;
    }
    ++used;
  }
  if (used == 0) return cudaSuccess;
  p.count = used;
  p.swiglu = swiglu ? 1 : 0;
  p.m = m;
  p.k = w0.k;
  p.scale_f16 = w0.scale_dtype == KQ_F16;
  const bool i4 = kind == kI4Tiled || kind == kI4Rows;
  const Steps steps = steps_of(w0.k, math, i4 ? w0.group_size : 0, max_chain);
  const uint32_t group = i4 ? w0.group_size : max_chain, chain = steps.drain16 * 16;
  p.ksteps = steps.ksteps;
  p.drain16 = steps.drain16;
  p.drains_per_group_shift = 0;
  while ((chain << p.drains_per_group_shift) < group) ++p.drains_per_group_shift;
  p.groups = i4 ? w0.k / w0.group_size : ~0u;
  p.row_scale = row_scale;
  p.n_total = n_total;
  p.status = env.status;
  p.partial = static_cast<float*>(scratch);
  const uint32_t parts = parts_of(math);
  uint32_t slots[kMaxClusterSplits + 1];
  cudaError_t ce = resident_pairs(env, slots);
  if (ce != cudaSuccess) return ce;
  const Geometry geo = choose_geometry(m, n_total, pairs, steps, math, !i4, may_split && !swiglu, slots,
                                       scratch != nullptr ? scratch_bytes : 0);
  p.nt = geo.nt;
  p.pairs = pairs;
  p.m_tiles = geo.m_tiles;
  p.ksteps_per_split = ((p.ksteps + geo.splits - 1) / geo.splits + steps.slice_unit - 1) / steps.slice_unit * steps.slice_unit;
  p.splits = (p.ksteps + p.ksteps_per_split - 1) / p.ksteps_per_split;
  p.cluster_splits = geo.cluster_splits;
  p.multi = int8 && p.splits == 1 && static_cast<uint64_t>(pairs) * geo.m_tiles > slots[1];
  p.resident = slots[1];
  // stage: weight tile, activation parts, raw weights
  p.raw_bytes = (tiled ? 8 : kRows) * unit;
  p.raw_box = unit / elem;
  const uint32_t raw_bytes = kind == kI8Rows && int8 ? 0 : p.raw_bytes;  // straight into the weight tile
  p.raw_off = kATile + parts * p.nt / 2 * 128;
  p.stage_bytes = (p.raw_off + raw_bytes + 1023) / 1024 * 1024;
  p.stages = std::min<uint32_t>(kMaxStages, (kSmemLimit - 1024 - smem_tail(p.multi != 0, p.nt)) / p.stage_bytes);
  cudaError_t e = encode_x_map(x, int8, m, w0.k, parts, p.nt / 2, &xm);
  if (e != cudaSuccess) return e;
  switch (kind) {
    case kI4Tiled: e = launch_math<kI4Tiled>(math, env, p, xm, wm); break;
    case kI4Rows: e = launch_math<kI4Rows>(math, env, p, xm, wm); break;
    case kI8Tiled: e = launch_math<kI8Tiled>(math, env, p, xm, wm); break;
    default: e = launch_math<kI8Rows>(math, env, p, xm, wm); break;
  }
  if (e != cudaSuccess) return e;
  if (launches) *launches += 1;
  if (p.splits > p.cluster_splits) {
    for (uint32_t i = 0; i < used; ++i) rp.t[i] = p.t[i];
    rp.count = used;
    rp.m = m;
    rp.n_total = n_total;
    rp.splits = p.splits;
    rp.scale_f16 = p.scale_f16;
    rp.per_channel = i4 ? 0u : 1u;
    rp.row_scale = row_scale;
    rp.partial = scratch;
    const uint64_t outs = static_cast<uint64_t>(m) * n_total;
    const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>((outs + 255) / 256, static_cast<uint64_t>(env.sm_count) * 8));
    e = int8 ? launch_dependent(exact_reduce_kernel<true>, dim3(grid), 256, 0, 1, env, rp)
             : launch_dependent(exact_reduce_kernel<false>, dim3(grid), 256, 0, 1, env, rp);
    if (e != cudaSuccess) return e;
    if (launches) *launches += 1;
  }
  return cudaSuccess;
}

uint64_t align256(uint64_t v) { return (v + 255) & ~uint64_t(255); }

}  // namespace

bool qgemm_exact_supports(int count, const LinearTarget* targets, uint32_t m, uint64_t workspace_bytes) {
  if (count < 1 || count > kMaxMulti || m == 0) return false;
  const Weight& w0 = *targets[0].w;
  // Tiled layouts have GEMVs of their own up to 16 rows.  A single untiled weight has kq_qgemv_rows.cu, whose line to this
  // kernel is drawn there; several of them (q|k|v), and rows that it does not hold, come here from the amount of work on
  // at which the generic kernel (one warp per channel) is behind: 13.5 us for anything up to 1 x 4096 -> 1000, then
  // 26 us for 1 x 4096 -> 4096 int4 (here 22) or 35 us int8 (here 19), and 242 us at 16 rows (here 25).
  uint64_t work = 0;
  for (int i = 0; i < count; ++i) work += static_cast<uint64_t>(m) * targets[i].w->n * w0.k;
  if (w0.layout != kLayoutNative ? m <= 16 : work < (w0.storage == KQ_STORAGE_I4 ? 12u << 20 : 8u << 20)) return false;
  for (int i = 0; i < count; ++i) {
    const Weight& w = *targets[i].w;
    if (w.layout != w0.layout || w.storage != w0.storage || w.k != w0.k || w.group_size != w0.group_size ||
        w.scale_dtype != w0.scale_dtype || w.k == 0 || !kind_ok(w))
      return false;
  }
  // a panel of 16 rows of split activations and its factors have to fit the scratch
  return align256(static_cast<uint64_t>(w0.k) * 2 * parts_of(kBf3) * 16) + 256 <= workspace_bytes;
}

uint64_t qgemm_exact_clocks(const LaunchEnv& env, const Weight& w, int x_dtype, uint32_t m) {
  const bool int8_weights = w.storage == KQ_STORAGE_I8;
  const int math = math_of(x_dtype, w);
  uint32_t slots[kMaxClusterSplits + 1];
  if (resident_pairs(env, slots) != cudaSuccess) return 0;
  return choose_geometry(m, w.n, (w.n + 2 * kRows - 1) / (2 * kRows), steps_of(w.k, math, int8_weights ? 0 : w.group_size, chain_of(math, int8_weights)), math,
                         int8_weights, true, slots, env.workspace != nullptr ? env.workspace_bytes : 0).clocks;
}

// A gate and its up projection in one launch, silu(gate) * up written by the epilogue, where the tiles fill half of the
// device; below that the two are worth cutting along K (the gate's own kernel then follows the matmul).
bool qgemm_exact_fuses_gate(const LaunchEnv& env, uint32_t n, uint32_t m) {
  return static_cast<uint64_t>((n + kRows - 1) / kRows) * ((m + kMaxNT - 1) / kMaxNT) * 4 >= static_cast<uint64_t>(env.sm_count);
}

cudaError_t launch_qgemm_exact(const LaunchEnv& env, int count, const LinearTarget* targets, const void* x, int x_dtype, uint32_t m,
                               bool swiglu, int* launches) {
  const Weight& w0 = *targets[0].w;
  const uint32_t k = w0.k;
  const bool direct = x_dtype == KQ_F16;  // binary16 rows are the operand
  if ((direct && env.norm_weight != nullptr) || (swiglu && (count != 2 || targets[0].w->n != targets[1].w->n || env.residual != nullptr)))
    return cudaErrorInvalidValue;
  const int math = math_of(x_dtype, w0);
  uint8_t* ws = static_cast<uint8_t*>(env.workspace);
  const uint64_t room = env.workspace != nullptr ? env.workspace_bytes : 0;
  // row panels whose split activations take at most three quarters of the scratch (the rest: partial sums, which
  // only calls of few tiles want)
  const uint64_t part_bytes = static_cast<uint64_t>(k) * 2 * parts_of(math), per_row = part_bytes + 4, share = room / 4 * 3;
  uint32_t panel = m;
  if (!direct && per_row * m > share) {
    panel = static_cast<uint32_t>(std::min<uint64_t>(m, std::max<uint64_t>(16, share / per_row)));
    if (panel >= 256) panel = panel / 256 * 256;
  }
  for (uint32_t r0 = 0; r0 < m; r0 += panel) {
    const uint32_t pm = std::min(panel, m - r0);
    LinearTarget t[kMaxMulti];
    for (int i = 0; i < count; ++i)
      t[i] = LinearTarget{targets[i].w, targets[i].bias, targets[i].out + static_cast<size_t>(r0) * targets[i].w->n};
    const float* residual = env.residual != nullptr ? env.residual + static_cast<size_t>(r0) * w0.n : nullptr;
    const uint32_t xb = x_dtype == KQ_F32 ? 4 : 2;
    const uint8_t* xp = static_cast<const uint8_t*>(x) + static_cast<size_t>(r0) * k * xb;
    cudaError_t e;
    if (direct) {
      e = run_exact(env, count, t, residual, xp, math, pm, chain_of(math, w0.storage == KQ_STORAGE_I8), nullptr, ws, room, true, swiglu, launches);
    } else {
      float* inv = reinterpret_cast<float*>(ws);
      uint16_t* parts = reinterpret_cast<uint16_t*>(ws + align256(static_cast<uint64_t>(pm) * 4));
      const uint64_t taken = align256(static_cast<uint64_t>(pm) * 4) + align256(pm * part_bytes);
      if (taken > room) return cudaErrorMemoryAllocation;
      auto split = [&](auto* rows, auto form) {
        using XT = std::remove_const_t<std::remove_pointer_t<decltype(rows)>>;
        constexpr int kForm = decltype(form)::value;
        auto launch = [&](auto kernel) {
          return launch_dependent(kernel, dim3(pm), 256, 0, 1, env, rows, pm, k, parts, inv, env.norm_weight, env.norm_eps);
        };
        if (k <= 2048) return launch(split_kernel<XT, kForm, 1>);
        if (k <= 4096) return launch(split_kernel<XT, kForm, 2>);
        if (k <= 16384) return launch(split_kernel<XT, kForm, 8>);
        return launch(split_kernel<XT, kForm, 0>);
      };
      if (math == kBf1) e = split(reinterpret_cast<const __nv_bfloat16*>(xp), std::integral_constant<int, kBf1>{});
      else if (math == kBf3) e = split(reinterpret_cast<const float*>(xp), std::integral_constant<int, kBf3>{});
      else e = split(reinterpret_cast<const float*>(xp), std::integral_constant<int, kHalf2>{});
      if (e != cudaSuccess) return e;
      if (launches) *launches += 1;
      e = run_exact(env, count, t, residual, parts, math, pm, chain_of(math, w0.storage == KQ_STORAGE_I8), inv, ws + taken, room - taken, true, swiglu, launches);
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Integer-dot form: int8 activations xq [m, k] with row scales xs.
bool qgemm_exact_a8_preferred(const Weight& w, uint32_t m) {
  // (us, the mma.sync kernel | here)  The mma.sync kernel streams a matrix of any size, this one starts over with
  // every wave of 74 CTA pairs (18,944 channels).
  //   int4, up to eight rows   the ascending fma chain over the groups allows no K split here, so one wave and no
  //                            more: 1 x 4096 -> 4096 43 | 29, 8 x 4096 -> 14336 47 | 30, 8 x 1536 -> 1024 14 | 15, but
  //                            8 x 1024 -> 32768 19 | 23, 8 x 4096 -> 65536 88 | 111
  //   int8, up to eight rows   1 x 256 -> 4096 7.4 | 4.6, 1 x 4096 -> 4096 41 | 10, 8 x 1536 -> 32768 22 | 18, but
  //                            1 x 1536 -> 65536 24 | 35, -> 151936 45 | 72
  //   nine to sixteen          are two launches there, which pay for many waves only with a short k: 12 x 256 ->
  //                            151936 26 | 48 (int4 29 | 59), 12 x 1024 -> 65536 33 | 32 (int4 49 | 44)
  //   untiled                  the generic kernel (0.09 us per k) only below k = 128
  const bool many_waves = w.n > 49152, short_k = w.k < 512;
  if (w.layout == kLayoutTiledI4) return m > 16 || (m > 8 ? !(many_waves && short_k) : w.n <= 18944);
  if (w.layout == kLayoutTiledI8) return m > 16 || !many_waves || (m > 8 && !short_k) || w.k > 65536;  // (its sums end at k = 65536)
  return w.k >= 128;
}
bool qgemm_exact_a8_supports(const Weight& w, const int8_t* xq, uint32_t m, uint64_t workspace_bytes) {
  if (m == 0 || w.k == 0 || !kind_ok(w) || w.k % 16 != 0 || (reinterpret_cast<uintptr_t>(xq) & 15u) != 0) return false;
  if (w.storage == KQ_STORAGE_I8) return true;
  return w.group_size <= kMaxChain && align256(static_cast<uint64_t>(w.k) * 2 * 32) <= workspace_bytes;
}

cudaError_t launch_qgemm_exact_a8(const LaunchEnv& env, const LinearTarget& target, const int8_t* xq, const float* xs, uint32_t m,
                                  int* launches) {
  const Weight& w = *target.w;
  uint8_t* ws = static_cast<uint8_t*>(env.workspace);
  const uint64_t room = env.workspace != nullptr ? env.workspace_bytes : 0;
  if (w.storage == KQ_STORAGE_I8) return run_exact(env, 1, &target, nullptr, xq, kInt8, m, kMaxChain, xs, ws, room, true, false, launches);
  // int4: per-group sums as binary16 products (exact), flushed in ascending order: no K slices
  const uint64_t per_row = static_cast<uint64_t>(w.k) * 2;
  uint32_t panel = static_cast<uint32_t>(std::min<uint64_t>(m, room / per_row));
  if (panel < m && panel >= 256) panel = panel / 256 * 256;
  if (panel == 0) return cudaErrorMemoryAllocation;
  for (uint32_t r0 = 0; r0 < m; r0 += panel) {
    const uint32_t pm = std::min(panel, m - r0);
    const uint64_t sixteens = static_cast<uint64_t>(pm) * w.k / 16;
    const uint32_t grid = static_cast<uint32_t>(std::min<uint64_t>((sixteens + 255) / 256, static_cast<uint64_t>(env.sm_count) * 16));
    cudaError_t e = launch_dependent(bytes_to_half_kernel, dim3(grid), 256, 0, 1, env, xq + static_cast<size_t>(r0) * w.k, sixteens,
                                     reinterpret_cast<__half*>(ws));
    if (e != cudaSuccess) return e;
    if (launches) *launches += 1;
    const LinearTarget t{target.w, target.bias, target.out + static_cast<size_t>(r0) * w.n};
    e = run_exact(env, 1, &t, nullptr, ws, kHalf1, pm, kMaxChain, xs + r0, nullptr, 0, false, false, launches);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace kq
