// qgemv_i4_xs — the decode linear for 1 to 16 activation rows with the activations held in
// REGISTERS:  y[m, n] = x[m, k] . W[n, k]^T + b, W in the tiled int4 / group-32 layout.
//
// Replaces the reference's small-M linear with in-kernel int4 dequant (pipeline key
// linear:v2:f32:reg16x16r1x4w4:wi4g32 — packages/runtime/src/kernels/gemm.ts:1187-1237, geometry
// packages/runtime/src/kernels/gemm-geometry.ts:243) and, around it, the rms_norm, the SiLU gate and
// the residual add of a decoder layer (packages/runtime/src/kernels/rms-norm.ts:60-90,
// packages/runtime/src/runtime/fusion.ts:453-511): one launch per matmul of a decode step.
//
// The arithmetic is that of kq_qgemv_i4.cu (nibble pairs as binary16 subnormals into mma.sync, the
// -8 as the accumulator's initial value, group scales in f32); what differs is who holds what.  A
// kernel whose warps walk along k for a few rows converts the activations in every CTA (or in a
// launch of its own), reads them from shared memory for every chunk of weights, and at 16 rows
// does little else.  Here a warp owns a SLAB of 128 k (64 k above eight rows) for the whole launch:
// its B fragments are built once, straight from x, and the warp then streams the 16-row blocks of
// the weight past them.  Per 576-byte chunk that leaves the weight load, the unpack, the MMAs and
// the scale.
//   * The power-of-two pre-scale is per (row, slab), so it costs one multiply per partial sum.
//   * rms_norm: the CTAs of a cluster share out the rows' sums of squares while the first weights are on
//     their way; what is staged is (x r) g as the reference computes it.
//   * The slabs of a CTA meet in shared memory, a batch of row blocks at a time, in slab order; a k
//     longer than a CTA's 16 slabs is spread over a thread-block cluster, whose CTAs add their
//     sums over distributed shared memory in rank order once per launch (and over several passes
//     where that is not enough).  No atomics: the same bits every time.
//
// What bounds it: the legacy mma.sync rate (one m16n8k16 per two clocks and SM; 16 a chunk for 16 f32
// rows is 5 TB/s of weights) and its issue slots for a large matrix; launch and load latency for the
// small matrices of a layer.
#include <algorithm>
#include <type_traits>

#include "kq_gemv_core.cuh"
#include "kq_internal.h"

namespace kq {
namespace {

constexpr int kXsWarps = 16, kXsThreads = kXsWarps * 32;
constexpr int kXsAhead = 4;            // row blocks a warp has in flight, in registers (two: 15 % slower on a large matrix)
constexpr uint32_t kXsMaxCluster = 8;
constexpr uint32_t kXsHead = 1024;     // sums of squares, row factors
constexpr uint32_t kXsSmem = 227 * 1024;

// How the columns of a warp's MMA tiles are used:
//   kPacked  up to four f32 / bf16 rows: columns 2r and 2r + 1 = the high and the low part of row r (one MMA carries
//            both, one lane holds both sums); a warp's slab is 128 k
//   kEight   up to eight rows, column c = row c, the low parts a second B operand; 128 k
//   kSixteen up to sixteen rows, two tiles: the nibbles are unpacked once for both; 64 k, so that the fragments
//            take the same registers
enum XsForm : int { kPacked, kEight, kSixteen };
template <int kForm>
struct XsShape {
  static constexpr uint32_t tiles = kForm == kSixteen ? 2 : 1, slab_chunks = kForm == kSixteen ? 1 : 2;
  static constexpr uint32_t sums = kForm == kPacked ? 64 : 128 * tiles;  // finished sums of a 16-row block
  static constexpr uint32_t batch = kForm == kPacked ? 8 : 4;            // row blocks per reduction
  static constexpr uint32_t red_bytes = 2u * batch * kXsWarps * sums * 4u;  // [buffer][block][warp][sums]
  static constexpr uint32_t part_blocks = (kXsSmem - kXsHead - red_bytes) / (sums * 4u);  // row blocks a CTA can hold the sums of
};

struct XsParams {
  const uint8_t* w[kMaxMulti];
  const float* bias[kMaxMulti];
  float* out[kMaxMulti];
  uint32_t n[kMaxMulti];
  uint32_t unit_begin[kMaxMulti + 1];  // units = 16-row blocks of all weights (SiLU gate: block pairs gate j, up j)
  uint32_t count, units, swiglu;
  const void* x;
  uint32_t m, k;
  const float* norm_weight;
  float norm_eps;
  const float* residual;
  uint32_t cluster;   // CTAs that share a row block's k
  uint32_t passes;    // ... and how often each comes back for more of it
  uint32_t clusters;
};

__device__ __forceinline__ uint4 xs_ldg128(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 xs_ldg64(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float xs_ld_rank(uint32_t addr, uint32_t rank) {
  float v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
               : "=f"(v) : "r"(addr), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t xs_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// D = A.B + C, C in registers that are not overwritten
__device__ __forceinline__ void xs_mma_from(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, const float (&c)[4]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void xs_mma_add(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool kScaleF16>
struct XsChunk {
  uint4 w;
  typename std::conditional<kScaleF16, uint2, uint4>::type s;
};

template <typename XT, bool kScaleF16, int kForm>
__global__ void __launch_bounds__(kXsThreads, 1) qgemv_i4_xs_kernel(const XsParams p) {
  constexpr bool kHasLo = !std::is_same<XT, __half>::value;
  constexpr bool kPackLo = kForm == kPacked, kLoSet = kHasLo && !kPackLo;
  using Shape = XsShape<kForm>;
  constexpr uint32_t kTiles = Shape::tiles, kSlabChunks = Shape::slab_chunks, kSums = Shape::sums;
  constexpr int kGroups = 2 * kSlabChunks, kBatch = Shape::batch;
  static_assert(kHasLo || !kPackLo, "binary16 activations have no low part");
  static_assert(kXsThreads * kTiles == kBatch * kSums && kBatch % kXsAhead == 0, "the reduction's thread layout");
  constexpr uint32_t kCB = kChunkWeightBytes + 32u * (kScaleF16 ? 2u : 4u);
  constexpr uint32_t kMask0 = 0x000F000Fu, kMask1 = 0x00F000F0u;
  extern __shared__ __align__(16) uint8_t smem[];
  float* squares = reinterpret_cast<float*>(smem);           // [18 rows][8 warps] sums of squares
  float* row_factor = squares + 18 * 8;                      // [16] the rows' rsqrt
  float* red = reinterpret_cast<float*>(smem + kXsHead);
  float* part = reinterpret_cast<float*>(smem + kXsHead + Shape::red_bytes);  // [block][sums]
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
  const uint32_t rank = p.cluster > 1 ? xs_rank() : 0u, cluster_id = blockIdx.x / p.cluster;
  const uint32_t chunks = p.k / kChunkK, per_unit = p.swiglu ? 2u : 1u;
  const uint32_t unit_first = static_cast<uint32_t>(static_cast<uint64_t>(p.units) * cluster_id / p.clusters);
  const uint32_t unit_last = static_cast<uint32_t>(static_cast<uint64_t>(p.units) * (cluster_id + 1) / p.clusters);
  const uint32_t round_units = Shape::part_blocks / per_unit;

  pdl_launch_dependents();

  for (uint32_t u0 = unit_first; u0 < unit_last; u0 += round_units) {
    const uint32_t units_now = min(round_units, unit_last - u0), blocks = units_now * per_unit;
    for (uint32_t pass = 0; pass < p.passes; ++pass) {
      const uint32_t chunk0 = ((pass * p.cluster + rank) * kXsWarps + warp) * kSlabChunks;  // this warp's slab
      const uint32_t live = chunk0 < chunks ? min(kSlabChunks, chunks - chunk0) : 0u;
      // ---- the weight stream: this lane's words of a row block, kXsAhead blocks ahead ----
      // Row blocks of one weight follow one another in memory, so the next address is one addition; only
      // where the list passes to the next weight is it looked up.  A warp whose slab is cut short by the
      // end of k reads chunks it has no activations for: their fragments are zero.
      XsChunk<kScaleF16> ring[kXsAhead][kSlabChunks];
      const size_t stride = static_cast<size_t>(chunks) * kCB;
      const uint32_t first_chunk = min(chunk0, chunks - 1u), second = first_chunk + 1u < chunks ? kCB : 0u;
      const uint32_t scale_off = kChunkWeightBytes + g * (kScaleF16 ? 8u : 16u);
      const size_t gate_to_up = p.swiglu ? static_cast<size_t>(p.w[1] - p.w[0]) : 0;
      const uint8_t* next = nullptr;  // chunk `first_chunk` of the next row block to fetch
      uint32_t next_unit = u0, weight_end = 0;
      auto seek = [&]() {
        uint32_t wi = 0;
#pragma unroll
        for (int i = 1; i < kMaxMulti; ++i)
          if (i < static_cast<int>(p.count) && next_unit >= p.unit_begin[i] && !p.swiglu) wi = i;
        weight_end = p.swiglu ? p.units : p.unit_begin[wi + 1];
        next = p.w[wi] + (next_unit - p.unit_begin[wi]) * stride + static_cast<size_t>(first_chunk) * kCB;
      };
      seek();
      auto fetch = [&](XsChunk<kScaleF16> (&dst)[kSlabChunks], bool up) {
        const uint8_t* src = up ? next + gate_to_up : next;
        const uint8_t *w_at = src + lane * 16, *s_at = src + scale_off;
        dst[0].w = xs_ldg128(w_at);
        if constexpr (kScaleF16) dst[0].s = xs_ldg64(s_at);
        else dst[0].s = xs_ldg128(s_at);
        if constexpr (kSlabChunks == 2) {
          dst[1].w = xs_ldg128(w_at + second);
          if constexpr (kScaleF16) dst[1].s = xs_ldg64(s_at + second);
          else dst[1].s = xs_ldg128(s_at + second);
        }
        if (up || !p.swiglu) {
          next += stride;
          if (++next_unit == weight_end) seek();
        }
      };
#pragma unroll
      for (int i = 0; i < kXsAhead; ++i) {
#pragma unroll
        for (uint32_t c = 0; c < kSlabChunks; ++c) {
          ring[i][c].w = make_uint4(0, 0, 0, 0);
          if constexpr (kScaleF16) ring[i][c].s = make_uint2(0, 0);
          else ring[i][c].s = make_uint4(0, 0, 0, 0);
        }
        if (static_cast<uint32_t>(i) < blocks) fetch(ring[i], p.swiglu && (i & 1));
      }
      // nothing the previous kernel writes has been touched so far
      if (pass == 0 && u0 == unit_first) pdl_wait_prior_grid();

      // ---- the slab's activations as B fragments ----
      // lane (g, t) prepares B column g (k-octet t of every group) of each tile
      auto row_of = [&](uint32_t tl) { return kPackLo ? g >> 1 : tl * 8u + g; };
      float v[kTiles][kGroups][8];
      auto load_slab = [&](uint32_t tl, uint32_t chunk, uint32_t chunks_live, float (&dst)[kGroups][8]) {
        const uint32_t row = row_of(tl);
        const XT* xr = static_cast<const XT*>(p.x) + static_cast<size_t>(row < p.m ? row : 0u) * p.k + chunk * kChunkK + t * 8u;
#pragma unroll
        for (int j = 0; j < kGroups; ++j) {
#pragma unroll
          for (int e = 0; e < 8; ++e) dst[j][e] = 0.0f;
          if (row < p.m && static_cast<uint32_t>(j) < 2 * chunks_live) load_x8<XT, true>(xr + j * 32, dst[j]);
        }
      };
#pragma unroll
      for (uint32_t tl = 0; tl < kTiles; ++tl) load_slab(tl, chunk0, live, v[tl]);
      if (p.norm_weight != nullptr) {
        if (pass == 0 && u0 == unit_first) {
          // The rows' factors: rows are dealt to the cluster's CTAs, 256 threads a row (shuffle tree, warps in
          // order), and the CTAs exchange the results.  One order whatever the cut of k, and that of the kernels
          // which do the norm elsewhere (rms_norm_kernel up to four rows, stage_x_global_kernel above): the same
          // bits.  A norm factor one ulp off is an error common to a whole row, which a chain of layers amplifies.
          const uint32_t half = threadIdx.x >> 8, th = threadIdx.x & 255u;
          for (uint32_t r0 = rank * 2u; r0 < p.m; r0 += p.cluster * 2u) {
            const uint32_t row = r0 + half;
            float sq = 0.0f;
            const XT* xr = static_cast<const XT*>(p.x) + static_cast<size_t>(row) * p.k;
            if (row < p.m && kPackLo) {
#pragma unroll 8
              for (uint32_t i = th; i < p.k; i += 256u) {
                const float u = to_f32(xr[i]);
                sq = fmaf(u, u, sq);
              }
            } else if (row < p.m) {
#pragma unroll 2
              for (uint32_t i = th * 8u; i < p.k; i += 2048u) {
                float u[8];
                load_x8<XT, true>(xr + i, u);
#pragma unroll
                for (int e = 0; e < 8; ++e) sq = fmaf(u[e], u[e], sq);
              }
            }
            sq = warp_sum(sq);
            if (lane == 0) squares[row * 8u + (warp & 7u)] = sq;  // rows up to m rounded up: 18 at most
          }
          __syncthreads();
          const uint32_t mine = (threadIdx.x >> 1) % p.cluster;  // rows 2r, 2r + 1 belong to rank r % cluster
          if (threadIdx.x < p.m && mine == rank) {
            float total = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) total += squares[threadIdx.x * 8 + w];
            row_factor[threadIdx.x] = rsqrtf(total * (1.0f / static_cast<float>(p.k)) + p.norm_eps);
          }
          if (p.cluster > 1) {
            cluster_sync_all();
            if (threadIdx.x < p.m && mine != rank)
              row_factor[threadIdx.x] = xs_ld_rank(static_cast<uint32_t>(__cvta_generic_to_shared(row_factor + threadIdx.x)), mine);
          }
          __syncthreads();
        }
        const float* gr = p.norm_weight + chunk0 * kChunkK + t * 8u;
#pragma unroll
        for (int j = 0; j < kGroups; ++j) {
          if (static_cast<uint32_t>(j) < 2 * live) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(gr + j * 32)), b = __ldg(reinterpret_cast<const float4*>(gr + j * 32 + 4));
            const float gw[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (uint32_t tl = 0; tl < kTiles; ++tl) {
              const float r = row_of(tl) < p.m ? row_factor[row_of(tl)] : 0.0f;
#pragma unroll
              for (int e = 0; e < 8; ++e) v[tl][j][e] = __fmul_rn(__fmul_rn(v[tl][j][e], r), gw[e]);
            }
          }
        }
      }
      uint4 bhi[kTiles][kGroups], blo[kTiles][kLoSet ? kGroups : 1];
      // -8 sum x of the lane's C columns: the MMA's C operand (rows g and g + 8 alike); packed: one value, added in f32
      float cterm[kTiles][kGroups][kPackLo ? 1 : 4], inv[kTiles][2];  // ... and the columns' 2^-e
#pragma unroll
      for (uint32_t tl = 0; tl < kTiles; ++tl) {
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < kGroups; ++j) amax = fmaxf(amax, absmax8(v[tl][j]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const Pow2 ps = pow2_prescale(amax);
        const float odd_scale = ps.scale * 0.0625f;  // odd k-slots: their nibbles come as u * 2^-20
#pragma unroll
        for (int j = 0; j < kGroups; ++j) {
          __half h[8], l[8];
          float sum = 0.0f;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float staged = v[tl][j][e] * ((e & 1) ? odd_scale : ps.scale);
            h[e] = __float2half_rn(staged);
            float used = __half2float(h[e]);
            if constexpr (kHasLo) {
              l[e] = __float2half_rn(staged - used);
              used += __half2float(l[e]);
              if (kPackLo && (g & 1u)) h[e] = l[e];
            }
            sum = fmaf(used, (e & 1) ? 16.0f : 1.0f, sum);
          }
          bhi[tl][j] = make_uint4(pack_half2(h[0], h[4]), pack_half2(h[1], h[5]), pack_half2(h[2], h[6]), pack_half2(h[3], h[7]));
          if constexpr (kLoSet)
            blo[tl][j] = make_uint4(pack_half2(l[0], l[4]), pack_half2(l[1], l[5]), pack_half2(l[2], l[6]), pack_half2(l[3], l[7]));
          sum += __shfl_xor_sync(0xffffffffu, sum, 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          // column c's sum sits in the lanes of g == c; this lane's C columns are 2t and 2t + 1
          const float c0 = __shfl_sync(0xffffffffu, sum, 8 * t) * (-8.0f / kUnscale);
          if constexpr (kPackLo) {
            cterm[tl][j][0] = c0;
          } else {
            cterm[tl][j][0] = cterm[tl][j][2] = c0;
            cterm[tl][j][1] = cterm[tl][j][3] = __shfl_sync(0xffffffffu, sum, 8 * t + 4) * (-8.0f / kUnscale);
          }
        }
        inv[tl][0] = __shfl_sync(0xffffffffu, ps.inv, 8 * t);
        inv[tl][1] = __shfl_sync(0xffffffffu, ps.inv, 8 * t + 4);
      }

      // ---- stream the row blocks ----
      for (uint32_t b0 = 0; b0 < blocks; b0 += kBatch) {
        float* red_now = red + ((b0 / kBatch) & 1u) * (kBatch * kXsWarps * kSums);
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const uint32_t b = b0 + i;
          if (b >= blocks) break;
          float acc[kTiles][4];
#pragma unroll
          for (uint32_t tl = 0; tl < kTiles; ++tl)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[tl][e] = 0.0f;
#pragma unroll
          for (uint32_t c = 0; c < kSlabChunks; ++c) {
            const XsChunk<kScaleF16> ch = ring[i % kXsAhead][c];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              const int j = 2 * c + jj;
              const uint32_t wa = jj ? ch.w.z : ch.w.x, wb = jj ? ch.w.w : ch.w.y;  // rows g, g + 8
              const uint32_t wa8 = wa >> 8, wb8 = wb >> 8;
              const uint32_t a0[4] = {wa & kMask0, wb & kMask0, wa & kMask1, wb & kMask1};
              const uint32_t a1[4] = {wa8 & kMask0, wb8 & kMask0, wa8 & kMask1, wb8 & kMask1};
              float2 s;
              if constexpr (kScaleF16) s = __half22float2(*reinterpret_cast<const __half2*>(jj ? &ch.s.y : &ch.s.x));
              else s = jj ? make_float2(__uint_as_float(ch.s.z), __uint_as_float(ch.s.w)) : make_float2(__uint_as_float(ch.s.x), __uint_as_float(ch.s.y));
              // (the tiles' chains side by side: each MMA of a chain waits for the one before it)
              float cf[kTiles][4];
              if constexpr (kPackLo) {
                mma_f16_zero(cf[0], a0, bhi[0][j].x, bhi[0][j].y);
                xs_mma_add(cf[0], a1, bhi[0][j].z, bhi[0][j].w);
                acc[0][0] = fmaf(s.x, (cf[0][0] + cf[0][1]) + cterm[0][j][0], acc[0][0]);
                acc[0][1] = fmaf(s.y, (cf[0][2] + cf[0][3]) + cterm[0][j][0], acc[0][1]);
              } else {
#pragma unroll
                for (uint32_t tl = 0; tl < kTiles; ++tl) xs_mma_from(cf[tl], a0, bhi[tl][j].x, bhi[tl][j].y, cterm[tl][j]);
#pragma unroll
                for (uint32_t tl = 0; tl < kTiles; ++tl) xs_mma_add(cf[tl], a1, bhi[tl][j].z, bhi[tl][j].w);
                if constexpr (kLoSet) {
#pragma unroll
                  for (uint32_t tl = 0; tl < kTiles; ++tl) xs_mma_add(cf[tl], a0, blo[tl][j].x, blo[tl][j].y);
#pragma unroll
                  for (uint32_t tl = 0; tl < kTiles; ++tl) xs_mma_add(cf[tl], a1, blo[tl][j].z, blo[tl][j].w);
                }
#pragma unroll
                for (uint32_t tl = 0; tl < kTiles; ++tl) {
                  acc[tl][0] = fmaf(s.x, cf[tl][0], acc[tl][0]);
                  acc[tl][1] = fmaf(s.x, cf[tl][1], acc[tl][1]);
                  acc[tl][2] = fmaf(s.y, cf[tl][2], acc[tl][2]);
                  acc[tl][3] = fmaf(s.y, cf[tl][3], acc[tl][3]);
                }
              }
            }
          }
          if (b + kXsAhead < blocks) fetch(ring[i % kXsAhead], p.swiglu && (i & 1));
          float* mine = red_now + (i * kXsWarps + warp) * kSums;
          if constexpr (kPackLo) {
            reinterpret_cast<float2*>(mine)[lane] = make_float2(acc[0][0] * inv[0][0], acc[0][1] * inv[0][0]);
          } else {
#pragma unroll
            for (uint32_t tl = 0; tl < kTiles; ++tl)
              reinterpret_cast<float4*>(mine + tl * 128)[lane] =
                  make_float4(acc[tl][0] * inv[tl][0], acc[tl][1] * inv[tl][1], acc[tl][2] * inv[tl][0], acc[tl][3] * inv[tl][1]);
          }
        }
        __syncthreads();
        // the slabs' sums meet, in slab order; the next batch goes to the other buffer
        // (thread = one of a tile's sums of one block of the batch, in every tile)
        constexpr uint32_t kTileSums = kSums / kTiles;
        const uint32_t bi = threadIdx.x / kTileSums, o = threadIdx.x % kTileSums;
        if (b0 + bi < blocks) {
          const float* src = red_now + bi * (kXsWarps * kSums) + o;
          float* dst = part + (b0 + bi) * kSums + o;
#pragma unroll
          for (uint32_t tl = 0; tl < kTiles; ++tl) {
            float sum = 0.0f;
#pragma unroll
            for (int s = 0; s < kXsWarps; ++s) sum += src[s * kSums + tl * 128];
            dst[tl * 128] = pass == 0 ? sum : dst[tl * 128] + sum;
          }
        }
      }
      if (p.passes > 1) __syncthreads();  // the reduction buffers are free for the next pass
    }

    // ---- the cluster's sums meet, in rank order, and leave with the neighbours applied ----
    if (p.cluster > 1) cluster_sync_all();
    else __syncthreads();
    const uint32_t part_addr = static_cast<uint32_t>(__cvta_generic_to_shared(part));
    const uint32_t outs = units_now * p.m * 16u;
    for (uint32_t idx = rank * kXsThreads + threadIdx.x; idx < outs; idx += p.cluster * kXsThreads) {
      const uint32_t r = idx & 15u, um = idx >> 4, ul = um / p.m, mm = um - ul * p.m, unit = u0 + ul;
      const uint32_t col = mm & 7u, tl = mm >> 3;
      // output (row r, column c) of a tile: lane (r & 7, c / 2), element 2 (r / 8) + c % 2; packed: lane (r & 7, row), element r / 8
      const uint32_t o = kPackLo ? ((r & 7u) * 4u + col) * 2u + (r >> 3) : tl * 128u + ((r & 7u) * 4u + (col >> 1)) * 4u + (r >> 3) * 2u + (col & 1u);
      auto total_of = [&](uint32_t block) {
        const uint32_t at = block * kSums + o;
        if (p.cluster == 1) return part[at] * kUnscale;
        float sum = 0.0f;
        for (uint32_t c = 0; c < p.cluster; ++c) sum += xs_ld_rank(part_addr + at * 4u, c);
        return sum * kUnscale;
      };
      if (p.swiglu) {
        const uint32_t row = unit * 16u + r;
        const float gate = total_of(2 * ul) + p.bias[0][row], up = total_of(2 * ul + 1) + p.bias[1][row];
        p.out[0][static_cast<size_t>(mm) * p.n[0] + row] = silu_mul(gate, up);
      } else {
        uint32_t wi = 0;
#pragma unroll
        for (int i = 1; i < kMaxMulti; ++i)
          if (i < static_cast<int>(p.count) && unit >= p.unit_begin[i]) wi = i;
        const uint32_t row = (unit - p.unit_begin[wi]) * 16u + r;
        float v = total_of(ul) + p.bias[wi][row];
        const size_t at = static_cast<size_t>(mm) * p.n[wi] + row;
        if (p.residual != nullptr) v = __fadd_rn(v, p.residual[at]);
        p.out[wi][at] = v;
      }
    }
    if (p.cluster > 1) cluster_sync_all();  // nobody's sums go away while a peer still reads them
    else __syncthreads();
  }
}

// Clusters of this size the device holds at once (0: the query failed).
template <typename Kernel>
uint32_t resident_clusters(Kernel kernel, uint32_t cluster, int sm_count) {
  if (cluster == 1) return static_cast<uint32_t>(sm_count);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(kXsThreads);
  cfg.dynamicSmemBytes = kXsSmem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = cluster;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 0) {
    (void)cudaGetLastError();
    n = 0;
  }
  return static_cast<uint32_t>(n);
}

template <typename XT, bool kScaleF16, int kForm>
cudaError_t launch_xs(const LaunchEnv& env, XsParams& p) {
  auto kernel = qgemv_i4_xs_kernel<XT, kScaleF16, kForm>;
  using Shape = XsShape<kForm>;
  constexpr uint32_t kSlabChunks = Shape::slab_chunks;
  struct Setup { uint32_t resident[kXsMaxCluster + 1]; };
  static PerDevice<Setup> setup_on;
  const Setup* setup = nullptr;
  const cudaError_t ready = setup_on.get([&](Setup& s) -> cudaError_t {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kXsSmem));
    if (e != cudaSuccess) return e;
    for (uint32_t c = 1; c <= kXsMaxCluster; ++c) s.resident[c] = resident_clusters(kernel, c, env.sm_count);
    return cudaSuccess;
  }, &setup);
  if (ready != cudaSuccess) return ready;
  // How many CTAs share a row block's k: the cluster size with the shortest longest list of (row block, pass)
  // pairs; a pass costs about two blocks (building the fragments), a cluster about one (its barriers).
  const uint32_t slabs = (p.k / kChunkK + kSlabChunks - 1) / kSlabChunks, per_unit = p.swiglu ? 2u : 1u;
  uint32_t best = ~0u;
  for (uint32_t c = 1; c <= kXsMaxCluster; ++c) {
    const uint32_t clusters = std::min(setup->resident[c], p.units);
    if (clusters == 0) continue;
    const uint32_t passes = (slabs + c * kXsWarps - 1) / (c * kXsWarps);
    const uint32_t cost = passes * ((p.units + clusters - 1) / clusters * per_unit + 2) + (c > 1 ? 1 : 0);
    if (cost < best) {
      best = cost;
      p.cluster = c;
      p.passes = passes;
      p.clusters = clusters;
    }
  }
  if (best == ~0u) return cudaErrorInvalidConfiguration;
  const uint32_t units_each = std::min((p.units + p.clusters - 1) / p.clusters, Shape::part_blocks / per_unit);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.clusters * p.cluster);
  cfg.blockDim = dim3(kXsThreads);
  cfg.dynamicSmemBytes = kXsHead + Shape::red_bytes + static_cast<size_t>(units_each) * per_unit * Shape::sums * 4;
  cfg.stream = env.stream;
  cudaLaunchAttribute attr[2];
  unsigned int na = 0;
  if (env.overlap) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (p.cluster > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.cluster;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}

template <typename XT>
cudaError_t launch_xs_typed(const LaunchEnv& env, XsParams& p, bool f16s) {
  if constexpr (!std::is_same<XT, __half>::value) {
    if (p.m <= 4) return f16s ? launch_xs<XT, true, kPacked>(env, p) : launch_xs<XT, false, kPacked>(env, p);
  }
  if (p.m <= 8) return f16s ? launch_xs<XT, true, kEight>(env, p) : launch_xs<XT, false, kEight>(env, p);
  return f16s ? launch_xs<XT, true, kSixteen>(env, p) : launch_xs<XT, false, kSixteen>(env, p);
}

}  // namespace

bool qgemv_i4_xs_supports(int count, const LinearTarget* targets, int x_dtype, uint32_t m) {
  if (count < 1 || count > kMaxMulti || m < 1 || m > 16) return false;
  if (x_dtype != KQ_F32 && x_dtype != KQ_F16 && x_dtype != KQ_BF16) return false;
  const Weight& w0 = *targets[0].w;
  for (int i = 0; i < count; ++i) {
    const Weight& w = *targets[i].w;
    if (w.layout != kLayoutTiledI4 || w.k != w0.k || w.scale_dtype != w0.scale_dtype || w.n == 0) return false;
  }
  return true;
}

// Which kernel a call of 1 .. 16 rows takes (us, f32 activations on distinct weights, this kernel | the others):
//   one row, two rows    4096 -> 4096 7.2 | 6.1 and 7.3 | 6.9; 8960 -> 1536 7.7 | 6.3: the group-packed kernel has
//                        less to set up.  With two rows it spends its MMAs on two groups at a time, and a matrix
//                        of 100 M weights is past its setup: 4096 -> 128256 65 | 87.  binary16 rows likewise,
//                        with twice the rows to a column.
//   three to sixteen     8 rows 4096 -> 4096 8.7 | 10.9, 8960 -> 1536 10.2 | 16.5; 16 rows 4096 -> 28672 43 | 54.
//                        From five rows on the wide kernel's many small CTAs stream a very large matrix
//                        faster: 4096 -> 128256 92 | 78 at eight rows, 72 | 66 with binary16.
//   with neighbours      this kernel is the whole launch sequence (a norm alone is 3 us), so the line for few
//                        rows only holds where the matrix is very large (one row, 63 | 54 + 3).
bool qgemv_i4_xs_preferred(int count, const LinearTarget* targets, int x_dtype, uint32_t m, bool norm_or_residual, bool swiglu) {
  if (!qgemv_i4_xs_supports(count, targets, x_dtype, m)) return false;
  if (swiglu) return true;
  uint64_t weights = 0;
  for (int i = 0; i < count; ++i) weights += static_cast<uint64_t>(targets[i].w->n) * targets[i].w->k;
  const uint32_t cols = x_dtype == KQ_F16 ? m : 2 * m;
  const bool very_large = weights > 200000000ull;
  if (cols <= 4) return cols <= 2 ? norm_or_residual && !very_large : norm_or_residual || weights > 100000000ull;
  return m < 5 || !very_large;
}

cudaError_t launch_qgemv_i4_xs(const LaunchEnv& env, int count, const LinearTarget* targets, const void* x, int x_dtype, uint32_t m,
                               bool swiglu, int* launches) {
  if (!qgemv_i4_xs_supports(count, targets, x_dtype, m) || (swiglu && count != 2)) return cudaErrorInvalidValue;
  XsParams p = {};
  p.count = static_cast<uint32_t>(count);
  for (int i = 0; i < count; ++i) {
    p.w[i] = static_cast<const uint8_t*>(targets[i].w->data);
    p.bias[i] = targets[i].bias;
    p.out[i] = targets[i].out;
    p.n[i] = targets[i].w->n;
    p.unit_begin[i] = p.units;
    p.units += targets[i].w->n / 16;
  }
  for (int i = count; i <= kMaxMulti; ++i) p.unit_begin[i] = p.units;
  p.swiglu = swiglu ? 1 : 0;
  if (swiglu) p.units = targets[0].w->n / 16;
  p.x = x;
  p.m = m;
  p.k = targets[0].w->k;
  p.norm_weight = env.norm_weight;
  p.norm_eps = env.norm_eps;
  p.residual = env.residual;
  const bool f16s = targets[0].w->scale_dtype == KQ_F16;
  cudaError_t e;
  switch (x_dtype) {
    case KQ_F32: e = launch_xs_typed<float>(env, p, f16s); break;
    case KQ_F16: e = launch_xs_typed<__half>(env, p, f16s); break;
    default: e = launch_xs_typed<__nv_bfloat16>(env, p, f16s); break;
  }
  if (e == cudaSuccess && launches) *launches += 1;
  return e;
}

}  // namespace kq
