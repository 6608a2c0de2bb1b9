// qgemv_rows — the linear for up to sixteen activation rows over weights that keep their row-major packing:
// int4 of any group size or ragged channel count, int8 with ragged channels (the tiled layouts take groups of 32
// and whole blocks of sixteen channels; kq_qgemv_i4*.cu, kq_qgemv_i8.cu).
//
// Replaces the reference's scalar and small-tile variants for those weights
// (packages/runtime/src/kernels/gemm-geometry.ts:243-267) and keeps their arithmetic: a weight is dequantised
// with one f32 multiply and enters an f32 multiply-add with the activation
// (packages/runtime/src/kernels/gemm.ts:642-718, :922-940).
//
// `lanes` threads share two channels' k: 16 bytes of each per step, loaded two steps in front of their use; the
// activations, up to four rows, lie in shared memory as f32.  Sixteen products are summed from zero and then added to the thread's sum; the threads meet in a shuffle tree and, above a warp, in warp order.
//
// What bounds it: instructions.  An int4 weight costs four (unpack, convert, scale) and one per activation row: one row of
// 1152 -> 60468 (46 MB with f32 scales) 19 us, where the generic kernel and the many-row one took 50; for small
// matrices the launch and two trips to memory (8064 -> 82: 12.8 us before, 5.2 now).
#include <type_traits>

#include "kq_common.cuh"
#include "kq_gemv_core.cuh"
#include "kq_internal.h"
#include "kq_rows_line.h"

namespace kq {
namespace {

constexpr uint32_t kRowsThreads = rows::kThreads, kRowsSmem = rows::kSmem;

rows::Call rows_call(const Weight& w, uint32_t m, int sm_count) {
  return rows::Call{w.storage == KQ_STORAGE_I4, w.n, w.k, m, static_cast<uint32_t>(sm_count)};
}

struct RowsParams {
  const uint8_t* w;
  const void* scale;
  const float* bias;
  float* out;
  const void* x;
  uint32_t m, n, k;
  uint32_t steps;       // 16-byte pieces of a channel
  uint32_t gshift;      // log2 of the group size (int4)
  uint32_t lanes_log2;  // threads that share two channels
  const float* norm_weight;  // null, or [k]: the f32 activations are rms-normalised as they are staged
  float norm_eps;
  const float* residual;  // null, or [m, n] added after the bias (may alias out)
};

__device__ __forceinline__ uint4 rows_ldg(const uint8_t* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// The weights of a word as f32, k ascending.
__device__ __forceinline__ void rows_nibbles(uint32_t w, float (&v)[8]) {
  __half2 h[4];
  nibble_pairs(w, h);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    v[i] = f.x;
    v[i + 4] = f.y;
  }
}
__device__ __forceinline__ void rows_bytes(uint32_t w, float* v) {
  __half2 h[2];
  byte_pairs(w ^ 0x80808080u, h);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float2 f = __half22float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

template <typename XT, bool kI8, bool kScaleF16, int kRowsX>
__global__ void __launch_bounds__(kRowsThreads, 2) qgemv_rows_kernel(const RowsParams p) {
  constexpr uint32_t kPer = kI8 ? 16u : 32u;  // weights of a step
  constexpr int kEights = kPer / 8;
  constexpr int kAhead = 2;  // steps of weights in flight besides the one at work
  __shared__ float part[kRowsThreads / 32][2 * kRowsX];
  __shared__ float row_norm[kRowsX];
  pdl_launch_dependents();
  const uint32_t m0 = blockIdx.y * kRowsX, live = min(p.m - m0, static_cast<uint32_t>(kRowsX));
  const uint32_t lanes = 1u << p.lanes_log2, me = threadIdx.x & (lanes - 1u);
  const uint32_t pair = blockIdx.x * (kRowsThreads >> p.lanes_log2) + (threadIdx.x >> p.lanes_log2);
  // (threads without a channel, or with one only, read the last channel's; they store nothing)
  const uint32_t ch[2] = {min(2u * pair, p.n - 1u), min(2u * pair + 1u, p.n - 1u)};
  const size_t row_bytes = static_cast<size_t>(p.steps) * 16u;
  const uint8_t* wr[2] = {p.w + ch[0] * row_bytes, p.w + ch[1] * row_bytes};
  const uint32_t groups = kI8 ? 1u : p.k >> p.gshift;

  struct Piece { uint4 w[2]; float s[2][2]; };
  auto fetch = [&](uint32_t step) {
    Piece q;
    const uint32_t at = min(step, p.steps - 1u);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      q.w[c] = rows_ldg(wr[c] + static_cast<size_t>(at) * 16u);
      if constexpr (kI8) {
        q.s[c][0] = q.s[c][1] = 1.0f;
      } else {
        const size_t g0 = static_cast<size_t>(ch[c]) * groups + ((at * kPer) >> p.gshift);
        q.s[c][0] = load_scale<kScaleF16>(p.scale, g0);
        q.s[c][1] = p.gshift == 4 ? load_scale<kScaleF16>(p.scale, g0 + 1u) : q.s[c][0];
      }
    }
    return q;
  };
  Piece ring[kAhead + 1];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) ring[i] = fetch(me + i * lanes);
  float cs[2] = {1.0f, 1.0f};
  if constexpr (kI8)
    for (int c = 0; c < 2; ++c) cs[c] = load_scale<kScaleF16>(p.scale, ch[c]);
  // nothing the previous kernel writes has been touched so far
  pdl_wait_prior_grid();

  // Activations -> shared memory as f32, a step's four neighbours of one place side by side over the steps: the threads
  // of a group, one step apart, then read consecutive 16-byte words (from global memory they are 64 or 128 bytes apart:
  // 1 x 1152 -> 60468 int4 26 us).  An odd row length keeps the stores off each other's banks.
  extern __shared__ float4 xs[];
  const uint32_t row4 = p.steps | 1u;
  {
    const XT* x = static_cast<const XT*>(p.x) + static_cast<size_t>(m0) * p.k;
    const uint32_t eights = p.k / 8u;
    const bool norm = std::is_same<XT, float>::value && p.norm_weight != nullptr;
    if (norm) {
      // sums of squares in a fixed order: thread-strided, shuffle tree, warps in order
      float sq[kRowsX];
#pragma unroll
      for (int r = 0; r < kRowsX; ++r) sq[r] = 0.0f;
      for (uint32_t i = threadIdx.x; i < eights; i += kRowsThreads)
#pragma unroll
        for (int r = 0; r < kRowsX; ++r) {
          if (static_cast<uint32_t>(r) >= live) continue;
          float v[8];
          load_x8<XT, false>(x + static_cast<size_t>(r) * p.k + i * 8u, v);
#pragma unroll
          for (int e = 0; e < 8; ++e) sq[r] = fmaf(v[e], v[e], sq[r]);
        }
#pragma unroll
      for (int r = 0; r < kRowsX; ++r) {
        sq[r] = warp_sum(sq[r]);
        if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5][r] = sq[r];
      }
      __syncthreads();
      if (threadIdx.x < kRowsX) {
        float total = 0.0f;
        for (uint32_t w = 0; w < kRowsThreads / 32; ++w) total += part[w][threadIdx.x];
        row_norm[threadIdx.x] = rsqrtf(total * (1.0f / static_cast<float>(p.k)) + p.norm_eps);
      }
      __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < kRowsX * eights; i += kRowsThreads) {
      const uint32_t r = kRowsX == 1 ? 0u : i / eights, at = kRowsX == 1 ? i : i - r * eights, step = at / kEights, e = at % kEights;
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (r < live) load_x8<XT, false>(x + static_cast<size_t>(r) * p.k + at * 8u, v);
      if (norm) {
        float wv[8];
        load_x8<float, false>(p.norm_weight + at * 8u, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(__fmul_rn(v[j], row_norm[r]), wv[j]);
      }
      float4* dst = xs + ((r * kEights + e) * 2u) * row4 + step;
      dst[0] = make_float4(v[0], v[1], v[2], v[3]);
      dst[row4] = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  __syncthreads();
  float acc[2][kRowsX];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < kRowsX; ++r) acc[c][r] = 0.0f;
  for (uint32_t i0 = 0; i0 * lanes < p.steps; i0 += kAhead + 1)
#pragma unroll
  for (uint32_t u = 0; u <= kAhead; ++u) {
    const uint32_t i = i0 + u;
    if (i * lanes >= p.steps) break;
    ring[(u + kAhead) % (kAhead + 1)] = fetch(me + (i + kAhead) * lanes);
    const Piece& q = ring[u];
    const uint32_t step = me + i * lanes;
    if (step < p.steps) {
      float sum[2][kRowsX];
#pragma unroll
      for (int e = 0; e < kEights; ++e) {
        if (e % 2 == 0) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int r = 0; r < kRowsX; ++r) sum[c][r] = 0.0f;
        }
        float wv[2][8];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t words[4] = {q.w[c].x, q.w[c].y, q.w[c].z, q.w[c].w};
          if constexpr (kI8) {
            rows_bytes(words[2 * e], wv[c]);
            rows_bytes(words[2 * e + 1], wv[c] + 4);
          } else {
            rows_nibbles(words[e], wv[c]);
          }
          const float s = kI8 ? cs[c] : q.s[c][e / 2];
#pragma unroll
          for (int j = 0; j < 8; ++j) wv[c][j] = __fmul_rn(wv[c][j], s);
        }
#pragma unroll
        for (int r = 0; r < kRowsX; ++r) {
          {
            const float4* src = xs + ((r * kEights + e) * 2) * row4 + step;
            const float4 a = src[0], b = src[row4];
            const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int j = 0; j < 8; ++j) sum[c][r] = fmaf(v[j], wv[c][j], sum[c][r]);
          }
        }
        if (e % 2 == 1) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int r = 0; r < kRowsX; ++r) acc[c][r] += sum[c][r];
        }
      }
    }
  }
  // the threads of a channel pair meet
  const uint32_t in_warp = min(lanes, 32u);
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < kRowsX; ++r)
      for (uint32_t off = in_warp >> 1; off > 0; off >>= 1) acc[c][r] += __shfl_xor_sync(0xffffffffu, acc[c][r], off);
  if (lanes > 32u) {
    if ((threadIdx.x & 31u) == 0)
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int r = 0; r < kRowsX; ++r) part[threadIdx.x >> 5][c * kRowsX + r] = acc[c][r];
    __syncthreads();
    const uint32_t first = (threadIdx.x >> 5) & ~((lanes >> 5) - 1u);
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int r = 0; r < kRowsX; ++r) {
        float total = 0.0f;
        for (uint32_t w = 0; w < lanes >> 5; ++w) total += part[first + w][c * kRowsX + r];
        acc[c][r] = total;
      }
  }
  // thread r of the group stores activation row r (or, of few threads, several)
#pragma unroll
  for (int r = 0; r < kRowsX; ++r) {
    if (static_cast<uint32_t>(r) < live && me == (static_cast<uint32_t>(r) & (lanes - 1u))) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (2u * pair + c < p.n) {
          const size_t at = static_cast<size_t>(m0 + r) * p.n + 2u * pair + c;
          float o = __fadd_rn(acc[c][r], p.bias[2u * pair + c]);
          if (p.residual != nullptr) o = __fadd_rn(o, p.residual[at]);
          p.out[at] = o;
        }
    }
  }
}

template <typename XT, bool kI8, bool kScaleF16, int kRowsX>
cudaError_t launch_rows(const LaunchEnv& env, const RowsParams& p) {
  auto kernel = qgemv_rows_kernel<XT, kI8, kScaleF16, kRowsX>;
  static OncePerDevice configured;
  const cudaError_t ready = configured.run([&] { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kRowsSmem)); });
  if (ready != cudaSuccess) return ready;
  cudaLaunchConfig_t cfg = {};
  const uint32_t pairs = (p.n + 1) / 2, per_cta = kRowsThreads >> p.lanes_log2;
  cfg.gridDim = dim3((pairs + per_cta - 1) / per_cta, (p.m + kRowsX - 1) / kRowsX);
  cfg.blockDim = dim3(kRowsThreads);
  cfg.dynamicSmemBytes = rows::staged_bytes(rows::Call{!kI8, p.n, p.k, p.m, 1});
  cfg.stream = env.stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = env.overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, p);
}
template <typename XT, bool kI8, bool kScaleF16>
cudaError_t launch_rows_m(const LaunchEnv& env, const RowsParams& p) {
  if (p.m == 1) return launch_rows<XT, kI8, kScaleF16, 1>(env, p);
  if (p.m == 2) return launch_rows<XT, kI8, kScaleF16, 2>(env, p);
  return launch_rows<XT, kI8, kScaleF16, 4>(env, p);
}
template <typename XT>
cudaError_t launch_rows_typed(const LaunchEnv& env, const RowsParams& p, bool i8, bool f16s) {
  if (i8) return f16s ? launch_rows_m<XT, true, true>(env, p) : launch_rows_m<XT, true, false>(env, p);
  return f16s ? launch_rows_m<XT, false, true>(env, p) : launch_rows_m<XT, false, false>(env, p);
}

}  // namespace

bool qgemv_rows_supports(const Weight& w, uint32_t m) { return w.layout == kLayoutNative && rows::supports(rows_call(w, m, 1)); }
bool qgemv_rows_preferred(const LaunchEnv& env, const LinearTarget& t, int x_dtype, uint32_t m) {
  const rows::Call call = rows_call(*t.w, m, env.sm_count);
  const uint64_t room = env.workspace != nullptr ? env.workspace_bytes : 0;
  if (qgemm_exact_supports(1, &t, m, room)) return rows::preferred(call, rows::estimate_many_row(qgemm_exact_clocks(env, *t.w, x_dtype, m), x_dtype == KQ_F16));
  const int neighbours = (env.norm_weight != nullptr) + (env.residual != nullptr);  // kernels of their own beside the generic one
  return rows::preferred(call, rows::estimate_generic(call) + neighbours * rows::kNeighbour);
}

cudaError_t launch_qgemv_rows(const LaunchEnv& env, const LinearTarget& t, const void* x, int x_dtype, uint32_t m) {
  const Weight& w = *t.w;
  if (!qgemv_rows_supports(w, m) || (env.norm_weight != nullptr && x_dtype != KQ_F32)) return cudaErrorInvalidValue;
  const bool i8 = w.storage == KQ_STORAGE_I8;
  RowsParams p = {};
  p.w = static_cast<const uint8_t*>(w.data);
  p.scale = w.scale;
  p.bias = t.bias;
  p.out = t.out;
  p.x = x;
  p.m = m;
  p.n = w.n;
  p.k = w.k;
  p.steps = w.k / (i8 ? 16u : 32u);
  p.norm_weight = env.norm_weight;
  p.norm_eps = env.norm_eps;
  p.residual = env.residual;
  while (!i8 && (1u << p.gshift) < w.group_size) ++p.gshift;
  p.lanes_log2 = rows::lanes_log2(rows_call(w, m, env.sm_count));
  const bool f16s = w.scale_dtype == KQ_F16;
  switch (x_dtype) {
    case KQ_F32: return launch_rows_typed<float>(env, p, i8, f16s);
    case KQ_F16: return launch_rows_typed<__half>(env, p, i8, f16s);
    case KQ_BF16: return launch_rows_typed<__nv_bfloat16>(env, p, i8, f16s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace kq
