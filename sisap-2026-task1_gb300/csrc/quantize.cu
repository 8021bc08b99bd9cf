// quantize.cu -- K1: float32 rows -> int8 codes + sign-bit sketches, one pass.
//
// Reference: src/main.cpp:179-192.  For every coordinate
//   scaled  = x * 127.0f
//   clamped = max(-128.0f, min(127.0f, scaled))    (std::min/max operand order,
//                                                   so NaN -> 127)
//   code    = (int8) clamped                       (truncation toward zero)
//   sketch bit k%64 of word k/64 = clamped > 0
// Subnormal inputs are read as zero, as the reference's -ffast-math build does.
// KNNG_QUANT_ROUND clamps to [-127, 127] and rounds half away from zero.
//
// Layout: the rows are one stream of 8-float groups, one group per lane and
// load pair, so a warp's pair of loads covers 1 KB without a gap: coalesced
// for HBM and for host rows read directly over the CPU link.  A sketch word
// covers 8 consecutive groups of one row (d % 64 == 0), combined across lanes
// by shuffles.
// Bound by the input stream: 4d + d + d/8 bytes per row.  1M x 1024 (5.25 GB):
// 0.72 ms, 7.3 TB/s (reads outnumber writes 4 to 1, so it can pass a plain
// copy's 6.8 TB/s); one float4 per lane and load with a persistent grid took
// 0.80 ms.  A whole call on rows not in L2: 0.73 ms, 0.97 before.  Pinned host rows come at the link's 211 GB/s either way.
#include "knng_internal.cuh"

namespace knng {
namespace {

// x * 127 with subnormal inputs read as zero.  The flush-to-zero multiply
// gives exactly that for every input: a subnormal x becomes a signed zero, and
// a normal x has a normal product, so nothing else is flushed.
__device__ __forceinline__ float scale127_daz(float v) {
  float s;
  asm("mul.ftz.f32 %0, %1, %2;" : "=f"(s) : "f"(v), "f"(127.0f));
  return s;
}

// The reference's std::max(lo, std::min(127.0f, s)): fminf/fmaxf return the
// non-NaN operand, so NaN becomes 127 as in std::min(127.0f, NaN).
template <int kMode>
__device__ __forceinline__ int quant1(float v, unsigned& bit) {
  const float s = scale127_daz(v);
  const float c = fmaxf(fminf(s, 127.0f), kMode == KNNG_QUANT_ROUND ? -127.0f : -128.0f);
  bit = c > 0.0f ? 1u : 0u;
  return kMode == KNNG_QUANT_ROUND ? __float2int_rz(roundf(c)) : __float2int_rz(c);
}

// One block covers kThreads x kUnroll groups: four pairs of loads in flight
// per lane.  Blocks that come and go kept HBM busier than a grid that stays
// and strides (0.80 ms against 0.78 with one float4 per lane, 0.72 against
// 0.77 with two), and eight groups per lane, or blocks of 512, were slower.
// Lane l quantises a group into two 4-byte code words and a sign byte; the
// sketch word of 8 consecutive groups (64 floats, bit j = float j > 0) takes
// lane l's byte at bit 8 (l % 8), combined by two xor-shuffle ORs within 4
// lanes and one shuffle for the upper half.  Two 16-byte loads and two 4-byte
// stores need no more alignment than the rows and codes have anyway; one
// 32-byte load and one 8-byte store per group measured within 1 %.
constexpr int kThreads = 128, kUnroll = 4;

template <int kMode>
__global__ void __launch_bounds__(kThreads) quantize_kernel(const float4* __restrict__ x, int64_t groups,
                                                            uint32_t* __restrict__ codes, uint64_t* __restrict__ sketch) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t g0 = int64_t(blockIdx.x) * (kThreads * kUnroll) + (threadIdx.x - lane) * kUnroll + lane;
  float4 v[kUnroll][2];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t g = g0 + 32 * u;
    v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g < groups) {
      v[u][0] = x[2 * g];
      v[u][1] = x[2 * g + 1];
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t g = g0 + 32 * u;
    unsigned w = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      unsigned b0, b1, b2, b3;
      const int q0 = quant1<kMode>(v[u][h].x, b0), q1 = quant1<kMode>(v[u][h].y, b1);
      const int q2 = quant1<kMode>(v[u][h].z, b2), q3 = quant1<kMode>(v[u][h].w, b3);
      if (g < groups)
        codes[2 * g + h] = (unsigned(q0) & 0xffu) | ((unsigned(q1) & 0xffu) << 8) | ((unsigned(q2) & 0xffu) << 16) |
                           ((unsigned(q3) & 0xffu) << 24);
      w |= (b0 | (b1 << 1) | (b2 << 2) | (b3 << 3)) << (4 * h);
    }
    w <<= 8 * (lane & 3);
    w |= __shfl_xor_sync(full, w, 1);
    w |= __shfl_xor_sync(full, w, 2);  // lanes 4q..4q+3: their 32 sign bits
    const unsigned hi = __shfl_down_sync(full, w, 4);
    // a multiple of 8 groups, so an 8-lane run is wholly in range or out
    if ((lane & 7) == 0 && g < groups) sketch[g >> 3] = uint64_t(w) | (uint64_t(hi) << 32);
  }
}

}  // namespace

cudaError_t launch_quantize(const float* x, int64_t n, int d, int quant_mode, int8_t* codes,
                            uint64_t* sketch, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int64_t groups = n * int64_t(d / 8);  // a multiple of 8: d % 64 == 0
  const int64_t blocks = (groups + kThreads * kUnroll - 1) / (kThreads * kUnroll);  // 16 KB of rows each
  if (blocks > 0x7fffffff) return cudaErrorInvalidValue;  // 35 TB of rows
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  const float4* x4 = reinterpret_cast<const float4*>(x);
  uint32_t* c4 = reinterpret_cast<uint32_t*>(codes);
  if (quant_mode == KNNG_QUANT_ROUND) quantize_kernel<KNNG_QUANT_ROUND><<<int(blocks), kThreads, 0, s>>>(x4, groups, c4, sketch);
  else quantize_kernel<KNNG_QUANT_TRUNC><<<int(blocks), kThreads, 0, s>>>(x4, groups, c4, sketch);
  note_launch();
  return cudaGetLastError();
}

}  // namespace knng
