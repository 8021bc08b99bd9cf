// gram_mma.cu -- K3, default form: leaf Gram blocks with warp-level tensor-core
// instructions straight from registers.
//
// Reference: the dots of src/main.cpp:261-269 (every pair of members of a
// leaf).  Same arithmetic as leaf_gram_tc (gram_tc.cu): the int8 codes widened
// to f16 and multiplied into fp32 accumulators, which gives the int32 dot bit
// for bit (f16_codes.cuh).
//
// One warp per leaf.  For mma.m16n8k16 a thread's A registers of rows
// 16R..16R+15 and its B registers of the same rows as columns hold the same
// elements, so each code is loaded and widened once and serves as both
// operands; the order of the K elements is free as long as both operands
// agree, so a lane simply takes 16 consecutive codes of its row (4 lanes of a
// row read 64 contiguous bytes, one 16-byte load each).  Nothing passes
// through shared memory, there is no barrier and no wait.
//
// The Gram is symmetric: only the 16 x 8 tiles that reach the diagonal or lie
// above it are computed (20 of 32 for a full leaf) and only those that hold
// members (9 for the usual 34 members); each value is stored at both of its
// places, 32-byte sectors at a time.
//
// tcgen05 (gram_tc.cu, what ran here before) wants its operands in shared
// memory, widened and in core-matrix order: 2 KB of writes and 4 KB of operand
// reads per 1 KB row, a barrier per 64 columns, and a 128 x 128 tile per two
// leaves of which 34 x 34 twice are wanted.  Here the usual leaf (34 members,
// d = 1024) takes 9 x 64 tensor instructions of 8 cycles, 5 instructions per 4
// codes of widening and 34 KB of rows, about 1,300-1,500 SM cycles each way.
// Measured (300k x 1024, 16 trees, 4.8M members): 4.26 -> 1.72 ms; 4.4 GB of
// DRAM reads, 0.38 of the DRAM peak, tensor pipe 0.33 busy.  What is left is
// the latency of a segment's loads at 12 warps per SM (168 registers hold the
// accumulators); prefetching the next leaf's rows into L2 and loading a
// segment ahead changed it by less than 2 %, four CTAs per SM spilled.  A warp
// ends with its leaf: a grid that stayed and strode over the leaves, the next
// leaf's ids loaded ahead, made the initial graph 2 % slower at 300k (3.17 ->
// 3.23 ms) and 8 % at 1M (10.7 -> 11.6).
#include "f16_codes.cuh"

namespace knng {
namespace {

constexpr int kGmThreads = 128;
constexpr int kGmWarps = kGmThreads / 32;
constexpr int kGmCtas = 3;      // CTAs per SM: 168 registers per thread
constexpr int kGroups = 8;      // 8-row groups of a leaf

// First tile of row tile R among G column groups: R-major, C = 2R..G-1.
__host__ __device__ constexpr int tile_base(int R, int G) { return R * (G + 1 - R); }

// The Gram block of a leaf of m <= 8 G members, by one warp.  id[i]: the row
// 8i + g of this lane.  One body per G: with the group count in a register
// every tensor instruction sat behind a branch of its own (285 instructions
// per member instead of 117).  Leaves of 1-16 and of 17-32 members share a body:
// all eight did not stay in the instruction cache (1.82 against 1.72 ms).
template <int G>
__device__ __forceinline__ void leaf_block(const int8_t* __restrict__ base, const int32_t (&id)[kGroups], int d, int m,
                                           int g, int c, int32_t* __restrict__ out) {
  constexpr int RT = (G + 1) / 2;  // 16-row tiles
  constexpr int kTiles = tile_base(RT, G);
  float acc[kTiles][4];
#pragma unroll
  for (int t = 0; t < kTiles; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[t][e] = 0.f;
#pragma unroll 1
  for (int k0 = 0; k0 < d; k0 += 64) {
    uint4 raw[G];
#pragma unroll
    for (int i = 0; i < G; ++i) raw[i] = __ldg(reinterpret_cast<const uint4*>(base + int64_t(id[i]) * d + k0));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t f0[2 * RT], f1[2 * RT];
#pragma unroll
      for (int i = 0; i < G; ++i) widen4(q == 0 ? raw[i].x : q == 1 ? raw[i].y : q == 2 ? raw[i].z : raw[i].w, f0[i], f1[i]);
      if (G < 2 * RT) f0[2 * RT - 1] = f1[2 * RT - 1] = 0;
#pragma unroll
      for (int R = 0; R < RT; ++R) {
#pragma unroll
        for (int C = 2 * R; C < G; ++C)
          mma16816(acc[tile_base(R, G) + C - 2 * R], f0[2 * R], f0[2 * R + 1], f1[2 * R], f1[2 * R + 1], f0[C], f1[C]);
      }
    }
  }
  // Element e of tile (R, C): row 16R + g (+ 8 for e >= 2), column 8C + 2c +
  // (e & 1).  Rows past the leaf are not stored (they are the next leaf's);
  // columns past it may be: a Gram row has room for 64 and its readers stop at
  // m.  So a store depends on its row alone, and every offset is a constant.
  int32_t* direct = out + g * kMaxLeaf + 2 * c;
  int32_t* mirror = out + 2 * c * kMaxLeaf + g;
#pragma unroll
  for (int R = 0; R < RT; ++R) {
#pragma unroll
    for (int C = 2 * R; C < G; ++C) {
      const float(&v)[4] = acc[tile_base(R, G) + C - 2 * R];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (2 * R + h < G) {
          const int v0 = __float2int_rn(v[2 * h]), v1 = __float2int_rn(v[2 * h + 1]);
          const int row0 = 16 * R + 8 * h, col0 = 8 * C;
          if (g < m - row0) *reinterpret_cast<int2*>(direct + row0 * kMaxLeaf + col0) = make_int2(v0, v1);
          if (C > 2 * R + h) {  // above the diagonal 8 x 8 blocks: also the mirrored place
            if (2 * c < m - col0) mirror[col0 * kMaxLeaf + row0] = v0;
            if (2 * c + 1 < m - col0) mirror[(col0 + 1) * kMaxLeaf + row0] = v1;
          }
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kGmThreads, kGmCtas) leaf_gram_mma(const int8_t* __restrict__ codes, int d,
                                                                    const int32_t* __restrict__ perm,
                                                                    const int32_t* __restrict__ leaf_start,
                                                                    int64_t nleaves, int64_t total,
                                                                    int32_t* __restrict__ gram, int64_t gram_pos0,
                                                                    unsigned* err, int64_t n_rows) {
  (void)err;
  (void)n_rows;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int64_t l = int64_t(blockIdx.x) * kGmWarps + (threadIdx.x >> 5);
  if (l >= nleaves) return;
  const int64_t s = leaf_start[l];
  int m = int((l + 1 < nleaves ? int64_t(leaf_start[l + 1]) : total) - s);
  m = m < kMaxLeaf ? m : kMaxLeaf;  // (a leaf holds at most kMaxLeaf members)
  int32_t id0 = 0, id1 = 0;         // the leaf's member ids, 2 per lane
  if (lane < m) id0 = perm[s + lane];
  if (32 + lane < m) id1 = perm[s + 32 + lane];
  // row 8i + g of this lane, the last member's in the rows past the end
  // (their results are not stored)
  int32_t id[kGroups];
#pragma unroll
  for (int i = 0; i < kGroups; ++i) {
    const int r = max(min(8 * i + g, m - 1), 0);
    const int32_t lo = __shfl_sync(full, id0, r & 31), hi = __shfl_sync(full, id1, r & 31);
    id[i] = r < 32 ? lo : hi;
    if (!KNNG_GUARD(err, id[i] >= 0 && id[i] < n_rows)) id[i] = 0;
  }
  const int8_t* base = codes + 16 * c;
  int32_t* out = gram + (s - gram_pos0) * int64_t(kMaxLeaf);
  switch ((m + 7) >> 3) {  // warp-uniform
    case 1:
    case 2: leaf_block<2>(base, id, d, m, g, c, out); break;
    case 3:
    case 4: leaf_block<4>(base, id, d, m, g, c, out); break;
    case 5: leaf_block<5>(base, id, d, m, g, c, out); break;
    case 6: leaf_block<6>(base, id, d, m, g, c, out); break;
    case 7: leaf_block<7>(base, id, d, m, g, c, out); break;
    case 8: leaf_block<8>(base, id, d, m, g, c, out); break;
    default: break;
  }
}

}  // namespace

cudaError_t launch_leaf_gram_mma(const int8_t* codes, int d, const int32_t* perm, const int32_t* leaf_start,
                                 int64_t nleaves, int64_t total, int32_t* gram, int64_t gram_pos0, unsigned* err,
                                 cudaStream_t s, int64_t n_rows) {
  if (d % 64 != 0) return cudaErrorInvalidValue;
  if (nleaves <= 0) return cudaSuccess;
  const int64_t blocks = (nleaves + kGmWarps - 1) / kGmWarps;  // below 2^31: num_trees * n is
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  leaf_gram_mma<<<unsigned(blocks), kGmThreads, 0, s>>>(codes, d, perm, leaf_start, nleaves, total, gram, gram_pos0,
                                                        err, n_rows);
  note_launch();
  return cudaGetLastError();
}

}  // namespace knng
