// forest.cu -- K2: random-projection forest, all trees level by level.
//
// Reference: build_tree, src/main.cpp:47-99, and the forest loop :205-216.  A
// node with more than leaf_size members picks two distinct members p1, p2 and
// splits stably: p1 goes left, p2 right, any other member x goes left iff
// dot(x, p1) > dot(x, p2) in exact int32 over the int8 codes.  The reference
// recurses depth first with one std::mt19937 per tree; here every tree's
// perm[t*n ...] array is split level-synchronously, one kernel sequence per
// level for all T trees at once.  A node always covers a contiguous range of
// its tree's perm, left child first, so the final perm of a tree is exactly
// the reference's DFS leaf order when the same pivots are used (replay mode),
// and node identity is (tree, start, size).
//
// Native pivots come from a counter-based hash of (seed, tree, start, size):
// the reference's pivot stream is a serial dependency through the whole DFS
// (the right subtree's draws wait for the left subtree's), so it is replayed
// only in tests, from the oracle's log.
//
// A batch of jobs is one problem of N rows (tree-major [T][N] arrays, job b at
// offset off[b] in every tree); every level serves all jobs' nodes at once.
//
// Per level (replay, or fusing off): pick_pivots -> scan(tiles) -> side (8 lanes per row, dp4a,
// HBM-bound: d bytes read per active member) -> scan(left counts) -> scatter
// (stable partition into perm_tmp) -> copy back -> children (leaf flags,
// next node list).
//
// Fused levels (native pivots, the default): the side pass is HBM-bound on
// reading every active member's code row once per level, so large nodes are
// split kFuse levels at a time from one read of each row.  A node's pivots
// and those of its descendants down to kFuse - 1 levels below are fixed
// before the pass from a seeded sample of up to kCand distinct members (the
// node's "candidates", in a hashed order): the node's pivots are the first
// two candidates; a descendant's are the first two candidates, not already
// an ancestor's pivot, that the splits above it send into it -- each
// candidate's path is computed with the same exact dot products the member
// pass uses, so these pivots are members of the descendant.  Given the
// ancestors' splits, the candidates in a descendant are a uniform sample of
// its members, so a descendant's pivot pair is a uniformly drawn pair of its
// distinct members other than its ancestors' pivots, as in the per-level
// rule.  A descendant that receives fewer than two free candidates is not
// split in the pass and is queued as a node of its own.  The member pass
// then gives every member a kFuse-bit path code (first split in the high
// bit; bits below an unsplit descendant are 0), and one stable counting
// sort by code per node lays out all kFuse levels at once: each descendant
// is a contiguous range, left before right, as the per-level splits would
// leave it (inside a descendant that turns out to be a leaf the members
// are also ordered by the deeper bits, which no later stage depends on).
// Nodes smaller than kFuseMin are parked (the sample would be a large
// fraction of them) and split to their leaves by one kernel after the fused
// rounds, one CTA per node (subtree_kernel), with the per-level rule's pivots
// and stable splits.
//
// Node lists are filled through atomic counters, so their order varies; a
// node's pivots depend on its identity only, so the forest does not.
#include "f16_codes.cuh"

#include <algorithm>
#include <vector>

namespace knng {
namespace {

constexpr int kTileElems = 256;
constexpr int kFuse = 3;                        // levels per fused pass
constexpr int kFuseNodes = (1 << kFuse) - 1;    // split nodes of one fused subtree (depth 0 .. kFuse-1)
constexpr int kFuseBins = 1 << kFuse;           // path codes
constexpr int kCand = 64;                       // pivot candidates per fused node
constexpr int32_t kFuseMin = 512;               // smaller nodes are left to subtree_kernel

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// The hash a node's pivots are drawn from: its identity (tree, start within
// the job's range, size) and the seed.
__device__ __forceinline__ uint64_t node_hash(uint32_t seed, int32_t tree, int32_t local, int32_t size) {
  uint64_t h = splitmix64((uint64_t(seed) << 32) ^ uint64_t(uint32_t(tree)));
  h = splitmix64(h ^ uint64_t(uint32_t(local)));
  return splitmix64(h ^ (uint64_t(uint32_t(size)) << 1));
}

struct NodeArr {
  int32_t *start, *size, *p1, *p2;
};
__host__ __device__ inline NodeArr node_arr(int32_t* base, int64_t cap) {
  return NodeArr{base, base + cap, base + 2 * cap, base + 3 * cap};
}

__global__ void init_perm(int32_t* perm, int64_t n, int T) {
  const int64_t tot = n * T;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < tot; i += int64_t(gridDim.x) * blockDim.x)
    perm[i] = int32_t(i % n);
}

// Roots: for tree t and job b the range t*N + off[b] of size n[b]; jobs with
// n[b] <= leaf are single leaves.  Node order is by start (tree, then job).
// For the fused rounds p1 holds a root's first tile (root_tiles per tree).
__global__ void root_nodes(NodeArr nd, int64_t N, int T, int leaf, uint8_t* leaf_flag, JobTable jt, int split_jobs,
                           int root_tiles) {
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    int k = t * split_jobs, tile = t * root_tiles;
    for (int b = 0; b < jt.count; ++b) {
      const int64_t start = int64_t(t) * N + jt.off[b];
      if (jt.n[b] > leaf) {
        nd.start[k] = int32_t(start);
        nd.size[k] = jt.n[b];
        nd.p1[k] = tile;
        tile += (jt.n[b] + kTileElems - 1) / kTileElems;
        ++k;
      } else {
        leaf_flag[start] = 1;
      }
    }
  }
}

// Node identity is job-local -- (tree, start within the job's range, size) --
// so a job draws the same pivots alone and inside any batch.
__global__ void pick_pivots(NodeArr nd, int cnt, int64_t n, uint32_t seed, int level, const int32_t* perm,
                            const int32_t* replay, int32_t* tile_cnt, unsigned* err, JobTable jt) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const int32_t start = nd.start[k], size = nd.size[k];
  const int32_t tree = int32_t(int64_t(start) / n);
  const int32_t in_tree = int32_t(int64_t(start) - int64_t(tree) * n);
  const int32_t local = in_tree - jt.off[job_of(jt, in_tree)];
  int32_t p1, p2;
  if (replay) {
    const int32_t* r = replay + 6 * int64_t(k);
    if (r[0] != tree || r[1] != level || r[2] != local || r[3] != size) {
      atomicOr(err, kErrReplay);
      p1 = perm[start];
      p2 = perm[start + 1];
    } else {
      p1 = r[4];
      p2 = r[5];
    }
  } else {
    const uint64_t h = node_hash(seed, tree, local, size);
    const uint64_t h2 = splitmix64(h ^ 0x5851F42D4C957F2Dull);
    int32_t a = int32_t(h % uint64_t(size));
    int32_t b = int32_t(h2 % uint64_t(size - 1));
    if (b >= a) ++b;
    p1 = perm[start + a];
    p2 = perm[start + b];
  }
  nd.p1[k] = p1;
  nd.p2[k] = p2;
  tile_cnt[k] = (size + kTileElems - 1) / kTileElems;
}

__device__ __forceinline__ int find_node(const int32_t* tile_off, int cnt, int b) {
  int lo = 0, hi = cnt - 1;  // largest k with tile_off[k] <= b
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (tile_off[mid] <= b) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One block per tile of <= 256 members of one node.  8 lanes per member: lane
// sub reads 16-byte chunks sub, sub+8, ... of the member's code row and
// accumulates dp4a against both pivot rows staged in shared memory.
__global__ void __launch_bounds__(256) side_kernel(const int8_t* __restrict__ codes, int d,
                                                   const int32_t* __restrict__ perm, NodeArr nd, int cnt,
                                                   const int32_t* __restrict__ tile_off,
                                                   uint8_t* __restrict__ side, int32_t* __restrict__ tile_left) {
  __shared__ uint4 piv[2][kMaxDim / 16];
  __shared__ int node_s;
  __shared__ int32_t warp_cnt[8];
  const int b = blockIdx.x;
  if (threadIdx.x == 0) node_s = find_node(tile_off, cnt, b);
  __syncthreads();
  const int k = node_s;
  const int32_t start = nd.start[k], size = nd.size[k], p1 = nd.p1[k], p2 = nd.p2[k];
  const int64_t e0 = int64_t(start) + int64_t(b - tile_off[k]) * kTileElems;
  const int64_t e1 = min(int64_t(start) + size, e0 + kTileElems);
  const int nchunk = d / 16;
  for (int c = threadIdx.x; c < 2 * nchunk; c += blockDim.x) {
    const int which = c / nchunk, cc = c % nchunk;
    const int32_t pid = which ? p2 : p1;
    piv[which][cc] = reinterpret_cast<const uint4*>(codes + int64_t(pid) * d)[cc];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, slot = lane >> 3;
  const int per_lane = d / 128;
  int my_left = 0;
  for (int step = 0; step < 8; ++step) {
    const int t = warp * 32 + step * 4 + slot;
    const int64_t e = e0 + t;
    const bool valid = e < e1;
    const int32_t id = valid ? perm[e] : 0;
    const uint4* row = reinterpret_cast<const uint4*>(codes + int64_t(id) * d);
    int d1 = 0, d2 = 0;
    if (valid) {
      uint4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (u < per_lane) v[u] = __ldg(row + sub + 8 * u);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (u < per_lane) {
          const uint4 a = piv[0][sub + 8 * u], c = piv[1][sub + 8 * u];
          d1 = __dp4a(int(v[u].x), int(a.x), d1);
          d1 = __dp4a(int(v[u].y), int(a.y), d1);
          d1 = __dp4a(int(v[u].z), int(a.z), d1);
          d1 = __dp4a(int(v[u].w), int(a.w), d1);
          d2 = __dp4a(int(v[u].x), int(c.x), d2);
          d2 = __dp4a(int(v[u].y), int(c.y), d2);
          d2 = __dp4a(int(v[u].z), int(c.z), d2);
          d2 = __dp4a(int(v[u].w), int(c.w), d2);
        }
      }
    }
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      d1 += __shfl_xor_sync(0xffffffffu, d1, o);
      d2 += __shfl_xor_sync(0xffffffffu, d2, o);
    }
    const bool left = (id == p1) || (id != p2 && d1 > d2);
    if (valid && sub == 0) {
      side[e] = left ? 1 : 0;
      my_left += left ? 1 : 0;
    }
  }
  for (int o = 16; o > 0; o >>= 1) my_left += __shfl_xor_sync(0xffffffffu, my_left, o);
  if (lane == 0) warp_cnt[warp] = my_left;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < 8; ++w) s += warp_cnt[w];
    tile_left[b] = s;
  }
}

__device__ __forceinline__ int32_t node_left(const NodeArr& nd, int k, const int32_t* tile_off,
                                             const int32_t* tile_left, const int32_t* tile_left_off) {
  const int f = tile_off[k];
  const int fl = f + (nd.size[k] + kTileElems - 1) / kTileElems - 1;
  return tile_left_off[fl] + tile_left[fl] - tile_left_off[f];
}

__global__ void __launch_bounds__(256) scatter_kernel(const int32_t* __restrict__ perm,
                                                      int32_t* __restrict__ perm_tmp, NodeArr nd, int cnt,
                                                      const int32_t* __restrict__ tile_off,
                                                      const uint8_t* __restrict__ side,
                                                      const int32_t* __restrict__ tile_left,
                                                      const int32_t* __restrict__ tile_left_off) {
  __shared__ int node_s;
  __shared__ int32_t warp_off[8];
  const int b = blockIdx.x;
  if (threadIdx.x == 0) node_s = find_node(tile_off, cnt, b);
  __syncthreads();
  const int k = node_s;
  const int32_t start = nd.start[k], size = nd.size[k];
  const int64_t e0 = int64_t(start) + int64_t(b - tile_off[k]) * kTileElems;
  const int64_t e1 = min(int64_t(start) + size, e0 + kTileElems);
  const int32_t nleft = node_left(nd, k, tile_off, tile_left, tile_left_off);
  const int32_t base = tile_left_off[b] - tile_left_off[tile_off[k]];
  const int64_t e = e0 + threadIdx.x;
  const bool valid = e < e1;
  const bool left = valid && side[e];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned bal = __ballot_sync(0xffffffffu, left);
  if (lane == 0) warp_off[warp] = __popc(bal);
  __syncthreads();
  int32_t pre = 0;
  for (int w = 0; w < warp; ++w) pre += warp_off[w];
  pre += __popc(bal & ((1u << lane) - 1u));
  if (valid) {
    const int32_t lrank = base + pre;
    const int32_t rrank = int32_t(e - start) - lrank;
    const int64_t np = int64_t(start) + (left ? lrank : nleft + rrank);
    perm_tmp[np] = perm[e];
  }
}

__global__ void __launch_bounds__(256) copyback_kernel(int32_t* __restrict__ perm,
                                                       const int32_t* __restrict__ perm_tmp, NodeArr nd,
                                                       int cnt, const int32_t* __restrict__ tile_off) {
  __shared__ int node_s;
  const int b = blockIdx.x;
  if (threadIdx.x == 0) node_s = find_node(tile_off, cnt, b);
  __syncthreads();
  const int k = node_s;
  const int64_t e0 = int64_t(nd.start[k]) + int64_t(b - tile_off[k]) * kTileElems;
  const int64_t e1 = min(int64_t(nd.start[k]) + nd.size[k], e0 + kTileElems);
  const int64_t e = e0 + threadIdx.x;
  if (e < e1) perm[e] = perm_tmp[e];
}

__global__ void children_count(NodeArr nd, int cnt, int leaf, const int32_t* tile_off, const int32_t* tile_left,
                               const int32_t* tile_left_off, uint8_t* leaf_flag, int32_t* child_cnt) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const int32_t nl = node_left(nd, k, tile_off, tile_left, tile_left_off);
  const int32_t nr = nd.size[k] - nl;
  const int64_t s = nd.start[k];
  if (nl <= leaf) leaf_flag[s] = 1;
  if (nr <= leaf) leaf_flag[s + nl] = 1;
  child_cnt[k] = (nl > leaf ? 1 : 0) + (nr > leaf ? 1 : 0);
}

__global__ void children_emit(NodeArr nd, int cnt, int leaf, const int32_t* tile_off, const int32_t* tile_left,
                              const int32_t* tile_left_off, const int32_t* child_off, NodeArr nx,
                              int64_t cap, unsigned* err) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const int32_t nl = node_left(nd, k, tile_off, tile_left, tile_left_off);
  const int32_t nr = nd.size[k] - nl;
  int32_t o = child_off[k];
  if (int64_t(o) + 2 > cap) {  // cannot happen: active nodes are disjoint and larger than leaf
    atomicOr(err, kErrBounds);
    return;
  }
  if (nl > leaf) {
    nx.start[o] = nd.start[k];
    nx.size[o] = nl;
    ++o;
  }
  if (nr > leaf) {
    nx.start[o] = nd.start[k] + nl;
    nx.size[o] = nr;
  }
}

inline unsigned grid1(int64_t n, int t = 256) { return unsigned((n + t - 1) / t); }

// Depth valve.  When pivots cannot separate a node (every member has the same
// code, so d1 == d2 sends all but p1 right) each level peels off one member and
// the depth grows with n; the reference recurses to that depth too.  Past
// kMaxLevels the remaining active nodes are cut into consecutive leaf_size
// leaves.  Real data stays far below (about 40 levels at 1M rows).
constexpr int kMaxLevels = 2048;

__global__ void chunk_leaves(NodeArr nd, int cnt, int leaf, uint8_t* leaf_flag) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const int64_t s = nd.start[k], e = s + nd.size[k];
  for (int64_t p = s; p < e; p += leaf) leaf_flag[p] = 1;
}

// ---- fused levels ------------------------------------------------------------

__device__ __forceinline__ uint32_t gcd32(uint32_t a, uint32_t b) {
  while (b) {
    const uint32_t t = a % b;
    a = b;
    b = t;
  }
  return a;
}

__device__ __forceinline__ int dot16(uint4 v, uint4 a, int acc) {
  acc = __dp4a(int(v.x), int(a.x), acc);
  acc = __dp4a(int(v.y), int(a.y), acc);
  acc = __dp4a(int(v.z), int(a.z), acc);
  return __dp4a(int(v.w), int(a.w), acc);
}

// Pivot table of fused node k, one CTA per node: piv[k][2j], piv[k][2j+1]
// are the pivots of descendant j (j = 0 the node; 2j+1 and 2j+2 the left and
// right children of j), or -1 where j is not split in the pass.  The node's
// candidates are the members at positions a + q*b (mod size), q < S, with b
// coprime to size (distinct positions), in q order; node identity is
// job-local, as for pick_pivots.  Warp 0 chooses the pivots; the candidates'
// sides are split over the 32 8-lane groups (two steps per level: with one
// warp per node the first rounds, a few nodes each, waited 100 us for 16
// steps of dependent gathers).  The CTA also fills the node's part of the
// tile -> node map.
__global__ void __launch_bounds__(256) fuse_pivots(NodeArr nd, int cnt, int64_t n, uint32_t seed,
                                                   const int32_t* __restrict__ perm,
                                                   const int8_t* __restrict__ codes, int d,
                                                   int32_t* __restrict__ piv, int32_t* __restrict__ tile_node,
                                                   int64_t tile_cap, unsigned* err, JobTable jt) {
  __shared__ int32_t s_id[kCand];
  __shared__ int32_t s_node[kCand];
  __shared__ int32_t s_side[kCand];
  __shared__ int32_t s_pv[2 * kFuseNodes];
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, sub = lane & 7, slot = lane >> 3;
  const int k = blockIdx.x;
  const int32_t start = nd.start[k], size = nd.size[k];
  const int S = size < kCand ? int(size) : kCand;
  int32_t cid[2] = {-1, -1};
  int cnode[2] = {-1, -1};
  bool cused[2] = {false, false};
  if (w == 0) {
    const int32_t tree = int32_t(int64_t(start) / n);
    const int32_t in_tree = int32_t(int64_t(start) - int64_t(tree) * n);
    const uint64_t h = node_hash(seed, tree, in_tree - jt.off[job_of(jt, in_tree)], size);
    const uint64_t h2 = splitmix64(h ^ 0x2545F4914F6CDD1Dull);
    const int64_t a = int64_t(h % uint64_t(size));
    int32_t b = 1 + int32_t(h2 % uint64_t(size - 1));  // size > leaf_size >= 2
    while (gcd32(uint32_t(b), uint32_t(size)) != 1) b = b + 1 == size ? 1 : b + 1;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int q = lane + 32 * u;
      if (q < S) {
        cid[u] = perm[start + (a + int64_t(q) * b) % size];
        cnode[u] = 0;
      }
      s_id[q] = cid[u];
      s_node[q] = cnode[u];
    }
    if (lane < 2 * kFuseNodes) s_pv[lane] = -1;
  } else {
    const int32_t f = nd.p1[k], nt = (size + kTileElems - 1) / kTileElems;
    if (f + int64_t(nt) > tile_cap) {  // cannot happen: tiles are counted against max_tiles
      if (tid == 32) atomicOr(err, kErrBounds);
    } else {
      for (int t = tid - 32; t < nt; t += 224) tile_node[f + t] = k;
    }
  }
  const int per_lane = d / 128;
  for (int dk = 0; dk < kFuse; ++dk) {
    const int j0 = (1 << dk) - 1;
    if (w == 0) {
      __syncwarp();
      // pivots of the depth-dk nodes: the two lowest-q free candidates in each
      for (int j = j0; j < 2 * j0 + 1; ++j) {
        const unsigned m0 = __ballot_sync(full, cnode[0] == j && !cused[0]);
        const unsigned m1 = __ballot_sync(full, cnode[1] == j && !cused[1]);
        uint64_t m = uint64_t(m0) | (uint64_t(m1) << 32);
        if (__popcll(m) >= 2) {  // warp-uniform
          const int q1 = __ffsll(m) - 1;
          m &= m - 1;
          const int q2 = __ffsll(m) - 1;
          const int32_t p1 = __shfl_sync(full, (q1 >> 5) ? cid[1] : cid[0], q1 & 31);
          const int32_t p2 = __shfl_sync(full, (q2 >> 5) ? cid[1] : cid[0], q2 & 31);
          if (lane == (q1 & 31)) cused[q1 >> 5] = true;
          if (lane == (q2 & 31)) cused[q2 >> 5] = true;
          if (lane == 0) {
            s_pv[2 * j] = p1;
            s_pv[2 * j + 1] = p2;
          }
        }
      }
    }
    __syncthreads();
    if (dk + 1 == kFuse) break;  // no pivots below the last fused level
    // every candidate in a split depth-dk node takes its side (8 lanes per candidate)
    for (int g = 4 * w; g < S; g += 32) {  // warp-uniform trip count
      const int q = g + slot;  // < kCand
      const int32_t myid = s_id[q];
      const int jn = s_node[q];
      const int32_t p1 = jn >= 0 ? s_pv[2 * jn] : -1;
      const int32_t p2 = jn >= 0 ? s_pv[2 * jn + 1] : -1;
      const bool live = p1 >= 0;
      int d1 = 0, d2 = 0;
      if (live) {
        const uint4* x = reinterpret_cast<const uint4*>(codes + int64_t(myid) * d);
        const uint4* r1 = reinterpret_cast<const uint4*>(codes + int64_t(p1) * d);
        const uint4* r2 = reinterpret_cast<const uint4*>(codes + int64_t(p2) * d);
#pragma unroll 4
        for (int u = 0; u < per_lane; ++u) {
          const uint4 xv = __ldg(x + sub + 8 * u), av = __ldg(r1 + sub + 8 * u), cv = __ldg(r2 + sub + 8 * u);
          d1 = dot16(xv, av, d1);
          d2 = dot16(xv, cv, d2);
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        d1 += __shfl_xor_sync(full, d1, o);
        d2 += __shfl_xor_sync(full, d2, o);
      }
      const int sd = myid == p1 ? 0 : myid == p2 ? 1 : (d1 > d2 ? 0 : 1);
      if (sub == 0) s_side[q] = live ? sd : -1;
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int q = lane + 32 * u;
        if (q < S && cnode[u] >= 0) {
          const int sd = s_side[q];
          cnode[u] = sd < 0 ? -1 : 2 * cnode[u] + 1 + sd;
          s_node[q] = cnode[u];
        }
      }
    }
  }
  if (tid < 2 * kFuseNodes) piv[int64_t(k) * (2 * kFuseNodes) + tid] = s_pv[tid];
}

// Member pass of the fused levels: one block per tile of <= 256 members of one
// node.  Every member's dots with all of the node's (up to 14) pivot rows are
// one tensor-core product, members x pivots, in f16 with fp32 accumulation,
// which is exact (f16_codes.cuh).  A warp takes 32 members (two
// mma.m16n8k16 row tiles) against 16 columns; a lane reads 16 consecutive
// codes of its rows (the K order is free as long as the pivots follow it) and
// widens them in registers; the pivots are widened once per block into shared
// memory, in the order the lanes read them.  Column 2j, 2j + 1 are the pivots
// of descendant j, so lane c of a row holds both dots of descendants c and
// 4 + c and decides their sides; the lanes exchange the seven bits and walk
// the member's path.  side[e] = the member's path code; per tile and code the
// member count, at bins[8*f + code*nt + (tile - f)] (f: the node's first tile,
// nt: its tile count), so one exclusive scan of bins gives every member's
// place.
// Per member: d bytes of HBM (44 SM cycles at d = 1024), 52 instructions, 8
// tensor instructions of 8 cycles, 2 shared-memory loads.  The dp4a form (the
// member's own path only, 6 dots, 8 lanes per member) read 6 KB of pivot rows
// from shared memory per member: 48 cycles that did not overlap the rows'
// latency.  First round at 300k x 1024: 1.10 -> 0.77 ms (6.4 TB/s of rows, 0.94 of
// the measured copy rate); all rounds at 1M 18.4 -> 13.5 ms.  Four CTAs per SM:
// five spill (+15 %), three with a segment loaded ahead are 5 % slower.
constexpr int kPivCols = 16;  // 14 pivots, two columns of zeros

__global__ void __launch_bounds__(256, 4) fuse_side(const int8_t* __restrict__ codes, int d,
                                                    const int32_t* __restrict__ perm, NodeArr nd,
                                                    const int32_t* __restrict__ tile_node,
                                                    const int32_t* __restrict__ piv, uint8_t* __restrict__ side,
                                                    int32_t* __restrict__ bins) {
  // [d / 64][2 column tiles][2 halves][32 lanes] 16-byte pieces: lane (g, c) of
  // column tile t finds pivot 8t + g's codes 16c..16c + 15 of the segment,
  // widened, 8 in each half
  extern __shared__ uint4 s_piv[];
  __shared__ int32_t spv[kPivCols];
  __shared__ int32_t sbins[kFuseBins];
  const unsigned full = 0xffffffffu;
  const int b = blockIdx.x, tid = threadIdx.x;
  const int k = tile_node[b];
  if (tid < kFuseBins) sbins[tid] = 0;
  if (tid < kPivCols) spv[tid] = tid < 2 * kFuseNodes ? piv[int64_t(k) * (2 * kFuseNodes) + tid] : -1;
  __syncthreads();
  const int nseg = d / 64;
  for (int q = tid; q < kPivCols * 4 * nseg; q += 256) {
    const int r = q / (4 * nseg), sc = q % (4 * nseg);  // pivot, 16-byte chunk of its row
    const int32_t id = spv[r];
    uint4 v = make_uint4(0, 0, 0, 0);
    if (id >= 0) v = __ldg(reinterpret_cast<const uint4*>(codes + int64_t(id) * d) + sc);
    uint4 h0, h1;
    widen4(v.x, h0.x, h0.y);
    widen4(v.y, h0.z, h0.w);
    widen4(v.z, h1.x, h1.y);
    widen4(v.w, h1.z, h1.w);
    uint4* dst = s_piv + ((sc >> 2) * 4 + (r >> 3) * 2) * 32 + (r & 7) * 4 + (sc & 3);
    dst[0] = h0;
    dst[32] = h1;
  }
  __syncthreads();
  const int32_t start = nd.start[k], size = nd.size[k];
  const int f = nd.p1[k], nt = (size + kTileElems - 1) / kTileElems;
  const int64_t e0 = int64_t(start) + int64_t(b - f) * kTileElems;
  const int ne = int(min(int64_t(kTileElems), int64_t(start) + size - e0));  // members of this tile
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
  if (32 * warp < ne) {  // warp-uniform
    // rows 8u + g of the warp's 32 members (past the end: the tile's last one)
    int32_t id[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) id[u] = perm[e0 + min(32 * warp + 8 * u + g, ne - 1)];
    const int8_t* lane_codes = codes + 16 * c;
    float acc[2][2][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][t][e] = 0.f;
#pragma unroll 1
    for (int s = 0; s < nseg; ++s) {
      uint4 raw[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        raw[u] = __ldg(reinterpret_cast<const uint4*>(lane_codes + int64_t(id[u]) * d + 64 * s));
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint4 b0 = s_piv[(s * 4 + h) * 32 + lane], b1 = s_piv[(s * 4 + 2 + h) * 32 + lane];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t f0[4], f1[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            widen4(h == 0 ? (q == 0 ? raw[u].x : raw[u].y) : (q == 0 ? raw[u].z : raw[u].w), f0[u], f1[u]);
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            mma16816(acc[m][0], f0[2 * m], f0[2 * m + 1], f1[2 * m], f1[2 * m + 1], q ? b0.z : b0.x, q ? b0.w : b0.y);
            mma16816(acc[m][1], f0[2 * m], f0[2 * m + 1], f1[2 * m], f1[2 * m + 1], q ? b1.z : b1.x, q ? b1.w : b1.y);
          }
        }
      }
    }
    // bit j of byte u: member 8u + g's side at descendant j
    uint32_t sides = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int j = 4 * t + c;
        const float d1 = acc[u >> 1][t][2 * (u & 1)], d2 = acc[u >> 1][t][2 * (u & 1) + 1];
        const bool right = id[u] != spv[2 * j] && (id[u] == spv[2 * j + 1] || !(d1 > d2));
        sides |= right ? 1u << (8 * u + j) : 0u;
      }
    sides |= __shfl_xor_sync(full, sides, 1);
    sides |= __shfl_xor_sync(full, sides, 2);
    // lane c walks member 8c + g's path
    const int x = 32 * warp + 8 * c + g;
    if (x < ne) {
      int j = 0, code = 0;
#pragma unroll
      for (int dk = 0; dk < kFuse; ++dk) {
        if (j < kFuseNodes && spv[2 * j] >= 0) {
          const int bit = int(sides >> (8 * c + j)) & 1;
          code |= bit << (kFuse - 1 - dk);
          j = 2 * j + 1 + bit;
        } else {
          j = kFuseNodes;  // not split below
        }
      }
      side[e0 + x] = uint8_t(code);
      atomicAdd(&sbins[code], 1);
    }
  }
  __syncthreads();
  if (tid < kFuseBins) bins[8 * int64_t(f) + int64_t(tid) * nt + (b - f)] = sbins[tid];
}

// Stable counting sort of each node's members by path code into perm_tmp.
__global__ void __launch_bounds__(256) fuse_scatter(const int32_t* __restrict__ perm,
                                                    int32_t* __restrict__ perm_tmp, NodeArr nd,
                                                    const int32_t* __restrict__ tile_node,
                                                    const uint8_t* __restrict__ side,
                                                    const int32_t* __restrict__ bins_off) {
  __shared__ int32_t wcnt[8][kFuseBins];
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = tile_node[b];
  const int32_t start = nd.start[k], size = nd.size[k];
  const int f = nd.p1[k], nt = (size + kTileElems - 1) / kTileElems;
  const int64_t e0 = int64_t(start) + int64_t(b - f) * kTileElems;
  const int64_t e1 = min(int64_t(start) + size, e0 + kTileElems);
  const int64_t e = e0 + tid;
  const bool valid = e < e1;
  const int code = valid ? int(side[e]) : kFuseBins;
  int rank = 0;
#pragma unroll
  for (int v = 0; v < kFuseBins; ++v) {
    const unsigned bal = __ballot_sync(0xffffffffu, code == v);
    if (code == v) rank = __popc(bal & ((1u << lane) - 1u));
    if (lane == 0) wcnt[warp][v] = __popc(bal);
  }
  __syncthreads();
  if (valid) {
    int pre = 0;
    for (int w = 0; w < warp; ++w) pre += wcnt[w][code];
    const int64_t base = int64_t(8) * f;
    const int32_t before = bins_off[base + int64_t(code) * nt + (b - f)] - bins_off[base];
    perm_tmp[int64_t(start) + before + pre + rank] = perm[e];
  }
}

// perm takes the sorted members over.
__global__ void __launch_bounds__(256) fuse_copyback(int32_t* __restrict__ perm, const int32_t* __restrict__ perm_tmp,
                                                     NodeArr nd, const int32_t* __restrict__ tile_node) {
  const int b = blockIdx.x, k = tile_node[b];
  const int64_t start = nd.start[k];
  const int64_t e = start + int64_t(b - nd.p1[k]) * kTileElems + threadIdx.x;
  if (e < start + nd.size[k]) perm[e] = perm_tmp[e];
}

// After a fused pass: the sizes of node k's descendants from the scanned code
// counts; leaves are flagged, and every descendant that is neither a leaf nor
// split in the pass becomes a node: of the next fused round when it has at
// least kFuseMin members (with its tiles reserved), else parked for the
// subtree kernel, with its depth (the levels done when this round ends) in p1.
// counts: nodes of the next round, their tiles, parked nodes.
__global__ void fuse_children(NodeArr nd, int cnt, int leaf, const int32_t* __restrict__ bins_off,
                              const int32_t* __restrict__ piv, uint8_t* __restrict__ leaf_flag, int32_t* counts,
                              NodeArr big, NodeArr small, int32_t depth, int64_t cap, unsigned* err) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const int32_t start = nd.start[k], size = nd.size[k];
  const int f = nd.p1[k], nt = (size + kTileElems - 1) / kTileElems;
  const int64_t base = int64_t(8) * f;
  int32_t pre[kFuseBins + 1];
  pre[0] = 0;
#pragma unroll
  for (int v = 0; v + 1 < kFuseBins; ++v) pre[v + 1] = bins_off[base + int64_t(v + 1) * nt] - bins_off[base];
  pre[kFuseBins] = size;
  bool split[kFuseNodes];
#pragma unroll
  for (int j = 0; j < kFuseNodes; ++j) split[j] = j == 0;
#pragma unroll
  for (int j = 0; j < kFuseNodes; ++j) {
    if (!split[j]) continue;
    const int dk = 31 - __clz(j + 1), cd = dk + 1;
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      const int ch = 2 * j + 1 + sd, p = ch - ((1 << cd) - 1);
      const int lo = p << (kFuse - cd), hi = (p + 1) << (kFuse - cd);
      const int32_t csize = pre[hi] - pre[lo];
      const int64_t cstart = int64_t(start) + pre[lo];
      if (csize <= 0) {  // cannot happen: a split sends its two pivots to different sides
        atomicOr(err, kErrBounds);
      } else if (csize <= leaf) {
        leaf_flag[cstart] = 1;
      } else if (cd < kFuse && piv[int64_t(k) * (2 * kFuseNodes) + 2 * ch] >= 0) {
        split[ch] = true;
      } else {
        const bool is_big = csize >= kFuseMin;
        const int o = atomicAdd(counts + (is_big ? 0 : 2), 1);
        if (o >= cap) {  // cannot happen: active nodes are disjoint and larger than leaf
          atomicOr(err, kErrBounds);
        } else if (is_big) {
          big.start[o] = int32_t(cstart);
          big.size[o] = csize;
          big.p1[o] = atomicAdd(counts + 1, (csize + kTileElems - 1) / kTileElems);
        } else {
          small.start[o] = int32_t(cstart);
          small.size[o] = csize;
          small.p1[o] = depth;
        }
      }
    }
  }
}

// Splits a parked node (fewer than kFuseMin members) down to its leaves, one
// CTA per node, level by level over all of its open descendants: the per-level
// rule's pivots (pick_pivots), stable splits and depth valve, with the node's
// part of the permutation in shared memory.  8 lanes per member and level: the
// member's row is read (by then from L2, for the most part), the pivot rows
// are staged in shared memory while at most kSubStage descendants are open
// (with the default leaf size at most 7 are).  Bound by those reads: the
// shared-memory pipe is 76 % busy at 300k x 1024 (1.78 ms); a warp per four
// members with the pivots in registers made the forest 3 to 20 % slower.  It replaces 10 to 16 rounds of
// 8 to 10 launches and two host waits each: with the wider fuse_pivots and one
// wait per fused round the forest went from 0.97 to 0.24 ms at 2,000 x 384,
// 4.71 to 2.66 ms at 100,000 x 1024 and 34.2 to 26.0 ms at 1M x 1024.
constexpr int kSubStage = 16;
constexpr int kSubNodes = 256;  // more open descendants than kFuseMin members can hold (each has at least 3)

template <int PL>  // 16-byte chunks per lane: d / 128
__global__ void __launch_bounds__(256) subtree_kernel(const int8_t* __restrict__ codes, int32_t* __restrict__ perm,
                                                      NodeArr nd, int64_t n, uint32_t seed, int leaf,
                                                      uint8_t* __restrict__ leaf_flag, int level0,
                                                      int32_t* __restrict__ max_level, JobTable jt) {
  constexpr int d = 128 * PL;
  extern __shared__ uint4 s_prow[];  // [2 * kSubStage][8 * PL]
  __shared__ int32_t s_perm[2][kFuseMin];
  __shared__ int16_t s_lpre[kFuseMin + 1];    // lefts before each position
  __shared__ int16_t s_node[kFuseMin];        // open descendant of each position, -1: in a leaf
  __shared__ uint8_t s_side[kFuseMin];
  __shared__ int16_t s_start[2][kSubNodes], s_size[2][kSubNodes];
  __shared__ int16_t s_nl[kSubNodes], s_cl[kSubNodes], s_cr[kSubNodes];
  __shared__ int32_t s_p1[kSubNodes], s_p2[kSubNodes];
  __shared__ int s_wcnt[16];
  __shared__ int s_next;
  __shared__ int32_t s_local, s_depth;
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane & 7;
  const int k0 = blockIdx.x;
  const int32_t start = nd.start[k0], size = nd.size[k0];
  const int32_t tree = int32_t(int64_t(start) / n);
  if (tid == 0) {
    const int32_t in_tree = int32_t(int64_t(start) - int64_t(tree) * n);
    s_local = in_tree - jt.off[job_of(jt, in_tree)];
    s_start[0][0] = 0;
    s_size[0][0] = int16_t(size);
    s_depth = nd.p1[k0];
  }
  for (int t = tid; t < size; t += 256) {
    s_perm[0][t] = perm[int64_t(start) + t];
    s_node[t] = 0;
  }
  // The valve counts from the node's own depth: a node of another tree or job
  // that kept the fused rounds going (thousands of equal rows) does not close
  // it.  The depth stays in shared memory: in a register beside the level it
  // made some dimensions spill (500,009 x 768 8.00 -> 8.14 ms, here 8.02).
  int cnt = 1, cur = 0, level = 0;
  __syncthreads();
  while (cnt > 0) {  // a level closes every node it splits; children are smaller: ends
    if (level + s_depth >= kMaxLevels) {  // depth valve: the rest become consecutive leaves
      for (int k = tid; k < cnt; k += 256)
        for (int p = s_start[cur][k], e = p + s_size[cur][k]; p < e; p += leaf) leaf_flag[int64_t(start) + p] = 1;
      break;
    }
    for (int k = tid; k < cnt; k += 256) {
      const int32_t st = s_start[cur][k], sz = s_size[cur][k];
      const uint64_t h = node_hash(seed, tree, s_local + st, sz);
      const uint64_t h2 = splitmix64(h ^ 0x5851F42D4C957F2Dull);
      const int32_t a = int32_t(h % uint64_t(sz));
      int32_t b = int32_t(h2 % uint64_t(sz - 1));
      if (b >= a) ++b;
      s_p1[k] = s_perm[cur][st + a];
      s_p2[k] = s_perm[cur][st + b];
    }
    __syncthreads();
    if (tid == 0) s_next = 0;  // everyone has read it; counted up two barriers on
    const bool staged = cnt <= kSubStage;
    if (staged) {
      for (int c = tid; c < 2 * cnt * 8 * PL; c += 256) {
        const int r = c / (8 * PL), cc = c % (8 * PL);
        const int32_t id = (r & 1) ? s_p2[r >> 1] : s_p1[r >> 1];
        s_prow[c] = __ldg(reinterpret_cast<const uint4*>(codes + int64_t(id) * d) + cc);
      }
      __syncthreads();
    }
    for (int t0 = 0; t0 < size; t0 += 32) {  // 32 members per step, 4 per warp
      const int t = t0 + (tid >> 3);
      const int k = t < size ? int(s_node[t]) : -1;
      if (!__any_sync(full, k >= 0)) continue;  // warp-uniform
      int d1 = 0, d2 = 0;
      int32_t id = -1;
      if (k >= 0) {
        id = s_perm[cur][t];
        const uint4* row = reinterpret_cast<const uint4*>(codes + int64_t(id) * d) + sub;
        uint4 v[PL];
#pragma unroll
        for (int u = 0; u < PL; ++u) v[u] = __ldg(row + 8 * u);
        if (staged) {
          const uint4* a = s_prow + (2 * k) * (8 * PL) + sub;
#pragma unroll
          for (int u = 0; u < PL; ++u) {
            d1 = dot16(v[u], a[8 * u], d1);
            d2 = dot16(v[u], a[8 * PL + 8 * u], d2);
          }
        } else {
          const uint4* a = reinterpret_cast<const uint4*>(codes + int64_t(s_p1[k]) * d) + sub;
          const uint4* c = reinterpret_cast<const uint4*>(codes + int64_t(s_p2[k]) * d) + sub;
#pragma unroll
          for (int u = 0; u < PL; ++u) {
            d1 = dot16(v[u], __ldg(a + 8 * u), d1);
            d2 = dot16(v[u], __ldg(c + 8 * u), d2);
          }
        }
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        d1 += __shfl_xor_sync(full, d1, o);
        d2 += __shfl_xor_sync(full, d2, o);
      }
      if (sub == 0 && k >= 0) s_side[t] = (id == s_p1[k]) || (id != s_p2[k] && d1 > d2) ? 1 : 0;
    }
    __syncthreads();
    // lefts before every position
    unsigned bal[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = tid + 256 * u;
      bal[u] = __ballot_sync(full, t < size && s_node[t] >= 0 && s_side[t]);
      if (lane == 0) s_wcnt[8 * u + warp] = __popc(bal[u]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = tid + 256 * u;
      int before = __popc(bal[u] & ((1u << lane) - 1u));
      for (int w = 0; w < 8 * u + warp; ++w) before += s_wcnt[w];
      if (t < size) s_lpre[t] = int16_t(before);
      if (t == size - 1) s_lpre[size] = int16_t(before + int((bal[u] >> lane) & 1u));
    }
    __syncthreads();
    for (int k = tid; k < cnt; k += 256) {
      const int st = s_start[cur][k], sz = s_size[cur][k];
      const int nl = s_lpre[st + sz] - s_lpre[st], nr = sz - nl;
      s_nl[k] = int16_t(nl);
      s_cl[k] = s_cr[k] = -1;
      if (nl <= leaf) {
        leaf_flag[int64_t(start) + st] = 1;
      } else {
        const int o = atomicAdd(&s_next, 1);
        s_cl[k] = int16_t(o);
        s_start[cur ^ 1][o] = int16_t(st);
        s_size[cur ^ 1][o] = int16_t(nl);
      }
      if (nr <= leaf) {
        leaf_flag[int64_t(start) + st + nl] = 1;
      } else {
        const int o = atomicAdd(&s_next, 1);
        s_cr[k] = int16_t(o);
        s_start[cur ^ 1][o] = int16_t(st + nl);
        s_size[cur ^ 1][o] = int16_t(nr);
      }
    }
    __syncthreads();
    for (int t = tid; t < size; t += 256) {
      const int k = s_node[t];
      int np = t;
      if (k >= 0) {
        const int st = s_start[cur][k], l = s_lpre[t] - s_lpre[st];
        np = s_side[t] ? st + l : st + s_nl[k] + (t - st - l);
        s_node[t] = t - st < s_nl[k] ? s_cl[k] : s_cr[k];  // of position t, whoever moves there
      }
      s_perm[cur ^ 1][np] = s_perm[cur][t];
    }
    __syncthreads();
    cnt = s_next;
    cur ^= 1;
    ++level;
  }
  for (int t = tid; t < size; t += 256) perm[int64_t(start) + t] = s_perm[cur][t];
  if (tid == 0) atomicMax(max_level, level0 + level);
}

template <int PL>
cudaError_t run_subtree(const int8_t* codes, int32_t* perm, const NodeArr& nd, int64_t cnt, int64_t n, uint32_t seed,
                        int leaf, uint8_t* leaf_flag, int level0, int32_t* max_level, const JobTable& jt,
                        cudaStream_t s) {
  const size_t smem = size_t(2) * kSubStage * 128 * PL;
  KNNG_CUDA_TRY(ensure_smem_attr(reinterpret_cast<const void*>(subtree_kernel<PL>), smem));
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  subtree_kernel<PL><<<unsigned(cnt), 256, smem, s>>>(codes, perm, nd, n, seed, leaf, leaf_flag, level0, max_level, jt);
  note_launch();
  return cudaGetLastError();
}

}  // namespace

int64_t forest_tiles(int64_t n) { return (n + kTileElems - 1) / kTileElems; }

size_t forest_bytes(int64_t n, int T, int leaf, int64_t* max_nodes, int64_t* max_tiles) {
  const int64_t mn = int64_t(T) * (n / (leaf + 1) + 1) + 16;
  const int64_t mt = int64_t(T) * n / kTileElems + mn + 16;
  if (max_nodes) *max_nodes = mn;
  if (max_tiles) *max_tiles = mt;
  size_t b = 0;
  b += size_t(T) * n * 4;                      // perm_tmp
  b += size_t(T) * n;                          // side (path codes)
  b += 3 * size_t(4 * mn) * 4;                 // node generations, parked nodes
  b += size_t(mn + 1) * 4 * 3;                 // tile_off, child_cnt, child_cnt2
  b += size_t(mn) * (2 * kFuseNodes) * 4;      // pivot tables
  b += 2 * size_t(kFuseBins) * size_t(mt) * 4; // tile_bins, tile_bins_off (tile_left, tile_left_off)
  b += scan_tmp_bytes(std::max<int64_t>(mn, int64_t(kFuseBins) * mt)) + 4096;
  return b;
}

int run_forest(const int8_t* codes, int64_t n, int d, int T, int leaf, uint32_t seed, const int32_t* replay_host,
               int64_t n_replay, int32_t* perm, uint8_t* leaf_flag, const ForestBufs& fb, cudaStream_t s,
               int64_t* levels_out, std::string* err, const JobTable& jt, int roots_with_split, int64_t root_tiles,
               int fuse) {
  auto fail = [&](cudaError_t e, const char* what) {
    if (err) *err = std::string(what) + ": " + cudaGetErrorString(e);
    return int(KNNG_E_CUDA);
  };
  cudaError_t e;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // replay table: sort by (level, tree, start) and index each level's slice
  std::vector<int32_t> rep;
  std::vector<int64_t> lvl_off;
  if (replay_host) {
    std::vector<int64_t> idx(n_replay);
    for (int64_t i = 0; i < n_replay; ++i) idx[i] = i;
    std::sort(idx.begin(), idx.end(), [&](int64_t a, int64_t b) {
      const int32_t* ra = replay_host + 6 * a;
      const int32_t* rb = replay_host + 6 * b;
      if (ra[1] != rb[1]) return ra[1] < rb[1];
      if (ra[0] != rb[0]) return ra[0] < rb[0];
      return ra[2] < rb[2];
    });
    rep.resize(6 * n_replay);
    for (int64_t i = 0; i < n_replay; ++i)
      std::copy(replay_host + 6 * idx[i], replay_host + 6 * idx[i] + 6, rep.begin() + 6 * i);
    int32_t maxl = n_replay ? rep[6 * (n_replay - 1) + 1] : -1;
    lvl_off.assign(size_t(maxl + 2), 0);
    for (int64_t i = 0; i < n_replay; ++i) lvl_off[size_t(rep[6 * i + 1]) + 1]++;
    for (size_t l = 1; l < lvl_off.size(); ++l) lvl_off[l] += lvl_off[l - 1];
    if (n_replay) {
      e = cudaMemcpyAsync(fb.replay_dev, rep.data(), rep.size() * 4, cudaMemcpyHostToDevice, s);
      if (e) return fail(e, "replay upload");
    }
  }
  e = cudaMemsetAsync(leaf_flag, 0, size_t(T) * n, s);
  if (e) return fail(e, "leaf_flag clear");
  e = cudaMemsetAsync(fb.err, 0, sizeof(unsigned), s);
  if (e) return fail(e, "err clear");
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  init_perm<<<std::min<int64_t>(grid1(n * T), int64_t(sms) * 16), 256, 0, s>>>(perm, n, T);
  note_launch();
  NodeArr cur = node_arr(fb.node_a, fb.max_nodes), nxt = node_arr(fb.node_b, fb.max_nodes);
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  root_nodes<<<1, 64, 0, s>>>(cur, n, T, leaf, leaf_flag, jt, roots_with_split, int(root_tiles));
  note_launch();
  int64_t cnt = int64_t(T) * roots_with_split;
  int level = 0;
  int64_t host_i64[3];
  if (fuse && !replay_host) {
    // fused rounds: kFuse levels per pass over nodes of >= kFuseMin members;
    // smaller nodes collect in `parked` for the subtree kernel.  The host only
    // waits for the next round's node and tile counts.
    NodeArr parked = node_arr(fb.node_c, fb.max_nodes);
    int32_t* counts = reinterpret_cast<int32_t*>(fb.dev_i64);  // next round's nodes, its tiles; parked nodes
    int32_t* tile_node = fb.child_cnt2;  // at most one tile per leaf_size + 1 members: fits
    int32_t host_cnt[3] = {0, 0, 0};
    int64_t tiles = int64_t(T) * root_tiles;
    const size_t side_smem = size_t(kPivCols) * d * 2;
    if ((e = ensure_smem_attr(reinterpret_cast<const void*>(fuse_side), side_smem))) return fail(e, "forest smem");
    if ((e = cudaMemsetAsync(fb.dev_i64, 0, 32, s))) return fail(e, "node counts");
    while (cnt > 0 && level < kMaxLevels) {
      if (tiles > fb.max_tiles || tiles > fb.max_nodes) {  // the tile -> node map has max_nodes entries
        if (err) *err = "forest tile overflow";
        return KNNG_E_ARGS;
      }
      cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
      fuse_pivots<<<unsigned(cnt), 256, 0, s>>>(cur, int(cnt), n, seed, perm, codes, d, fb.piv, tile_node,
                                                fb.max_nodes, fb.err, jt);
      note_launch();
      cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
      fuse_side<<<unsigned(tiles), 256, side_smem, s>>>(codes, d, perm, cur, tile_node, fb.piv, fb.side, fb.tile_bins);
      note_launch();
      if ((e = exclusive_scan_i32(fb.tile_bins, fb.tile_bins_off, int64_t(kFuseBins) * tiles, nullptr, fb.scan_tmp, s)))
        return fail(e, "code scan");
      cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
      fuse_children<<<grid1(cnt, 64), 64, 0, s>>>(cur, int(cnt), leaf, fb.tile_bins_off, fb.piv, leaf_flag, counts, nxt,
                                                  parked, level + kFuse, fb.max_nodes, fb.err);
      note_launch();
      // the counts first: the next round is queued while the members are sorted
      if ((e = cudaMemcpyAsync(host_cnt, counts, sizeof(host_cnt), cudaMemcpyDeviceToHost, s)) ||
          (e = cudaStreamSynchronize(s)) || (e = cudaMemsetAsync(counts, 0, 2 * sizeof(int32_t), s)))
        return fail(e, "fused forest round");
      cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
      fuse_scatter<<<unsigned(tiles), 256, 0, s>>>(perm, fb.perm_tmp, cur, tile_node, fb.side, fb.tile_bins_off);
      note_launch();
      fuse_copyback<<<unsigned(tiles), 256, 0, s>>>(perm, fb.perm_tmp, cur, tile_node);
      note_launch();
      if ((e = cudaGetLastError())) return fail(e, "fused forest round");
      cnt = host_cnt[0];
      tiles = host_cnt[1];
      if (cnt > fb.max_nodes || host_cnt[2] > fb.max_nodes) {
        if (err) *err = "forest node overflow";
        return KNNG_E_ARGS;
      }
      std::swap(cur, nxt);
      level += kFuse;
    }
    if (cnt > 0) {  // depth valve (see kMaxLevels): the rest become consecutive leaves
      cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
      chunk_leaves<<<grid1(cnt), 256, 0, s>>>(cur, int(cnt), leaf, leaf_flag);
      note_launch();
    }
    cnt = 0;
    if (host_cnt[2] > 0) {
      int32_t* max_level = reinterpret_cast<int32_t*>(fb.dev_i64 + 3);
      const int64_t parked_cnt = host_cnt[2];
#define KNNG_SUBTREE(PL) \
  case PL: e = run_subtree<PL>(codes, perm, parked, parked_cnt, n, seed, leaf, leaf_flag, level, max_level, jt, s); break;
      switch (d / 128) {
        KNNG_SUBTREE(1) KNNG_SUBTREE(2) KNNG_SUBTREE(3) KNNG_SUBTREE(4)
        KNNG_SUBTREE(5) KNNG_SUBTREE(6) KNNG_SUBTREE(7) KNNG_SUBTREE(8)
        default: e = cudaErrorInvalidValue;
      }
#undef KNNG_SUBTREE
      if (e) return fail(e, "forest subtrees");
      int32_t deepest = 0;
      if ((e = cudaMemcpyAsync(&deepest, max_level, sizeof(int32_t), cudaMemcpyDeviceToHost, s)) ||
          (e = cudaStreamSynchronize(s)))
        return fail(e, "forest subtrees");
      level = std::max(level, deepest);
    }
  }
  while (cnt > 0) {
    if (level >= kMaxLevels) {
      cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
      chunk_leaves<<<grid1(cnt), 256, 0, s>>>(cur, int(cnt), leaf, leaf_flag);
      note_launch();
      break;
    }
    const int32_t* rep_dev = nullptr;
    if (replay_host) {
      if (size_t(level) + 1 >= lvl_off.size() || lvl_off[level + 1] - lvl_off[level] != cnt) {
        if (err) *err = "replay table does not match the forest at level " + std::to_string(level);
        return KNNG_E_REPLAY;
      }
      rep_dev = fb.replay_dev + 6 * lvl_off[level];
    }
    cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
    pick_pivots<<<grid1(cnt), 256, 0, s>>>(cur, int(cnt), n, seed, level, perm, rep_dev, fb.child_cnt, fb.err, jt);
    note_launch();
    if ((e = exclusive_scan_i32(fb.child_cnt, fb.tile_off, cnt, fb.dev_i64, fb.scan_tmp, s))) return fail(e, "tile scan");
    if ((e = cudaMemcpyAsync(host_i64, fb.dev_i64, 8, cudaMemcpyDeviceToHost, s))) return fail(e, "tile count");
    if ((e = cudaStreamSynchronize(s))) return fail(e, "forest level");
    const int64_t tiles = host_i64[0];
    if (tiles > fb.max_tiles) {
      if (err) *err = "forest tile overflow";
      return KNNG_E_ARGS;
    }
    cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
    side_kernel<<<unsigned(tiles), 256, 0, s>>>(codes, d, perm, cur, int(cnt), fb.tile_off, fb.side, fb.tile_left);
    note_launch();
    if ((e = exclusive_scan_i32(fb.tile_left, fb.tile_left_off, tiles, nullptr, fb.scan_tmp, s))) return fail(e, "left scan");
    cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
    scatter_kernel<<<unsigned(tiles), 256, 0, s>>>(perm, fb.perm_tmp, cur, int(cnt), fb.tile_off, fb.side,
                                                   fb.tile_left, fb.tile_left_off);
    note_launch();
    cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
    copyback_kernel<<<unsigned(tiles), 256, 0, s>>>(perm, fb.perm_tmp, cur, int(cnt), fb.tile_off);
    note_launch();
    cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
    children_count<<<grid1(cnt), 256, 0, s>>>(cur, int(cnt), leaf, fb.tile_off, fb.tile_left, fb.tile_left_off,
                                              leaf_flag, fb.child_cnt);
    note_launch();
    if ((e = exclusive_scan_i32(fb.child_cnt, fb.child_cnt, cnt, fb.dev_i64 + 1, fb.scan_tmp, s))) return fail(e, "child scan");
    cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
    children_emit<<<grid1(cnt), 256, 0, s>>>(cur, int(cnt), leaf, fb.tile_off, fb.tile_left, fb.tile_left_off,
                                             fb.child_cnt, nxt, fb.max_nodes, fb.err);
    note_launch();
    if ((e = cudaMemcpyAsync(host_i64 + 1, fb.dev_i64 + 1, 8, cudaMemcpyDeviceToHost, s))) return fail(e, "child count");
    if ((e = cudaStreamSynchronize(s))) return fail(e, "forest level");
    cnt = host_i64[1];
    if (cnt > fb.max_nodes) {
      if (err) *err = "forest node overflow";
      return KNNG_E_ARGS;
    }
    std::swap(cur, nxt);
    ++level;
  }
  unsigned herr = 0;
  if ((e = cudaMemcpyAsync(&herr, fb.err, sizeof(unsigned), cudaMemcpyDeviceToHost, s))) return fail(e, "err read");
  if ((e = cudaStreamSynchronize(s))) return fail(e, "forest");
  if (herr & kErrBounds) {
    if (err) *err = "forest node list overflow";
    return KNNG_E_ARGS;
  }
  if (herr & kErrReplay) {
    if (err) *err = "replay pivot table does not match the forest nodes";
    return KNNG_E_REPLAY;
  }
  if (replay_host && size_t(level) + 1 != lvl_off.size()) {
    if (err) *err = "replay table has more levels than the forest";
    return KNNG_E_REPLAY;
  }
  if (levels_out) *levels_out = level;
  return 0;
}

}  // namespace knng
