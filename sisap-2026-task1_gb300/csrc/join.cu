// join.cu -- K5: one NN-Descent iteration, one CTA (8 warps) per row at a time.
//
// Reference: src/main.cpp:324-430.  For row i:
//   candidates c_j = G[G[i][k]][k2], j = k*K + k2, minus i;
//   h_j = 1024 - sum_w popcount(b_i[w] ^ b_c[w]);
//   the R = K*rerank_mult best by h are visited in order, skipped when the id
//   is in the row's current pool, otherwise scored by exact int8 dot and
//   shift-inserted when dot > pool[K-1].score (existing entries keep ties);
//   positions whose id changed are written back and counted.
// The reference picks the R best with std::nth_element (ties unspecified) and
// visits them in the order it leaves.  Here the R best are taken by
// (h desc, j asc) and visited in that order, which the oracle's TIE_STABLE
// mode reproduces; every other step is the reference's sequential semantics.
//
// Only visits that can change the pool need work: a candidate whose id sits
// in the starting pool with a real score is either still there (skipped) or
// was evicted with a score <= the rising threshold (rejected), and a
// candidate whose dot is <= the starting pool[K-1].score is always rejected.
// So the kernel computes dots for the selected candidates not in the starting
// pool and keeps those above the starting threshold ("survivors"), whose
// insertion in visit order (h desc, j asc) is then resolved by rank counting.
//
// Duplicates: about half of the K*K two-hop candidates of a row repeat an id
// (1317 distinct of 2500 at 6.35M rows).  Every occurrence of an id has the
// same h, so h and the dot are computed once per distinct id, at its first
// occurrence (its "representative").  Among the occurrences of one id only
// the first in visit order can change the list (a later one finds the id in
// the list, or scores <= the threshold that evicted or rejected it), and when
// one occurrence is selected so is the first (ties at the cut are taken in j
// order), so the visit key of a distinct id is (h, first j).
//
// Finding the representatives is what the kernel used to spend most of its
// instructions on: an open-addressing insert per occurrence (a probe loop with
// a compare-and-swap, then an atomic for the first j) took 20k of the 38.6k
// warp instructions of a cached row, with issue slots 61 % busy.  Now it takes
// rounds without probing: every unresolved occurrence does one
// atomicMin(table[hash_round(id)], tag | j); after a barrier the slot holds
// the smallest j that hashed there, so an occurrence whose id equals the
// winner's id has found its representative, the first occurrence, and the
// others go to the next round with another hash.  Each round resolves at least
// the winner of every slot, so it ends; with about 1300 ids in 4096 slots 84 %
// resolve in the first round and three rounds are usual.  Rounds alternate
// between two tables, so one barrier per round separates the inserts from the
// reads, and the tag falls with every round and row, so an older entry loses
// to any newer one and the tables are cleared once per million tags.  The
// row's cached ids and starting list only look ids up in the same rounds: a
// slot without this round's tag says that the id is absent.
//
// Across iterations a row's candidate set barely changes (over 80 % of the
// distinct ids recur from the third iteration on), and its pool threshold
// never falls, so with the candidate cache each row keeps its distinct ids
// with their h and a "dot <= threshold" flag for the next iteration.
//
// Sketches: W 64-bit words per row, d / 64 for the reference's coordinate-sign
// sketch or 2 for the optional 128-hyperplane sketch (hyperplane.cu); the
// score is 1024 - popcount over the W words either way.
//
// What bounds it: instruction issue (63 % busy) and the shared-memory pipe
// (58 %) with four CTAs per SM and a barrier between stages, about 20,000 warp
// instructions per computed row; the first two iterations, where most
// candidates are new, the gathers of sketches and code rows.  Forms that only
// shorten latencies (next row's two-hop ids fetched early, two table losers per
// step, wider threshold scans) changed nothing or cost 1 to 4 %.
// 100,000 x 1024: the phase takes 9.7 ms (probing tables: 19.8), two iterations
// of 300,000 x 1024 rows of 64-dimensional data 45.6 ms (93.6).
//
// Stages per row (shared memory, K = 50, R = 400: 54 KB, FAR 48 KB); thread t
// owns the occurrences j = 2p and 2p + 1 of the pairs p = t + 256r in every
// stage:
//   A  own list (loaded while the previous row was computed); the unchanged-
//      row test; start copying the row's cache entries, code row and sketch
//      into shared memory (cp.async)
//   B  two-hop ids, all loaded first, then one table insert each; rounds as
//      above: rep[j], the first-occurrence bits (registers), info[rep] of the
//      ids found in the cache
//   C  Hamming of the first occurrences without a cached score, each warp its
//      own (CB in flight per 8-lane group, the autotuned candidate block): one
//      16-byte sketch chunk per lane (128-byte rows = one line per
//      candidate), group popcount
//   D  histogram of h over all occurrences; every warp finds the threshold
//      h_t from it
//   E  selection: every occurrence with h > h_t plus the first
//      R - count(h > h_t) occurrences with h == h_t in j order, ranked by
//      ballot counts per (round, warp), where a warp has a tie that could need
//      a dot; the selected first occurrences that are neither starting-list
//      members nor known to be rejected need one
//   F  dp4a dots, a warp per four candidates (short rows: 8 lanes each); keep
//      those above the starting pool[K-1].score, flag the others as rejected
//   G  write the row's cache (this iteration's distinct ids, h and flags);
//      insertion by rank counting over 64-bit survivor keys {dot, visit key}
//      (or the reference's sequential loop for an unsorted or unscored pool),
//      written straight to the output list; the update count
// The row's bookkeeping (update count, flags, statistics) is finished by
// thread 0 after the next row's first barrier, and what the last stage reads
// is not written before that barrier, so a row ends without one.
// Per row HBM/L2 bytes: K*8 (own list) + K*K*4 (two-hop ids) + d + d/8 (own
// row, sketch) + U*d/8 (U sketches scored) + r*d (r reranked rows) + 12 per
// distinct id (cache read and write).
#include "knng_internal.cuh"

#include <algorithm>
#include <map>
#include <mutex>
#include <cstdio>
#include <tuple>

namespace knng {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kGroups = kThreads / 8;  // 8-lane groups per CTA
constexpr int kHBins = 1152;           // distances 0..1024, padded to 9 x 128 for the threshold scan
constexpr uint32_t kNoDist = kHBins - 1;     // "distance" of an occurrence without a candidate: behind every real one
constexpr int kMaxPairs = (kMaxK * kMaxK / 2 + kThreads - 1) / kThreads;  // occurrence pairs per thread
constexpr int kCachePairs = kCacheCap / 2 / kThreads;                     // pairs of cached ids per thread
static_assert(kCacheCap % (2 * kThreads) == 0, "cached ids per thread");
constexpr uint32_t kJBits = 12;              // occurrence index j < kMaxK * kMaxK
constexpr uint32_t kJMask = (1u << kJBits) - 1u;
static_assert(kMaxK * kMaxK <= (1 << kJBits), "occurrence index");
constexpr uint32_t kTagTop = 0xffffeu;       // tags count down from here; 0xfffff marks a cleared slot
static_assert(2 * kMaxPairs <= 16 && kMaxPairs * kThreads * 2 < int(0x8000), "an occurrence's bit and entry");
constexpr int kTableB = 1024;                // second table (odd rounds): slots
constexpr int kTableBShift = 22;
constexpr uint32_t kXMask = 0x7ffu;          // info bits 0..10: Hamming distance
constexpr uint32_t kKnown = 0x800u;          // info bit 11: distance taken from the row's candidate cache
constexpr uint32_t kRej = 0x1000u;           // info bit 12: dot known to be <= the row's pool threshold
constexpr uint32_t kPtr = 0x8000u;           // (FAR) entry bit 15: bits 0..14 are the id's first occurrence
constexpr uint32_t kNone = 0xffffffffu;      // ids: no candidate (no id equals it: num_trees * n < 2^31)
// The default parameters get a kernel of their own whose sizes and
// shared-memory offsets are compile-time constants: read from the parameter
// block they cost about 4,000 more instructions per row.
constexpr int kDefK = 50, kDefR = 400;
// FAR form of that kernel: 49 KB of shared memory per CTA instead of 55, which
// leaves four CTAs 60 KB of L1 instead of 28.  Gathers in flight hold L1
// lines, and with rows that come from beyond L2 there are many of them: at
// 300,000 x 1024 (64-dimensional data) the first iteration reads the same
// 113 GB of DRAM in 23.3 ms instead of 32.6.  It saves the space by keeping an
// occurrence's info word and its pointer to the id's first occurrence in one
// entry, and the survivors in the first table, at 2 % more instructions.

// Shared-memory layout of one CTA (byte offsets).
struct JoinLayout {
  int KK;                  // K * K occurrences
  int pairs;               // pairs of consecutive occurrences
  int ta_slots, ta_shift;  // first table: slots and hash shift
  uint32_t kdiv;           // j / K = (j * kdiv) >> 20 for j < 4096
  uint32_t dummy;          // info index of occurrences without a candidate
  uint32_t kp;             // words of a starting list
  uint32_t survivors;      // most survivors of a row
  uint32_t o_code, o_sk, o_ids, o_rep, o_info, o_ta, o_tb, o_hist, o_x, o_pool, o_row, o_cell, o_member;
  uint32_t bytes;
};

__host__ __device__ constexpr uint32_t align16(uint32_t x) { return (x + 15u) & ~15u; }
__host__ __device__ constexpr uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }

__host__ __device__ constexpr JoinLayout join_layout(int K, int R, int d, bool def, bool far) {
  JoinLayout s{};
  s.KK = K * K;
  s.pairs = (s.KK + 1) / 2;
  s.kdiv = ((1u << 20) + uint32_t(K) - 1) / uint32_t(K);
  // first table: 4096 slots for K = 50 (at most 2500 ids, about 1300 usual)
  s.ta_slots = 1024;
  s.ta_shift = 22;
  while (s.ta_slots < (3 * (s.KK + K)) / 2) {
    s.ta_slots <<= 1;
    --s.ta_shift;
  }
  const uint32_t kk = uint32_t(2 * s.pairs), r = uint32_t(R < s.KK ? R : s.KK);
  const uint32_t rounds = uint32_t(def ? (s.pairs + kThreads - 1) / kThreads : kMaxPairs);
  s.survivors = r;
  s.kp = uint32_t(K);
  // behind every occurrence index that a thread of the kernel forms
  s.dummy = rounds * kThreads * 2;
  uint32_t o = 0;
  s.o_ids = o;   o += align16(4 * kk);
  s.o_rep = o;   o += far ? 0 : align16(umax(2 * kk, 14 * r));  // representatives, then the survivors' keys, ids and order
  s.o_info = o;  o += 2 * s.dummy + 16;
  s.o_ta = o;    o += uint32_t(s.ta_slots) * 4;
  s.o_tb = o;    o += kTableB * 4;
  s.o_hist = o;  o += kHBins * 4;  // also the row's cached distances, staged and gathered
  // staged cached ids, then the warps' miss lists, then the rerank list, then
  // the ids of the row's next cache
  s.o_x = o;     o += align16(umax(umax(kCacheCap * 4, uint32_t((s.pairs + kThreads - 1) / kThreads) * kThreads * 4), 2 * r));
  s.o_pool = o;  o += align16(2 * 2 * s.kp * 4);  // starting lists of this row and of the previous one: ids, scores
  s.o_row = o;   o += 2 * 32;             // row counters, by row parity
  s.o_cell = o;  o += align16(rounds * kWarps * 4);  // threshold ties per (round, warp)
  s.o_member = o; o += kThreads * 2;      // 16 bits per thread: its occurrences whose id is in the starting list
  s.o_sk = o;    o += 128;                // the widest sketch
  s.o_code = o;  o += align16(uint32_t(d));
  s.bytes = o;
  return s;
}
static_assert(join_layout(kDefK, kDefR, kMaxDim, true, true).bytes <= 49072, "four FAR CTAs in 196 KB");
// An SM's 228 KB hold four CTAs of 57,344 bytes each (and 1 KB of the system's),
// 80 of them static.  With lists of kMaxK entries the general form missed the
// fourth by 192 bytes at K = 50, R < 400, d = 1024: 100,000 rows, phase at
// R = 350 / 200 / 50: 13.2 / 12.5 / 11.3 ms with three, 12.2 / 11.6 / 10.5 with four.
static_assert(join_layout(kDefK, kDefR - kDefK, kMaxDim, false, false).bytes <= 57264, "four general CTAs at K = 50, R < 400");
static_assert(join_layout(kDefK, kDefR, kMaxDim, true, true).ta_slots * 4 >= 14 * kDefR, "survivors in the first table");
static_assert(kHBins * 4 >= kCacheCap * 2, "the histogram region stages the cached distances");

// A row's counters (byte offsets from its set's start).
enum : uint32_t {
  kRowCnt = 0,       // occurrences with a candidate
  kRowNu = 4,        // distinct candidates
  kRowMiss = 8,      // of these without a cached distance
  kRowNeed = 12,     // selected ones that need a dot
  kRowProm = 16,     // survivors
  kRowChanged = 20,  // list positions whose id changed
};

// Shared memory is addressed through one 32-bit base register: with C++
// pointers into the dynamic array the compiler recomputed the window's base
// (three to four uniform instructions) at most of the accesses, about 5,000
// instructions per row.
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"(uint16_t(v)) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void red_min(uint32_t a, uint32_t v) {
  asm volatile("red.shared.min.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// The table steps, each one piece so that its predicates stay predicates (a
// C++ condition around an asm statement becomes a branch or a 0/1 register).
// Insert: a candidate id (in range, not the row itself) writes `val` to its
// slot and sets `bit`; any other id becomes kNone.
__device__ __forceinline__ void table_insert(uint32_t& id, uint32_t n, uint32_t self, uint32_t slot, uint32_t val,
                                             unsigned& valid, unsigned bit) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.lt.u32 p, %0, %2;\n"
      "setp.ne.and.u32 p, %0, %3, p;\n"
      "@p red.shared.min.u32 [%4], %5;\n"
      "@p or.b32 %1, %1, %6;\n"
      "selp.b32 %0, %0, 0xffffffff, p;\n}"
      : "+r"(id), "+r"(valid)
      : "r"(n), "r"(self), "r"(slot), "r"(val), "r"(bit)
      : "memory");
}
// Settle an occurrence j of `id` whose slot's winner w holds id `got`: a loser
// enters the next round's table and sets its bit in `todo`; the winner itself
// sets its bit in `first`.
template <bool FAR>
__device__ __forceinline__ void table_settle(uint32_t id, uint32_t got, uint32_t& w, uint32_t dummy, uint32_t j, uint32_t a_info, uint32_t next_slot,
                                             uint32_t next_val, unsigned& todo, unsigned& first, unsigned bit) {
  if (FAR) {
    asm volatile(
        "{\n.reg .pred p, q;\n.reg .b32 t;\n"
        "setp.ne.u32 q, %3, 0xffffffff;\n"
        "selp.b32 %2, %2, %5, q;\n"
        "setp.ne.and.u32 p, %4, %3, q;\n"
        "@p red.shared.min.u32 [%7], %8;\n"
        "@p or.b32 %0, %0, %9;\n"
        "setp.eq.u32 q, %2, %6;\n"
        "@q or.b32 %1, %1, %9;\n"
        "or.pred p, p, q;\n"
        "or.b32 t, %2, 0x8000;\n"
        "@!p st.shared.u16 [%10], t;\n}"
        : "+r"(todo), "+r"(first), "+r"(w)
        : "r"(id), "r"(got), "r"(dummy), "r"(j), "r"(next_slot), "r"(next_val), "r"(bit), "r"(a_info + 2 * j)
        : "memory");
  } else {
    asm volatile(
        "{\n.reg .pred p, q;\n"
        "setp.ne.u32 q, %3, 0xffffffff;\n"
        "selp.b32 %2, %2, %5, q;\n"
        "setp.ne.and.u32 p, %4, %3, q;\n"
        "@p red.shared.min.u32 [%7], %8;\n"
        "@p or.b32 %0, %0, %9;\n"
        "setp.eq.u32 q, %2, %6;\n"
        "@q or.b32 %1, %1, %9;\n}"
        : "+r"(todo), "+r"(first), "+r"(w)
        : "r"(id), "r"(got), "r"(dummy), "r"(j), "r"(next_slot), "r"(next_val), "r"(bit)
        : "memory");
  }
}
// Look a cached id up in round 0: `e` is its slot, `base` the round's tag.  A
// slot of an older round: absent.  Else the winner's id decides: equal, and the
// cached info goes to the winner; other, and `bit` asks for the next round.
__device__ __forceinline__ void table_find(uint32_t id, bool live, uint32_t e, uint32_t base, uint32_t a_ids, uint32_t a_info,
                                           uint32_t info, unsigned& todo, unsigned bit) {
  asm volatile(
      "{\n.reg .pred p, q;\n.reg .b32 w, x, a;\n.reg .b16 h;\n"
      "sub.u32 w, %2, %3;\n"
      "setp.ne.u32 p, %7, 0;\n"
      "setp.lt.and.u32 p, w, 4096, p;\n"
      "mov.b32 x, 0xffffffff;\n"
      "mad.lo.u32 a, w, 4, %4;\n"
      "@p ld.shared.u32 x, [a];\n"
      "setp.eq.and.u32 q, x, %1, p;\n"
      "setp.ne.and.u32 p, x, %1, p;\n"
      "mad.lo.u32 a, w, 2, %5;\n"
      "cvt.u16.u32 h, %6;\n"
      "@q st.shared.u16 [a], h;\n"
      "@p or.b32 %0, %0, %8;\n}"
      : "+r"(todo)
      : "r"(id), "r"(e), "r"(base), "r"(a_ids), "r"(a_info), "r"(info), "r"(uint32_t(live)), "r"(bit)
      : "memory");
}
// Threshold step of stage E: `bit` goes to `near` if key < xt, to `at` if dist == xt, to `open` if key == xt.
__device__ __forceinline__ void mark_near(uint32_t key, uint32_t dist, uint32_t xt, unsigned& near, unsigned& at,
                                          unsigned& open, unsigned bit) {
  asm("{\n.reg .pred p, q, t;\n"
      "setp.lt.u32 p, %3, %5;\n"
      "setp.eq.u32 q, %4, %5;\n"
      "setp.eq.u32 t, %3, %5;\n"
      "@p or.b32 %0, %0, %6;\n"
      "@q or.b32 %1, %1, %6;\n"
      "@t or.b32 %2, %2, %6;\n}"
      : "+r"(near), "+r"(at), "+r"(open)
      : "r"(key), "r"(dist), "r"(xt), "r"(bit));
}
// If `bit` of `m` is set: store the half word at `at` and step on.
__device__ __forceinline__ void list_push(unsigned m, unsigned bit, uint32_t& at, uint32_t val) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b32 t;\n.reg .b16 h;\n"
      "and.b32 t, %1, %2;\n"
      "setp.ne.u32 p, t, 0;\n"
      "cvt.u16.u32 h, %3;\n"
      "@p st.shared.u16 [%0], h;\n"
      "@p add.u32 %0, %0, 2;\n}"
      : "+r"(at)
      : "r"(m), "r"(bit), "r"(val)
      : "memory");
}
// The same for an entry of a row's next cache: id and info word, while at < end.
__device__ __forceinline__ void cache_push(unsigned m, unsigned bit, uint32_t& at_id, uint32_t& at_info, uint32_t end,
                                           uint32_t id, uint32_t info) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b32 t;\n.reg .b16 h;\n"
      "and.b32 t, %2, %3;\n"
      "setp.ne.u32 p, t, 0;\n"
      "setp.lt.and.u32 p, %0, %4, p;\n"
      "cvt.u16.u32 h, %6;\n"
      "@p st.shared.u32 [%0], %5;\n"
      "@p st.shared.u16 [%1], h;\n"
      "@p add.u32 %0, %0, 4;\n"
      "@p add.u32 %1, %1, 2;\n}"
      : "+r"(at_id), "+r"(at_info)
      : "r"(m), "r"(bit), "r"(end), "r"(id), "r"(info)
      : "memory");
}
// (FAR) The info word behind an entry: its own, or that of the first occurrence it points to.
__device__ __forceinline__ uint32_t info_of(uint32_t e, uint32_t a_info) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b32 a;\n"
      "setp.ge.u32 p, %0, 0x8000;\n"
      "mad.lo.u32 a, %0, 2, %1;\n"
      "@p ld.shared.u16 %0, [a + -65536];\n}"
      : "+r"(e)
      : "r"(a_info)
      : "memory");
  return e;
}
__device__ __forceinline__ void red_or(uint32_t a, uint32_t v) {
  asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add(uint32_t a, uint32_t v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t atom_add(uint32_t a, uint32_t v) {
  uint32_t o;
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
  return o;
}
// 16-byte global -> shared copy that holds no registers (cp.async, L2 only).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Popcount of four words with three popc instructions: a carry-save adder
// turns three of them into a sum and a carry word (popc runs at a quarter of
// the rate of logic instructions).
__device__ __forceinline__ uint32_t popc_u4(uint4 a, uint4 b) {
  const uint32_t x = a.x ^ b.x, y = a.y ^ b.y, z = a.z ^ b.z, w = a.w ^ b.w;
  const uint32_t sum = x ^ y ^ z, carry = (x & y) | (x & z) | (y & z);
  return uint32_t(__popc(sum) + __popc(w) + 2 * __popc(carry));
}

__device__ __forceinline__ int dot_u4(uint4 a, uint4 b, int acc) {
  acc = __dp4a(int(a.x), int(b.x), acc);
  acc = __dp4a(int(a.y), int(b.y), acc);
  acc = __dp4a(int(a.z), int(b.z), acc);
  return __dp4a(int(a.w), int(b.w), acc);
}

// What stage F does with a candidate's dot: above the starting threshold it is
// a survivor, else (with a candidate cache) flagged as rejected.
struct DotSink {
  uint32_t a_row, a_need, a_ids, a_info, a_thr, a_key, a_sid;
  bool flag_rejected;
  __device__ __forceinline__ void take(int q, int dot) const {
    const uint32_t j = lds16(a_need + 2 * q), f = lds16(a_info + 2 * j);
    if (dot > int32_t(lds32(a_thr))) {
      const uint32_t at = atom_add(a_row + kRowProm, 1u);
      sts64(a_key + 8 * at, ((1024u - (f & kXMask)) << 13) | (0x1fffu - j), uint32_t(dot) ^ 0x80000000u);
      sts32(a_sid + 4 * at, lds32(a_ids + 4 * j));
    } else if (flag_rejected) {
      sts16(a_info + 2 * j, f | kRej);
    }
  }
};

// Stage F for rows of 257 to 512 * HALVES codes: a warp per four candidates, a
// lane the 16-byte chunks lane and lane + 32 of each, so the row's own chunks
// stay in registers.  (With 8 lanes per candidate they were read from shared
// memory for every candidate, four wavefronts per load like the gather itself.)
// The four sums are reduced together: each exchange keeps half of them.
template <int HALVES>
__device__ __forceinline__ void dots_wide(const int8_t* __restrict__ codes, int d, uint32_t self, uint32_t a_code, int tid,
                                          const DotSink& sink) {
  const unsigned full = 0xffffffffu;
  const int lane = tid & 31;
  const int nneed = int(lds32(sink.a_row + kRowNeed));
  int b = 4 * (tid >> 5);
  if (b >= nneed) return;  // warp-uniform
  const uint4 zero = make_uint4(0, 0, 0, 0);
  bool live[HALVES];
  uint4 mine[HALVES];
#pragma unroll
  for (int h = 0; h < HALVES; ++h) {
    live[h] = 512 * h + 16 * lane < d;
    mine[h] = live[h] ? lds128(a_code + 512 * h + 16 * lane) : zero;
  }
  const int8_t* lane_codes = codes + 16 * lane;
#pragma unroll 1
  for (; b < nneed; b += 4 * kWarps) {
    const uint2 list = lds64(sink.a_need + 2 * b);  // four entries; the row itself past the list's end
    uint4 x[4][HALVES];
    int acc[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t j = ((c < 2 ? list.x : list.y) >> (16 * (c & 1))) & 0xffffu;
      const uint32_t id = b + c < nneed ? lds32(sink.a_ids + 4 * j) : self;
      const int8_t* row = lane_codes + uint64_t(id) * uint32_t(d);
#pragma unroll
      for (int h = 0; h < HALVES; ++h) {
        x[c][h] = zero;
        if (live[h]) x[c][h] = __ldg(reinterpret_cast<const uint4*>(row + 512 * h));
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[c] = 0;
#pragma unroll
      for (int h = 0; h < HALVES; ++h) acc[c] = dot_u4(x[c][h], mine[h], acc[c]);
    }
    const bool hi = lane & 16, mid = lane & 8;
    int k0 = hi ? acc[2] : acc[0], k1 = hi ? acc[3] : acc[1];
    k0 += __shfl_xor_sync(full, hi ? acc[0] : acc[2], 16);
    k1 += __shfl_xor_sync(full, hi ? acc[1] : acc[3], 16);
    int k = mid ? k1 : k0;
    k += __shfl_xor_sync(full, mid ? k0 : k1, 8);
    k += __shfl_xor_sync(full, k, 4);
    k += __shfl_xor_sync(full, k, 2);
    k += __shfl_xor_sync(full, k, 1);
    const int q = b + (lane >> 3);  // lanes 8c..8c + 7 hold candidate c's sum
    if ((lane & 7) == 0 && q < nneed) sink.take(q, k);
  }
}

// Stage F for short rows: 8 lanes per candidate, 128 * CHUNKS codes.
template <int CHUNKS>
__device__ __forceinline__ void dots_narrow(const int8_t* __restrict__ codes, uint32_t a_code, int tid, const DotSink& sink) {
  const unsigned full = 0xffffffffu;
  const int sub = tid & 7, slot8 = (tid & 31) >> 3;
  const int nneed = int(lds32(sink.a_row + kRowNeed));
#pragma unroll 1
  for (int q = tid >> 3; q - slot8 < nneed; q += kGroups) {
    int acc = 0;
    if (q < nneed) {
      const uint32_t id = lds32(sink.a_ids + 4 * lds16(sink.a_need + 2 * q));
      const int8_t* row = codes + uint64_t(id) * uint32_t(128 * CHUNKS) + 16 * sub;
      uint4 x[CHUNKS];
#pragma unroll
      for (int u = 0; u < CHUNKS; ++u) x[u] = __ldg(reinterpret_cast<const uint4*>(row + 128 * u));
#pragma unroll
      for (int u = 0; u < CHUNKS; ++u) acc = dot_u4(x[u], lds128(a_code + 16 * sub + 128 * u), acc);
    }
    acc += __shfl_xor_sync(full, acc, 1);
    acc += __shfl_xor_sync(full, acc, 2);
    acc += __shfl_xor_sync(full, acc, 4);
    if (sub == 0 && q < nneed) sink.take(q, acc);
  }
}

// Byte offset of id's slot in a table of 2^(32 - shift) words, round 0 or
// later: a multiplicative hash whose odd multiplier changes with the round,
// so ids that met in one round part in the next.
__device__ __forceinline__ uint32_t slot_of(uint32_t id, uint32_t round, int shift) {
  return ((id * (2654435761u + round * 0x3C6EF372u)) >> shift) << 2;
}

__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// CB: sketches in flight per 8-lane group (Hamming stage); MINB: resident CTAs
// per SM the register budget allows; DEF: the default K and R (and 8-byte
// aligned input lists), else any.
template <int CB, int MINB, bool DEF, bool FAR>
__global__ void __launch_bounds__(kThreads, MINB) join_kernel(
    const int8_t* __restrict__ codes, const uint64_t* __restrict__ sketch, int64_t n64, int d, int K_, int R_, int W,
    const int32_t* ids_in, const int32_t* scores_in, int32_t* ids_out, int32_t* scores_out,
    const int32_t* __restrict__ row_order, unsigned long long* __restrict__ counters, JobTable jt, JoinCtl ctl,
    const JoinLayout LA) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (ctl.all_done && *reinterpret_cast<volatile int*>(ctl.all_done)) return;
  if (ctl.iter) {
    const int it = *ctl.iter;
    if (it >= ctl.max_iter) return;
    counters += 8 * it;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl.times[2 * it] = global_ns();
  }
  static_assert(DEF || !FAR, "FAR is a form of the default kernel");
  constexpr JoinLayout LD = join_layout(kDefK, kDefR, kMaxDim, true, FAR);
#define KNNG_L(f) (DEF ? LD.f : LA.f)
  constexpr int NP = DEF ? (LD.pairs + kThreads - 1) / kThreads : kMaxPairs;  // pairs per thread
  const int K = DEF ? kDefK : K_, R = DEF ? kDefR : R_;
  uint32_t sb, tid_;
  asm volatile("{\n.reg .u64 t;\ncvta.to.shared.u64 t, %1;\ncvt.u32.u64 %0, t;\n}" : "=r"(sb) : "l"(smem));
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid_));
  const int tid = int(tid_);
  const unsigned full = 0xffffffffu;
  const int lane = tid & 31, warp = tid >> 5, sub = lane & 7, slot8 = lane >> 3;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t n = uint32_t(n64);  // num_trees * n fits in int32
  const int sk_chunks = W / 2;       // W: sketch words per row
  const bool inplace = ids_out == ids_in;
  const bool cached = ctl.cache_ids != nullptr;
  const uint32_t a_ids = sb + KNNG_L(o_ids), a_rep = sb + KNNG_L(o_rep), a_info = sb + KNNG_L(o_info);
  const uint32_t a_ta = sb + KNNG_L(o_ta), a_tb = sb + KNNG_L(o_tb), a_hist = sb + KNNG_L(o_hist);
  const uint32_t a_x = sb + KNNG_L(o_x), a_cell = sb + KNNG_L(o_cell), a_code = sb + KNNG_L(o_code);
  const uint32_t a_member = sb + KNNG_L(o_member);
  // survivors: 64-bit keys {dot, visit key}, then ids, then (sequential
  // insertion) their visit order; with FAR over the first table, which stage F
  // no longer reads
  const uint32_t a_key = FAR ? a_ta : a_rep;
  const uint32_t a_sid = a_key + 8u * KNNG_L(survivors), a_sorder = a_key + 12u * KNNG_L(survivors);
  // per-CTA statistics, kept by thread 0 in shared memory (no registers held
  // across the row loop): updates, sketches scored, rows reranked, distinct
  // candidates, rows skipped
  __shared__ unsigned long long s_stat[5];
  __shared__ unsigned long long s_run_upd;  // updates of job s_run_job not yet added to its count
  __shared__ int s_run_job;
  __shared__ int s_pend_i, s_pend_job;      // the computed row whose bookkeeping is still open, and its job
  __shared__ int s_job[2];                  // job of the row in each list buffer (thread 0)
  if (tid == 0) {
    for (int q = 0; q < 5; ++q) s_stat[q] = 0;
    s_run_upd = 0;
    s_run_job = -1;
    s_pend_i = -1;
    s_job[0] = s_job[1] = 0;
  }
  if (tid < 16) sts32(sb + KNNG_L(o_row) + 4 * tid, 0);
  if (tid == 0) sts16(a_info + 2 * KNNG_L(dummy), kNoDist);
  auto clear_tables = [&]() {
    const uint4 e = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (int t = tid; t < KNNG_L(ta_slots) / 4; t += kThreads) sts128(a_ta + 16 * t, e);
    for (int t = tid; t < kTableB / 4; t += kThreads) sts128(a_tb + 16 * t, e);
  };
  clear_tables();
  sts16(a_member + 2 * tid, 0);
  // (bounds-checked build) few tags, so that a few rows wear them out
  const uint32_t tag_top = kChecked ? uint32_t(KNNG_L(KK)) + 64u : kTagTop;
  uint32_t tag = tag_top;           // block-uniform
  uint32_t par = 0;                 // parity of the computed rows

  // Bookkeeping of the last computed row, by thread 0 once a barrier has
  // passed since its last stage; frees its counters for the row after next.
  auto finish_row = [&]() {
    if (tid != 0 || s_pend_i < 0) return;
    const uint32_t c = sb + KNNG_L(o_row) + 32u * (par ^ 1u);
    const uint4 u = lds128(c);
    const uint2 w = lds64(c + kRowProm);
    sts128(c, make_uint4(0, 0, 0, 0));
    sts64(c + kRowProm, 0, 0);
    s_stat[0] += w.y;
    s_stat[1] += u.z;
    s_stat[2] += u.w;
    s_stat[3] += u.y;
    if (ctl.chg_out) ctl.chg_out[s_pend_i] = w.y ? 1 : 0;
    if (ctl.job_upd) {
      if (s_pend_job != s_run_job) {
        if (s_run_job >= 0 && s_run_upd) atomicAdd(ctl.job_upd + s_run_job, s_run_upd);
        s_run_job = s_pend_job;
        s_run_upd = 0;
      }
      s_run_upd += w.y;
    }
    s_pend_i = -1;
  };

  // A row's index is loaded two rows ahead; its own list (cp.async into the
  // other list buffer), cache count, change flags and its job's state while
  // the row before is computed.  The flags are combined at the row's start, so
  // nothing waits for them before.
  const int nrows = int((ctl.row_limit > 0 && ctl.row_limit < n64) ? ctl.row_limit : n64);
  auto row_at = [&](int r) { return r < nrows && r >= 0 ? (row_order ? row_order[r] : r) : -1; };
  int32_t nx_i = row_at(blockIdx.x), nx2_i = row_at(int(blockIdx.x) + int(gridDim.x));
  uint32_t slot = 0;                    // list buffer of the current row
  int nx_cc = 0, nx_flag = 0, nx_done = 0;
  auto fetch_list = [&](uint32_t to) {  // list and cache count of row nx_i
    if (nx_i >= 0 && KNNG_GUARD(ctl.check_err, nx_i < int(n))) {
      if (tid < K) {
        const uint32_t dst = sb + KNNG_L(o_pool) + to * (8u * KNNG_L(kp)) + 4u * uint32_t(tid);
        cp_async4(dst, ids_in + int64_t(nx_i) * K + tid);
        cp_async4(dst + 4u * KNNG_L(kp), scores_in + int64_t(nx_i) * K + tid);
      }
      if (cached) nx_cc = ctl.cache_cnt[nx_i];
    }
    cp_async_commit();
  };
  // (unchanged-row skip, double-buffered iterations only) a row whose own
  // list and every neighbour's list came out of the previous iteration
  // unchanged sees exactly the inputs it saw then, so its result is its
  // current list: it is copied through without any work, as are the rows of a
  // stopped job
  auto fetch_flags = [&](uint32_t to) {
    cp_async_wait_all();
    nx_flag = nx_done = 0;
    if (tid <= K && nx_i >= 0 && (!kChecked || nx_i < int(n))) {
      nx_flag = 1;
      if (ctl.chg_in) {
        const uint32_t at = tid < K ? lds32(sb + KNNG_L(o_pool) + to * (8u * KNNG_L(kp)) + 4u * uint32_t(tid)) : uint32_t(nx_i);
        if (at < n) nx_flag = int(ctl.chg_in[at]);
      }
      if (ctl.job_done) {
        const int job = job_of(jt, nx_i);
        nx_done = ctl.job_done[job];
        if (tid == 0) s_job[to] = job;
      }
    }
  };
  fetch_list(0);
  fetch_flags(0);
  for (int r0 = int(blockIdx.x); r0 < nrows && r0 >= 0; r0 += int(gridDim.x), slot ^= 1u) {
    const int i = nx_i;
    const int cc = cached ? min(nx_cc, ctl.cache_cap) : 0;
    const int moved = nx_done ? 0 : nx_flag;
    const int stopped = nx_done;  // threads 0..K
    nx_i = nx2_i;
    nx2_i = row_at(r0 + 2 * int(gridDim.x));
    if (i < 0 || !KNNG_GUARD(ctl.check_err, i < int(n))) {  // block-uniform
      KNNG_FLAG_IF(ctl.check_err, i < 0);
      __syncthreads();  // the other list buffer may still be read
      fetch_list(slot ^ 1u);
      fetch_flags(slot ^ 1u);
      continue;
    }
    // ---- A
    const uint32_t a_pool = sb + KNNG_L(o_pool) + slot * (8u * KNNG_L(kp));  // ids, then scores
    const uint32_t a_psc = a_pool + 4u * KNNG_L(kp);
    const uint32_t a_row = sb + KNNG_L(o_row) + 32u * par;
    const bool work = __syncthreads_or(moved) != 0;  // block-uniform
    finish_row();
    if (!work) {
      if (!inplace && tid < K) {
        ids_out[int64_t(i) * K + tid] = int32_t(lds32(a_pool + 4 * tid));
        scores_out[int64_t(i) * K + tid] = int32_t(lds32(a_psc + 4 * tid));
      }
      if (tid == 0 && !stopped) {
        ctl.chg_out[i] = 0;
        ++s_stat[4];
      }
      fetch_list(slot ^ 1u);
      fetch_flags(slot ^ 1u);
      continue;
    }
    // own code row and sketch, and the row's cache entries (ids over the miss
    // list, distances over the histogram); the rows' cache slices are 16-byte
    // aligned and sized for cache_cap
    {
      const int nchunk = d / 16;
      const int n_id = (cc * 4 + 15) / 16, n_hr = (cc * 2 + 15) / 16;
      const char* gid = reinterpret_cast<const char*>(ctl.cache_ids + int64_t(i) * ctl.cache_cap);
      const char* ghr = reinterpret_cast<const char*>(ctl.cache_hr + int64_t(i) * ctl.cache_cap);
      for (int t = tid; t < n_id; t += kThreads) cp_async16(a_x + 16 * t, gid + 16 * t);
      for (int t = tid; t < n_hr; t += kThreads) cp_async16(a_hist + 16 * t, ghr + 16 * t);
      if (tid < nchunk) cp_async16(a_code + 16 * tid, codes + int64_t(i) * d + 16 * tid);
      else if (tid - nchunk < sk_chunks)
        cp_async16(sb + KNNG_L(o_sk) + 16 * (tid - nchunk),
                   reinterpret_cast<const char*>(sketch + int64_t(i) * W) + 16 * (tid - nchunk));
      cp_async_commit();
    }
    if (tag < uint32_t(KNNG_L(KK)) + 16u) {  // a row uses at most KK + 1 tags; block-uniform, once per ~300,000 rows
      clear_tables();
      tag = tag_top;
      __syncthreads();
    }
    // ---- B  two-hop occurrences, pair p = tid + 256r holding j = 2p, 2p + 1;
    //         all loaded first
    uint32_t v[2 * NP];
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      const int p = tid + kThreads * r;
      v[2 * r] = v[2 * r + 1] = ~0u;
      if (DEF) {  // a pair lies in one list and is 8-byte aligned
        if (p < LD.pairs) {
          const int k = p / (kDefK / 2);
          const uint32_t n1 = lds32(a_pool + 4 * k);
          if (n1 < n) {
            const int2 g = *reinterpret_cast<const int2*>(ids_in + int64_t(n1) * kDefK + 2 * (p - k * (kDefK / 2)));
            v[2 * r] = uint32_t(g.x);
            v[2 * r + 1] = uint32_t(g.y);
            KNNG_FLAG_IF(ctl.check_err, v[2 * r] >= n || v[2 * r + 1] >= n);
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int j = 2 * p + e;
          if (j < LA.KK) {
            const int k = int((uint32_t(j) * LA.kdiv) >> 20);
            const uint32_t n1 = lds32(a_pool + 4 * k);
            if (n1 < n) {
              v[2 * r + e] = uint32_t(ids_in[int64_t(n1) * K + (j - k * K)]);
              KNNG_FLAG_IF(ctl.check_err, v[2 * r + e] >= n);
            }
          }
        }
      }
    }
    for (int t = tid; t < (KNNG_L(pairs) * 4 + 15) / 16; t += kThreads) sts128(a_info + 16 * t, make_uint4(0, 0, 0, 0));
    // unscored entries (INT32_MIN, tiny inputs only) can share their id with a
    // survivor, and an unsorted pool (possible through the stage entry point)
    // breaks the rank formulas of stage G: both take the sequential loop
    int irregular = 0;
    uint32_t find_id = ~0u;  // this thread's starting-list id, while it is still looked up
    if (tid < K) {
      const uint32_t my_id = lds32(a_pool + 4 * tid);
      const int32_t my_sc = int32_t(lds32(a_psc + 4 * tid));
      KNNG_FLAG_IF(ctl.check_err, my_id >= n);
      irregular = (my_sc == kScoreMinI) | (tid + 1 < K && my_sc < int32_t(lds32(a_psc + 4 * tid + 4)));
      if (my_sc != kScoreMinI && my_id < n) find_id = my_id;
    }
    // a valid id goes into the first table; without a candidate the register
    // holds kNone, which no id in shared memory equals
    unsigned valid = 0;  // bit 2r + e
    uint32_t sl[2 * NP];
#pragma unroll
    for (int x = 0; x < 2 * NP; ++x) sl[x] = a_ta + slot_of(v[x], 0u, KNNG_L(ta_shift));
    const uint32_t tagj = (tag << kJBits) + 2u * uint32_t(tid);
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      const int p = tid + kThreads * r;
#pragma unroll
      for (int e = 0; e < 2; ++e)
        table_insert(v[2 * r + e], n, uint32_t(i), sl[2 * r + e],
                     tagj + uint32_t(2 * kThreads * r + e), valid, 1u << (2 * r + e));
      if (p < KNNG_L(pairs)) sts64(a_ids + 8 * p, v[2 * r], v[2 * r + 1]);
    }
    {
      const int c = __reduce_add_sync(full, __popc(valid));
      if (lane == 0) red_add(a_row + kRowCnt, uint32_t(c));
    }
    cp_async_wait_all();  // this thread's copies of stage A; the barrier publishes them
    const bool serial_insert = __syncthreads_or(irregular) != 0;
    unsigned fm = 0;     // bit 2r + e: the occurrence is the first of its id
    int find_rep = -1;   // representative of the starting-list id, if it occurs
    unsigned ctodo = 0;  // bit 2u + e: the cached id is not resolved
    unsigned todo = 0;   // bit 2r + e: the occurrence is not resolved
    // round 0: every occurrence, every cached id, the starting list
    {
      uint32_t w[2 * NP];
#pragma unroll
      for (int x = 0; x < 2 * NP; ++x) {
        w[x] = lds32(sl[x]) & kJMask;
      }
#pragma unroll
      for (int r = 0; r < NP; ++r) {
        const int p = tid + kThreads * r;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t id = v[2 * r + e];
          table_settle<FAR>(id, lds32(a_ids + 4 * w[2 * r + e]), w[2 * r + e], KNNG_L(dummy), uint32_t(2 * p + e), a_info,
                            a_tb + slot_of(id, 1u, kTableBShift), tagj - (1u << kJBits) + uint32_t(2 * kThreads * r + e), todo,
                            fm, 1u << (2 * r + e));
        }
        if (!FAR && p < KNNG_L(pairs)) sts32(a_rep + 4 * p, w[2 * r] | (w[2 * r + 1] << 16));
      }
    }
#pragma unroll 1
    for (int u = 0; u < kCachePairs; ++u) {
      if (2 * kThreads * u >= cc) break;  // block-uniform
      const int q = tid + kThreads * u;
      const uint2 id = lds64(a_x + 8 * q);
      const uint32_t hr = lds32(a_hist + 4 * q);
      const uint32_t e0 = lds32(a_ta + slot_of(id.x, 0u, KNNG_L(ta_shift)));
      const uint32_t e1 = lds32(a_ta + slot_of(id.y, 0u, KNNG_L(ta_shift)));
      table_find(id.x, 2 * q < cc, e0, tag << kJBits, a_ids, a_info, hr | kKnown, ctodo, 1u << (2 * u));
      table_find(id.y, 2 * q + 1 < cc, e1, tag << kJBits, a_ids, a_info, (hr >> 16) | kKnown, ctodo, 2u << (2 * u));
    }
    if (find_id != ~0u) {
      const uint32_t e = lds32(a_ta + slot_of(find_id, 0u, KNNG_L(ta_shift)));
      if ((e >> kJBits) != tag) {
        find_id = ~0u;
      } else if (lds32(a_ids + 4 * (e & kJMask)) == find_id) {
        find_rep = int(e & kJMask);
        find_id = ~0u;
      }
    }
    uint32_t round = 1;
#pragma unroll 1
    while (__syncthreads_or(int(todo))) {
      const bool odd = round & 1u;
      const uint32_t t_cur = odd ? a_tb : a_ta, t_nxt = odd ? a_ta : a_tb;
      const int sh_cur = odd ? kTableBShift : KNNG_L(ta_shift), sh_nxt = odd ? KNNG_L(ta_shift) : kTableBShift;
      const uint32_t tc = tag - round;
#pragma unroll 1
      for (unsigned m = todo; m; m &= m - 1u) {
        const int b = __ffs(m) - 1;
        const uint32_t j = 2u * uint32_t(tid + kThreads * (b >> 1)) + uint32_t(b & 1);
        const uint32_t id = lds32(a_ids + 4 * j);
        const uint32_t w = lds32(t_cur + slot_of(id, round, sh_cur)) & kJMask;
        if (lds32(a_ids + 4 * w) == id) {
          if (!FAR) sts16(a_rep + 2 * j, w);
          todo ^= 1u << b;
          if (w == j) fm |= 1u << b;
          else if (FAR) sts16(a_info + 2 * j, w | kPtr);
        } else {
          red_min(t_nxt + slot_of(id, round + 1u, sh_nxt), ((tc - 1u) << kJBits) + j);
        }
      }
#pragma unroll 1
      for (unsigned m = ctodo; m; m &= m - 1u) {
        const int b = __ffs(m) - 1;
        const uint32_t q = 2u * uint32_t(tid + kThreads * (b >> 1)) + uint32_t(b & 1);
        const uint32_t id = lds32(a_x + 4 * q);
        const uint32_t e = lds32(t_cur + slot_of(id, round, sh_cur));
        if ((e >> kJBits) != tc) {
          ctodo ^= 1u << b;
        } else if (lds32(a_ids + 4 * (e & kJMask)) == id) {
          ctodo ^= 1u << b;
          sts16(a_info + 2 * (e & kJMask), lds16(a_hist + 2 * q) | kKnown);
        }
      }
      if (find_id != ~0u) {
        const uint32_t e = lds32(t_cur + slot_of(find_id, round, sh_cur));
        if ((e >> kJBits) != tc) {
          find_id = ~0u;
        } else if (lds32(a_ids + 4 * (e & kJMask)) == find_id) {
          find_rep = int(e & kJMask);
          find_id = ~0u;
        }
      }
      ++round;
    }
    tag -= round + 1u;
    fetch_list(slot ^ 1u);  // the previous row's list is no longer read
    // ---- C  Hamming once per distinct id without a cached distance: each warp
    //         lists its own first occurrences that are misses and scores them
    //         (groups of 8 lanes, CB candidates in flight per group)
    if (find_rep >= 0) {  // occurrence 2 (t + 256 r) + e: bit 2r + e of thread t's half word
      const uint32_t p = uint32_t(find_rep) >> 1, t = p % kThreads;
      red_or(a_member + 4 * (t >> 1), 1u << (16 * (t & 1u) + 2 * (p / kThreads) + (uint32_t(find_rep) & 1u)));
    }
    for (int t = tid; t < kHBins / 4; t += kThreads) sts128(a_hist + 16 * t, make_uint4(0, 0, 0, 0));
    int first_at;  // this thread's place among the row's distinct ids (stage G)
    {
      unsigned mm = fm;
      if (cc > 0) {  // block-uniform
#pragma unroll
        for (int r = 0; r < NP; ++r) {
          const int p = tid + kThreads * r;
          if (p < KNNG_L(pairs)) {
            const uint32_t f = lds32(a_info + 4 * p);
            if (f & kKnown) mm &= ~(1u << (2 * r));
            if (f & (kKnown << 16)) mm &= ~(2u << (2 * r));
          }
        }
      }
      const int c = __popc(mm), nfirst = __popc(fm);
      const int both = warp_incl_scan(c | (nfirst << 16), lane);  // two sums, at most 32 * 2 NP each
      const int incl = both & 0xffff, fincl = both >> 16;
      const int nm = __shfl_sync(full, incl, 31);
      int wbase = 0;
      if (lane == 31) {
        wbase = int(atom_add(a_row + kRowNu, uint32_t(fincl)));
        red_add(a_row + kRowMiss, uint32_t(incl));
      }
      first_at = __shfl_sync(full, wbase, 31) + fincl - nfirst;
      // up to 64 NP misses per warp
      const uint32_t a_miss = a_x + uint32_t(warp) * (DEF ? uint32_t(NP) * 128u : uint32_t((LA.pairs + kThreads - 1) / kThreads) * 128u);
      uint32_t at = a_miss + 2 * (incl - c);
      const uint32_t j0 = 2u * uint32_t(tid);
#pragma unroll
      for (int b = 0; b < 2 * NP; ++b) list_push(mm, 1u << b, at, j0 + uint32_t(2 * kThreads * (b >> 1) + (b & 1)));
      __syncwarp();
      const char* sk_base = reinterpret_cast<const char*>(sketch);
      const uint32_t sk_bytes = uint32_t(W) * 8u;
      if (sk_chunks == 1) {  // 16-byte sketches: one lane per candidate
        const uint4 mine = lds128(sb + KNNG_L(o_sk));
#pragma unroll 1
        for (int q = lane; q < nm; q += 32) {
          const uint32_t j = lds16(a_miss + 2 * q), id = lds32(a_ids + 4 * j);
          sts16(a_info + 2 * j, popc_u4(__ldg(reinterpret_cast<const uint4*>(sk_base + uint64_t(id) * 16u)), mine));
        }
      } else {
        // 32 candidates per step, 8 lanes each: lane 8g + s reads the 16-byte
        // chunk s of candidates 4u + g (u = 0..7) and ends up with the
        // distance of candidate 4 t(s) + g, where t reverses s's three bits:
        // the group's 8 partial sums are two to a word, and each exchange
        // keeps half of the words (14 instructions for 8 sums, against 48
        // for one butterfly per sum)
        const uint4 mine = sub < sk_chunks ? lds128(sb + KNNG_L(o_sk) + 16 * sub) : make_uint4(0, 0, 0, 0);
        const char* sk_lane = sk_base + 16 * (sub < sk_chunks ? sub : 0);
        const int t = ((sub & 1) << 2) | (sub & 2) | (sub >> 2);
#pragma unroll 1
        for (int b = 0; b < nm; b += 32) {
          const int q = b + 4 * t + slot8;
          uint32_t j = 0, id = uint32_t(i);  // past the list: the row itself
          if (q < nm) {
            j = lds16(a_miss + 2 * q);
            id = lds32(a_ids + 4 * j);
          }
          uint32_t pw[4] = {0, 0, 0, 0};  // word k: candidates u = k (low half) and u = k + 4
#pragma unroll
          for (int u0 = 0; u0 < 8; u0 += CB) {
            if (b + 4 * u0 >= nm) break;  // warp-uniform
            uint4 x[CB];
#pragma unroll
            for (int u = 0; u < CB; ++u) {
              const int uu = u0 + u, src = ((uu & 1) << 2) | (uu & 2) | (uu >> 2);  // the lane whose t is uu
              const uint32_t cid = __shfl_sync(full, id, 8 * slot8 + src);
              x[u] = __ldg(reinterpret_cast<const uint4*>(sk_lane + uint64_t(cid) * sk_bytes));
            }
#pragma unroll
            for (int u = 0; u < CB; ++u) {
              const uint32_t pc = popc_u4(x[u], mine);
              pw[(u0 + u) & 3] += (u0 + u) < 4 ? pc : pc << 16;
            }
          }
          if (sub >= sk_chunks) pw[0] = pw[1] = pw[2] = pw[3] = 0;  // lanes beyond a narrow sketch
          // exchange 1 (lane bit 0 = bit 2 of t): nothing to choose between, both
          // halves of a word stay together; it is left for the last step.
          // Lane bit 1 is bit 1 of t (word pairs 0,1 / 2,3), lane bit 2 bit 0.
          const bool s1 = sub & 2, s2 = sub & 4;
          uint32_t k0 = s1 ? pw[2] : pw[0], k1 = s1 ? pw[3] : pw[1];
          k0 += __shfl_xor_sync(full, s1 ? pw[0] : pw[2], 2);
          k1 += __shfl_xor_sync(full, s1 ? pw[1] : pw[3], 2);
          uint32_t k = s2 ? k1 : k0;
          k += __shfl_xor_sync(full, s2 ? k0 : k1, 4);
          k += __shfl_xor_sync(full, k, 1);
          if (q < nm) sts16(a_info + 2 * j, (sub & 1) ? k >> 16 : k & 0xffffu);
        }
      }
    }
    fetch_flags(slot ^ 1u);
    __syncthreads();
    // ---- D  histogram over occurrences, threshold
    uint32_t hv[NP];  // info of each occurrence's id, two per word
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      const int p = tid + kThreads * r;
      hv[r] = kNoDist | (kNoDist << 16);
      if (p < KNNG_L(pairs)) {
        const uint32_t w = lds32((FAR ? a_info : a_rep) + 4 * p);
        const uint32_t f0 = FAR ? info_of(w & 0xffffu, a_info) : lds16(a_info + 2 * (w & 0xffffu));
        const uint32_t f1 = FAR ? info_of(w >> 16, a_info) : lds16(a_info + 2 * (w >> 16));
        hv[r] = f0 | (f1 << 16);
        red_add(a_hist + 4 * (f0 & kXMask), 1u);
        red_add(a_hist + 4 * (f1 & kXMask), 1u);
      }
    }
    __syncthreads();
    uint32_t xt = kXMask;  // threshold distance; none: every occurrence is nearer
    int need_eq = 0;
    const bool cut = int(lds32(a_row + kRowCnt)) > R;  // block-uniform
    if (cut) {
      // every warp by itself: bins from distance 0 up, 128 per step
      int acc = 0;
#pragma unroll 1
      for (int base = 0; base < kHBins; base += 128) {
        const uint4 b4 = lds128(a_hist + 4 * (base + 4 * lane));
        const int sum = int(b4.x + b4.y + b4.z + b4.w);
        const int tot = __reduce_add_sync(full, sum);
        if (acc + tot >= R) {  // warp-uniform; reached, as the bins hold cnt > R occurrences
          const int incl = warp_incl_scan(sum, lane);
          int run = acc + incl - sum, x = base + 4 * lane;
          const bool here = run < R && R <= run + sum;
          if (run + int(b4.x) < R) {
            run += int(b4.x);
            ++x;
            if (run + int(b4.y) < R) {
              run += int(b4.y);
              ++x;
              if (run + int(b4.z) < R) {
                run += int(b4.z);
                ++x;
              }
            }
          }
          const int src = __ffs(__ballot_sync(full, here)) - 1;
          xt = uint32_t(__shfl_sync(full, x, src));
          need_eq = R - __shfl_sync(full, run, src);
          break;
        }
        acc += tot;
      }
    }
    // ---- E  selected first occurrences that are neither starting-list members
    //         nor known to be rejected need a dot; one at the threshold is
    //         selected iff fewer than need_eq ties come before it in j order
    //         (a cached rejection stands: the row's threshold never falls, so
    //         a dot once <= it stays <= it)
    unsigned wm = 0, eqm = 0, open = 0;  // nearer than the threshold; at it; at it and not rejected
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      // a rejection's bit lies above the distance: such a word is never below xt
      mark_near(hv[r] & (kXMask | kRej), hv[r] & kXMask, xt, wm, eqm, open, 1u << (2 * r));
      mark_near(hv[r] & ((kXMask | kRej) << 16), hv[r] & (kXMask << 16), xt << 16, wm, eqm, open, 2u << (2 * r));
    }
    const unsigned want = fm & ~lds16(a_member + 2 * tid);
    sts16(a_member + 2 * tid, 0);
    wm &= want;
    open &= want;
    if (cut) {
      // ties per (round, warp): j ascends with round, warp, lane, element
      const unsigned any = __reduce_or_sync(full, eqm);
#pragma unroll
      for (int r = 0; r < NP; ++r) {
        int c = 0;
        if ((any >> (2 * r)) & 3u) {  // warp-uniform
          c = __popc(__ballot_sync(full, (eqm >> (2 * r)) & 1u)) + __popc(__ballot_sync(full, (eqm >> (2 * r)) & 2u));
        }
        if (lane == 0) sts32(a_cell + 4 * (r * kWarps + warp), uint32_t(c));
      }
      __syncthreads();
      const unsigned decide = __reduce_or_sync(full, open);
      if (decide) {  // warp-uniform
        uint2 c2 = make_uint2(0, 0);
        if (2 * lane < NP * kWarps) c2 = lds64(a_cell + 8 * lane);
        const int sum = int(c2.x + c2.y);
        const int pre = warp_incl_scan(sum, lane) - sum + ((warp & 1) ? int(c2.x) : 0);
#pragma unroll
        for (int r = 0; r < NP; ++r) {
          if ((decide >> (2 * r)) & 3u) {  // warp-uniform
            const unsigned b0 = __ballot_sync(full, (eqm >> (2 * r)) & 1u), b1 = __ballot_sync(full, (eqm >> (2 * r)) & 2u);
            const int before = __shfl_sync(full, pre, 4 * r + (warp >> 1)) + __popc(b0 & lt) + __popc(b1 & lt);
            const unsigned e0 = (eqm >> (2 * r)) & 1u;
            if (before < need_eq) wm |= open & (1u << (2 * r));
            if (before + int(e0) < need_eq) wm |= open & (2u << (2 * r));
          }
        }
      }
    }
    {
      if (__any_sync(full, wm != 0)) {
        const int c = __popc(wm), incl = warp_incl_scan(c, lane);
        uint32_t base = 0;
        if (lane == 31) base = atom_add(a_row + kRowNeed, uint32_t(incl));
        uint32_t at = a_x + 2 * (__shfl_sync(full, base, 31) + uint32_t(incl - c));
#pragma unroll 1
        for (; wm; wm &= wm - 1u, at += 2) {
          const int b = __ffs(wm) - 1;
          sts16(at, 2u * uint32_t(tid + kThreads * (b >> 1)) + uint32_t(b & 1));
        }
      }
    }
    __syncthreads();
    // ---- F  dots
    {
      const DotSink sink{a_row, a_x, a_ids, a_info, a_psc + 4 * (K - 1), a_key, a_sid, cached};
      if (d > 512) dots_wide<2>(codes, d, uint32_t(i), a_code, tid, sink);  // uniform
      else if (d > 256) dots_wide<1>(codes, d, uint32_t(i), a_code, tid, sink);
      else if (d > 128) dots_narrow<2>(codes, a_code, tid, sink);
      else dots_narrow<1>(codes, a_code, tid, sink);
    }
    __syncthreads();
    // ---- G  the row's cache for the next iteration: this iteration's distinct
    //         candidates (the first cache_cap of them) with distance and flag,
    //         gathered in shared memory (over the rerank list and the
    //         histogram) and written out 16 bytes at a time below
    if (cached) {
      uint32_t at_id = a_x + 4u * uint32_t(first_at), at_info = a_hist + 2u * uint32_t(first_at);
      const uint32_t end = a_x + 4u * uint32_t(ctl.cache_cap);
#pragma unroll
      for (int r = 0; r < NP; ++r) {
        const int p = tid + kThreads * r;
        if (p < KNNG_L(pairs)) {
          const uint2 id = lds64(a_ids + 8 * p);
          const uint32_t f = lds32(a_info + 4 * p) & ~(kKnown | (kKnown << 16));
          cache_push(fm, 1u << (2 * r), at_id, at_info, end, id.x, f);
          cache_push(fm, 2u << (2 * r), at_id, at_info, end, id.y, f >> 16);
        }
      }
    }
    //         insertion of the survivors in visit order.  The pool's last score
    //         only rises during the visits, and a rejected survivor's dot is <=
    //         the last score at its visit, so survivor t is rejected iff at
    //         least K of {starting scores} and {dots of the survivors visited
    //         before t} are >= its dot: iff K entries come before it in the
    //         order (score desc, starting entries in pool order first, then
    //         earlier visits).  The final pool, which the shift-insert loop
    //         leaves in that order, is therefore the first K of the starting
    //         entries and all survivors.  Needs a sorted starting pool without
    //         unscored entries (else serial_insert is set).
    const int P = int(lds32(a_row + kRowProm));
    int32_t* out_id = ids_out + int64_t(i) * K;
    int32_t* out_sc = scores_out + int64_t(i) * K;
    if (P == 0) {  // block-uniform: the list stays
      if (!inplace && tid < K) {
        out_id[tid] = int32_t(lds32(a_pool + 4 * tid));
        out_sc[tid] = int32_t(lds32(a_psc + 4 * tid));
      }
    } else if (!serial_insert) {
      int changed = 0;
      // one unit per thread: starting entries 0..K-1, then survivors
#pragma unroll 1
      for (int u = tid; u < K + P; u += kThreads) {
        uint64_t me;
        uint32_t id;
        int rank;
        if (u < K) {
          // survivors with a larger dot come first: their keys are above (score, all ones)
          me = (uint64_t(lds32(a_psc + 4 * u) ^ 0x80000000u) << 32) | 0xffffffffu;
          id = lds32(a_pool + 4 * u);
          rank = u;
        } else {
          const uint2 k2 = lds64(a_key + 8 * (u - K));
          me = (uint64_t(k2.y) << 32) | k2.x;
          id = lds32(a_sid + 4 * (u - K));
          const int32_t dot = int32_t(k2.y ^ 0x80000000u);
          int lo = 0, hi = K;  // first pool position with a score < dot (scores descend)
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (int32_t(lds32(a_psc + 4 * mid)) >= dot) lo = mid + 1;
            else hi = mid;
          }
          rank = lo;
        }
        int q = 0;
#pragma unroll 2
        for (; q + 1 < P; q += 2) {
          const uint4 o = lds128(a_key + 8 * q);
          rank += ((uint64_t(o.y) << 32) | o.x) > me ? 1 : 0;
          rank += ((uint64_t(o.w) << 32) | o.z) > me ? 1 : 0;
        }
        if (q < P) {
          const uint2 o = lds64(a_key + 8 * q);
          rank += ((uint64_t(o.y) << 32) | o.x) > me ? 1 : 0;
        }
        if (rank < K) {
          const bool ch = id != lds32(a_pool + 4 * rank);
          changed += ch ? 1 : 0;
          if (ch || !inplace) {
            out_id[rank] = int32_t(id);
            out_sc[rank] = int32_t(uint32_t(me >> 32) ^ 0x80000000u);
          }
        }
      }
      changed = __reduce_add_sync(full, changed);
      if (lane == 0 && changed) red_add(a_row + kRowChanged, uint32_t(changed));
    } else {
      // rank sort by (h desc, first j asc), then the reference's shift-insert
      // loop in warp 0 with the pool held two entries per lane
#pragma unroll 1
      for (int p = tid; p < P; p += kThreads) {
        const uint32_t kp = lds32(a_key + 8 * p);
        int rank = 0;
        for (int q = 0; q < P; ++q) rank += lds32(a_key + 8 * q) > kp ? 1 : 0;
        sts16(a_sorder + 2 * rank, uint32_t(p));
      }
      __syncthreads();
      if (warp == 0) {
        const int32_t pidA = lane < K ? int32_t(lds32(a_pool + 4 * lane)) : -1;
        const int32_t pidB = 32 + lane < K ? int32_t(lds32(a_pool + 4 * (32 + lane))) : -1;
        int32_t idA = pidA, scA = lane < K ? int32_t(lds32(a_psc + 4 * lane)) : kScoreMinI;
        int32_t idB = pidB, scB = 32 + lane < K ? int32_t(lds32(a_psc + 4 * (32 + lane))) : kScoreMinI;
#pragma unroll 1
        for (int rr = 0; rr < P; ++rr) {
          const uint32_t p = lds16(a_sorder + 2 * rr);
          const int32_t id = int32_t(lds32(a_sid + 4 * p)), dot = int32_t(lds32(a_key + 8 * p + 4) ^ 0x80000000u);
          if (__any_sync(full, idA == id || idB == id)) continue;
          const int32_t last = (K - 1) < 32 ? __shfl_sync(full, scA, K - 1) : __shfl_sync(full, scB, K - 33);
          if (!(dot > last)) continue;
          const int pos = __popc(__ballot_sync(full, lane < K - 1 && scA >= dot)) +
                          __popc(__ballot_sync(full, 32 + lane < K - 1 && scB >= dot));
          const int32_t upIdA = __shfl_up_sync(full, idA, 1), upScA = __shfl_up_sync(full, scA, 1);
          const int32_t upIdB = __shfl_up_sync(full, idB, 1), upScB = __shfl_up_sync(full, scB, 1);
          const int32_t id31 = __shfl_sync(full, idA, 31), sc31 = __shfl_sync(full, scA, 31);
          if (lane < K) {
            if (lane > pos) { idA = upIdA; scA = upScA; }
            else if (lane == pos) { idA = id; scA = dot; }
          }
          const int qb = 32 + lane;
          if (qb < K) {
            if (qb > pos) {
              idB = lane == 0 ? id31 : upIdB;
              scB = lane == 0 ? sc31 : upScB;
            } else if (qb == pos) {
              idB = id;
              scB = dot;
            }
          }
        }
        const bool chA = lane < K && idA != pidA, chB = 32 + lane < K && idB != pidB;
        if (lane < K && (chA || !inplace)) {
          out_id[lane] = idA;
          out_sc[lane] = scA;
        }
        if (32 + lane < K && (chB || !inplace)) {
          out_id[32 + lane] = idB;
          out_sc[32 + lane] = scB;
        }
        const int changed = __popc(__ballot_sync(full, chA)) + __popc(__ballot_sync(full, chB));
        if (lane == 0) sts32(a_row + kRowChanged, uint32_t(changed));
      }
    }
    if (cached || (FAR && P > 0)) __syncthreads();  // block-uniform
    if (FAR) {  // the slots that held survivors are empty again before the next row's first barrier
#pragma unroll 1
      for (int p = tid; p < P; p += kThreads) {
        sts64(a_key + 8 * p, ~0u, ~0u);
        sts32(a_sid + 4 * p, ~0u);
        if (serial_insert) sts16(a_sorder + 2 * p, 0xffffu);
      }
    }
    if (cached) {
      const int nc = min(int(lds32(a_row + kRowNu)), ctl.cache_cap);
      uint4* cid = reinterpret_cast<uint4*>(ctl.cache_ids + int64_t(i) * ctl.cache_cap);
      uint4* chr = reinterpret_cast<uint4*>(ctl.cache_hr + int64_t(i) * ctl.cache_cap);
      const int n_id = (nc * 4 + 15) / 16, n_hr = (nc * 2 + 15) / 16;  // the last words' ends are never read
      for (int t = tid; t < n_id; t += kThreads) cid[t] = lds128(a_x + 16 * t);
      for (int t = tid; t < n_hr; t += kThreads) chr[t] = lds128(a_hist + 16 * t);
      if (tid == 0) ctl.cache_cnt[i] = nc;
    }
    if (tid == 0) {
      s_pend_i = i;
      s_pend_job = s_job[slot];
    }
    par ^= 1u;
  }
  __syncthreads();
  finish_row();
  if (tid == 0) {
    atomicAdd(counters + 0, s_stat[0]);
    atomicAdd(counters + 1, s_stat[1]);
    atomicAdd(counters + 2, s_stat[2]);
    atomicAdd(counters + 3, s_stat[3]);
    if (ctl.chg_in) atomicAdd(counters + 4, s_stat[4]);
    if (ctl.job_upd && s_run_job >= 0 && s_run_upd) atomicAdd(ctl.job_upd + s_run_job, s_run_upd);
  }
#undef KNNG_L
}

// Per-job early stop after an iteration, src/main.cpp:432-439 in float
// arithmetic: rate = float(updates) / float(n * K); a job stops when
// rate < stop or (iter > 0 and prev - rate < diff).  When every job has
// stopped, all_done is set and final_buf records the buffer that holds the
// final graphs; later iterations of the launch sequence then do nothing.
__global__ void stop_check_kernel(JobTable jt, JoinCtl ctl, int K, int out_buf, float stop_rate, float diff_tol,
                                  cudaGraphConditionalHandle loop, int has_loop) {
  const int iter = *ctl.iter;
  int all = 1;
  const bool ran = !*ctl.all_done && iter < ctl.max_iter;  // block-uniform: written below, behind a barrier
  if (ran) {
    if (threadIdx.x == 0) ctl.times[2 * iter + 1] = global_ns();
    for (int b = threadIdx.x; b < jt.count; b += blockDim.x) {
      if (!ctl.job_done[b]) {
        const unsigned long long upd = ctl.job_upd[b];
        ctl.upd_log[int64_t(iter) * jt.count + b] = (long long)upd;
        const float rate = float(upd) / float((unsigned long long)jt.n[b] * (unsigned long long)K);
        const bool stop = rate < stop_rate || (iter > 0 && (ctl.job_prev[b] - rate) < diff_tol);
        ctl.job_prev[b] = rate;
        ctl.job_iters[b] = iter + 1;
        ctl.job_upd[b] = 0;
        if (stop) ctl.job_done[b] = 1;
        else all = 0;
      }
    }
  }
  all = __syncthreads_and(all);
  if (threadIdx.x == 0) {
    if (ran) {
      *ctl.iter = iter + 1;
      *ctl.final_buf = out_buf;
      if (all) *ctl.all_done = 1;
    }
    if (has_loop) cudaGraphSetConditional(loop, !all && iter + 1 < ctl.max_iter ? 1u : 0u);
  }
}

}  // namespace

// Resident CTAs per SM of a join variant at `smem` bytes of dynamic shared
// memory.  The attribute is set and the occupancy queried once per process and
// variant (under a mutex, so concurrent contexts and stream captures never
// issue these calls); a failure is returned as a CUDA error, not masked.
std::mutex g_variant_mu;
std::map<std::pair<const void*, uint32_t>, int> g_variant_ctas;
char g_variant_err[256] = "";

using JoinKernel = void (*)(const int8_t*, const uint64_t*, int64_t, int, int, int, int, const int32_t*, const int32_t*,
                            int32_t*, int32_t*, const int32_t*, unsigned long long*, JobTable, JoinCtl, JoinLayout);

// ctas_per_sm 3: up to 80 registers per thread, 3 resident CTAs; otherwise 64
// registers, 4 resident CTAs.
template <bool DEF>
JoinKernel pick_variant(int ctas_per_sm, int cblock) {
  if (ctas_per_sm == 3)
    return cblock == 2 ? join_kernel<2, 3, DEF, false> : cblock == 8 ? join_kernel<8, 3, DEF, false> : join_kernel<4, 3, DEF, false>;
  return cblock == 2 ? join_kernel<2, 4, DEF, false> : cblock == 8 ? join_kernel<8, 4, DEF, false> : join_kernel<4, 4, DEF, false>;
}
// The kernel and shared-memory layout of a launch: the default K and R have
// their own kernel, which reads the lists 8 bytes at a time (`aligned`), and
// its FAR form (four CTAs, 4 or 8 sketches in flight: what the tuner offers).
JoinKernel variant(int K, int R, int d, bool aligned, int ctas_per_sm, int cblock, bool far, JoinLayout* L) {
  const bool def = K == kDefK && R == kDefR && aligned;
  far = far && def && ctas_per_sm == 4 && cblock != 2;
  *L = join_layout(K, R, def ? kMaxDim : d, def, far);
  if (far) return cblock == 8 ? join_kernel<8, 4, true, true> : join_kernel<4, 4, true, true>;
  return def ? pick_variant<true>(ctas_per_sm, cblock) : pick_variant<false>(ctas_per_sm, cblock);
}

bool join_has_far(int K, int R) { return K == kDefK && R == kDefR; }

// While most candidates are new, the FAR form is the faster one from about
// where the codes outgrow L2.  First iteration with four CTAs, without / with
// it: 100,000 x 1024 3.82 / 3.78 ms, 150,000 x 1024 6.24 / 6.04, 300,000 x 1024
// 14.6 / 13.4, 600,000 x 1024 33.7 / 29.4, 300,000 x 384 11.87 / 11.98,
// 600,000 x 384 26.6 / 26.5.
bool join_far(int64_t n, int d) { return n * d >= int64_t(120) << 20; }

cudaError_t max_ctas(JoinKernel kern, int ctas_per_sm, int cblock, uint32_t smem, int* per_sm_out) {
  std::lock_guard<std::mutex> lk(g_variant_mu);
  const void* func = reinterpret_cast<const void*>(kern);
  const auto key = std::make_pair(func, smem);
  auto it = g_variant_ctas.find(key);
  if (it != g_variant_ctas.end()) {
    *per_sm_out = it->second;
    return cudaSuccess;
  }
  cudaFuncAttributes fa{};
  cudaError_t e = cudaFuncGetAttributes(&fa, func);  // loads the function
  const char* what = "cudaFuncGetAttributes";
  if (e == cudaSuccess) {
    e = ensure_smem_attr(func, smem);
    what = "cudaFuncSetAttribute";
  }
  int per_sm = 0;
  if (e == cudaSuccess) {
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, func, kThreads, smem);
    what = "cudaOccupancyMaxActiveBlocksPerMultiprocessor";
  }
  if (e != cudaSuccess) {
    cudaGetLastError();  // reported through the return value
    std::snprintf(g_variant_err, sizeof(g_variant_err), "%s(join_kernel<%d,%d>, smem %u, static smem %zu, regs %d): %s",
                  what, cblock, ctas_per_sm, smem, size_t(fa.sharedSizeBytes), fa.numRegs, cudaGetErrorString(e));
    return e;
  }
  per_sm = per_sm < 1 ? 1 : per_sm;
  g_variant_ctas.emplace(key, per_sm);
  *per_sm_out = per_sm;
  return cudaSuccess;
}

const char* join_variant_error() { return g_variant_err; }

cudaError_t join_prepare_all(int K, int R, int d) {
  for (int c : {3, 4})
    for (int b : {2, 4, 8})
      for (bool far : {false, true}) {  // far only where variant() has such a form
        const cudaError_t e = join_prepare(K, R, d, c, b, far);
        if (e != cudaSuccess) return e;
      }
  return cudaSuccess;
}

cudaError_t join_prepare(int K, int R, int d, int ctas_per_sm, int cblock, bool far) {
  JoinLayout L;
  int per_sm = 0;
  const JoinKernel kern = variant(K, R, d, true, ctas_per_sm, cblock, far, &L);
  return max_ctas(kern, ctas_per_sm, cblock, L.bytes, &per_sm);
}

cudaError_t launch_stop_check(const JobTable& jt, const JoinCtl& ctl, int K, int out_buf, float stop_rate,
                              float diff_tol, const cudaGraphConditionalHandle* loop, cudaStream_t s) {
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  stop_check_kernel<<<1, 256, 0, s>>>(jt, ctl, K, out_buf, stop_rate, diff_tol, loop ? *loop : cudaGraphConditionalHandle{},
                                      loop ? 1 : 0);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_join(const int8_t* codes, const uint64_t* sketch, int64_t n, int d, int K, int R,
                        const int32_t* ids_in, const int32_t* scores_in, int32_t* ids_out, int32_t* scores_out,
                        const int32_t* row_order, unsigned long long* counters, int num_sms, cudaStream_t s,
                        const JobTable* jt, const JoinCtl* ctl, int ctas_per_sm, int cblock, int sk_words, bool far) {
  JoinLayout L;
  const JoinKernel kern = variant(K, R, d, (reinterpret_cast<uintptr_t>(ids_in) & 7) == 0, ctas_per_sm, cblock, far, &L);
  int per_sm = 1;
  KNNG_CUDA_TRY(max_ctas(kern, ctas_per_sm, cblock, L.bytes, &per_sm));
  const int64_t blocks = std::min<int64_t>(n, int64_t(num_sms) * per_sm);
  cudaGetLastError();  // clear a stale, non-sticky error: the launch reports only its own
  kern<<<unsigned(blocks), kThreads, L.bytes, s>>>(codes, sketch, n, d, K, R, sk_words > 0 ? sk_words : d / 64, ids_in,
                                                   scores_in, ids_out, scores_out, row_order, counters,
                                                   jt ? *jt : JobTable{}, ctl ? *ctl : JoinCtl{}, L);
  note_launch();
  return cudaGetLastError();
}

}  // namespace knng
