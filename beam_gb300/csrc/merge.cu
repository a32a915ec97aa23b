// Merge on the GPU: the blocked EA merge loop (Sweg::Merge, blocked mode,
// src/sweg.cpp:953-1145), one block of group_batch_size groups at a time
// (64 in the reference's recommended mode; one block of all groups in the
// batched form).
//
//   Plan*Kernel        the bookkeeping of large blocks on the device (lists and
//                      offsets of the groups, sums at the blocks' borders)
//   Prepare*Kernel     EA-proxy candidates per group (src/sweg.cpp:1598-1727,
//                      1800-1999): a warp per small group; big groups by CTA
//                      or by a GPU-wide sort of their row entries
//   ScoreKernel        exact merge gain per candidate pair
//                      (QuotientGraph::ExactMergeGainPersistentImpl,
//                      src/quotient_graph.cpp:340-462)
//   Select*Kernel      reciprocal threshold filter + g0 greedy selection
//                      (src/sweg.cpp:2146-2186, 2188-2281)
//   Commit*Kernel,     CommitSelectedPairs + Update_S + QuotientGraph::Merge
//   RewriteRowsKernel  for the block (src/sweg.cpp:2665-2769, 2977-3015,
//                      src/quotient_graph.cpp:628-742): sizes, internal
//                      counts, member lists, keep rows rebuilt from
//                      keep+remove, neighbour rows of removed supernodes
//                      rewritten in place
//   VerifyKernel       optional commit-time re-scoring (--verify-cuda-gain)
//
// The reference validates every selected pair of a block before applying any
// of them (Update_S runs after the validation loop), and the pairs of a block
// are endpoint-disjoint, so the block's merges are applied as one batch; the
// resulting rows are the canonical sorted, count-summed rows, identical to
// the reference's sequential incremental updates.

#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>

#include "engine.h"

namespace beam {
namespace {

// Shared memory of an SM, and what every resident CTA takes of it beside its own.
constexpr size_t kSmemPerSm = 228 << 10;
constexpr size_t kSmemReserved = 1 << 10;
constexpr int kPrepThreads = 512;
constexpr int kLaneTopK = 32;        // per-lane candidate lists for top_k up to this
constexpr int kSmemEntries = 2048;   // bucket entries held in shared memory
constexpr int kSmemHeads = 4096;     // bucket hash heads in shared memory
// Groups of more than this many members take the sorted (GPU-wide) path
// even when their rows fit the shared-memory table: the pairs of members
// sharing a target grow with the square of the member count, too much work
// for one CTA.
constexpr int kSmemMaxGroup = 48;
constexpr int kScoreThreads = 256;
constexpr int kFewGroups = 256;  // blocks of at most this many groups take fewer, wider launches
// Selection by group size: at most kSelectSmallGroup members, a warp each;
// up to kSelectMidGroup, a small CTA each (sort + greedy pass); larger groups,
// matching rounds. The two are equal: the matching rounds measured faster
// than the small CTAs for groups of 9..32 members.
constexpr int kSelectMidGroup = 8;
constexpr int kSelectMidThreads = 128;
constexpr int kSelectMidKeys = 512;   // >= min(C(32,2), 16 * 32) candidates
constexpr int kRowsThreads = 256;
constexpr int kRowSmem = 2048;       // staged row entries in shared memory
constexpr int kWarpRow = 32;         // neighbour rows rewritten by one warp in registers
constexpr int kWarpRowMax = 256;     // neighbour rows rewritten by one warp through shared memory
// Neighbour rows of more than kRowSmem entries are rewritten in two steps: the
// renamed entries found by warps over kHugeUnit entries each, the row moved by
// one CTA in chunks of kHugeChunk.
// (A window's batch claims few rows: the shorter ones gain from it too.)
constexpr int kWindowRow = 256;
constexpr int kHugeUnit = 1024;
constexpr int kHugeThreads = 1024;
constexpr int kHugePer = 8;
constexpr int kHugeChunk = kHugeThreads * kHugePer;
constexpr int kHugeGrid = 152;
constexpr int kKeyIdxBits = 10;      // a_idx, b_idx < kMaxGroup
constexpr long long kKeyGainMax = (1ll << (64 - 2 * kKeyIdxBits)) - 1;
constexpr unsigned long long kKeyIdxMask = (1ull << kKeyIdxBits) - 1;

// Selection key: ascending order is g0's (gain desc, a_idx asc, b_idx asc).
__device__ __forceinline__ unsigned long long PackKey(long long gain, int a, int b) {
  return (static_cast<unsigned long long>(kKeyGainMax - gain) << (2 * kKeyIdxBits)) |
         (static_cast<unsigned long long>(a) << kKeyIdxBits) | static_cast<unsigned long long>(b);
}

__device__ __forceinline__ unsigned long long* ScratchAlloc(unsigned char* base, unsigned long long cap,
                                                           BlockCtl* ctl, unsigned long long bytes,
                                                           DevError* err) {
  bytes = (bytes + 255) & ~255ull;
  const unsigned long long at = atomicAdd(&ctl->scratch_top, bytes);
  if (at + bytes > cap) {
    RaiseError(err, kErrScratch, static_cast<int>(bytes >> 20), static_cast<int>(cap >> 20), 0);
    return nullptr;
  }
  return reinterpret_cast<unsigned long long*>(base + at);
}

// ------------------------------------------------------------ exact gain

struct GainWork {
  long long raw_a, raw_b, uni, ovl;
  long long bytes;  // algorithmic bytes of the gain computations
};

// The before and after terms of the union of two sorted row ranges (entries
// toward a and b themselves aside), by a warp, as a tiled merge: each step
// loads the next 32 entries of both (coalesced); with lim = the smaller of the
// two tiles' last neighbours, every entry <= lim is final in this step (an
// equal neighbour in the other range, if any, is in the other tile), and each
// lane finds its entry in the other tile by a 5-step shuffle search. Shared
// neighbours give two before-terms, one-sided neighbours one. Every term is
// exact int64; the work is O(la + lb). Sums are the lanes' own.
struct MergeTerms {
  long long before = 0, after = 0, eab_a = 0, eab_b = 0;  // e(a, b) as read from either row
  int uni = 0, ovl = 0, bad = 0;
};

__device__ __forceinline__ void WarpMergeTerms(const QuotientView& Q, int a, int b, long long sa, long long sb,
                                               const Entry* ra, int la, const Entry* rb, int lb, MergeTerms* T) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr Entry kPadEntry = static_cast<Entry>(0x7fffffffull) << 32;  // neighbour INT_MAX, count 0
  const int lane = threadIdx.x & 31;
  const long long sw = sa + sb;
  int pa = 0, pb = 0;
  while (pa < la || pb < lb) {
    const bool va = pa + lane < la;
    const bool vb = pb + lane < lb;
    const Entry ea_e = va ? ra[pa + lane] : kPadEntry;
    const Entry eb_e = vb ? rb[pb + lane] : kPadEntry;
    const int xa = EntNb(ea_e);
    const int xb = EntNb(eb_e);
    const int last_a = __shfl_sync(kFull, xa, 31);
    const int last_b = __shfl_sync(kFull, xb, 31);
    const int lim = last_a < last_b ? last_a : last_b;
    // lower bound of xa in the b tile and of xb in the a tile
    int pos_b = 0, pos_a = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const int probe_b = __shfl_sync(kFull, xb, pos_b + step - 1);
      const int probe_a = __shfl_sync(kFull, xa, pos_a + step - 1);
      if (probe_b < xa) pos_b += step;
      if (probe_a < xb) pos_a += step;
    }
    const Entry cand_b = __shfl_sync(kFull, eb_e, pos_b);
    const Entry cand_a = __shfl_sync(kFull, ea_e, pos_a);
    const bool fin_a = va && xa <= lim;
    const bool fin_b = vb && xb <= lim;
    if (fin_a) {
      const long long ca = EntCnt(ea_e);
      if (xa == b) {
        T->eab_a = ca;
      } else {
        const long long sx = Q.size[xa];
        if (EntNb(cand_b) == xa) {
          const long long cb = EntCnt(cand_b);
          T->before += BlockCost(sa, sx, ca, false, T->bad) + BlockCost(sb, sx, cb, false, T->bad);
          T->after += BlockCost(sw, sx, ca + cb, false, T->bad);
          ++T->ovl;
        } else {
          T->before += BlockCost(sa, sx, ca, false, T->bad);
          T->after += BlockCost(sw, sx, ca, false, T->bad);
        }
        ++T->uni;
      }
    }
    if (fin_b) {
      const long long cb = EntCnt(eb_e);
      if (xb == a) {
        T->eab_b = cb;
      } else if (EntNb(cand_a) != xb) {
        const long long sx = Q.size[xb];
        T->before += BlockCost(sb, sx, cb, false, T->bad);
        T->after += BlockCost(sw, sx, cb, false, T->bad);
        ++T->uni;
      }
    }
    pa += __popc(__ballot_sync(kFull, fin_a));
    pb += __popc(__ballot_sync(kFull, fin_b));
  }
}

// ExactMergeGainPersistentImpl by a warp; e(a,b) is read from both rows and
// must agree.
__device__ void WarpExactGain(const QuotientView& Q, int a, int b, long long* gain_out, long long* before_out,
                              GainWork* work, DevError* err) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long sa = Q.size[a];
  const long long sb = Q.size[b];
  const long long sw = sa + sb;
  const int la = Q.len[a];
  const int lb = Q.len[b];
  MergeTerms T;
  WarpMergeTerms(Q, a, b, sa, sb, Q.ent + Q.off[a], la, Q.ent + Q.off[b], lb, &T);
  long long before = T.before, after = T.after, eab_a = T.eab_a, eab_b = T.eab_b;
  int uni = T.uni, ovl = T.ovl, bad = T.bad;
  before = WarpSum(before);
  after = WarpSum(after);
  // e(a,b) is read by one lane per row (counts < 2^32)
  eab_a = __reduce_max_sync(kFull, static_cast<unsigned>(eab_a));
  eab_b = __reduce_max_sync(kFull, static_cast<unsigned>(eab_b));
  uni = static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(uni)));
  ovl = static_cast<int>(__reduce_add_sync(kFull, static_cast<unsigned>(ovl)));
  bad = __any_sync(kFull, bad);
  if (eab_a != eab_b) {
    if (lane == 0) RaiseError(err, kErrAsymmetric, a, b, 0);
  }
  const long long ia = Q.internal[a];
  const long long ib = Q.internal[b];
  before += BlockCost(sa, sa, ia, true, bad) + BlockCost(sb, sb, ib, true, bad) + BlockCost(sa, sb, eab_a, false, bad);
  after += BlockCost(sw, sw, ia + ib + eab_a, true, bad);
  if (bad && lane == 0) RaiseError(err, kErrBlockCost, a, b, 0);
  *gain_out = before - after;
  *before_out = before;
  if (work) {
    work->raw_a += la;
    work->raw_b += lb;
    work->uni += uni;
    work->ovl += ovl;
    // 8 B per row entry, 4 B per union-neighbour size gather
    work->bytes += 8ll * (la + lb) + 4ll * uni;
  }
}

// The exact gain from sums. The gain
// of a pair is a sum over the union of its two rows. The prepare kernels read
// every member row with its target sizes anyway, and visit every target that
// two members share, so they leave behind all that the gain needs: sums per
// row (RowSums) and the shared targets' part per candidate (PairInfo). The
// scoring pass then reads no row at all.
//
// With s = size_a + size_b and f_s(c) = min(c, 1 + s * size_x - c):
//   before = before[a] + before[b] - BC(s_b, s_a, e_ab) + BC_int(a) + BC_int(b)
//   after  = F_a(s) + F_b(s) - BC(s, s_b, e_ab) - BC(s, s_a, e_ab) + shared
//            + BC_int(s, i_a + i_b + e_ab),
//   F_r(s) = sum over row r of f_s(c),
//   shared = sum over shared x of [f_s(c_ax + c_bx) - f_s(c_ax) - f_s(c_bx)]:
// the integers of QuotientGraph::ExactMergeGainPersistentImpl, regrouped.
//
// F_r(s) without the row: an entry is light when 1 + (size_r + 1) * size_x >=
// 2c, so f_s(c) = c for every merged size; of the others (heavy) each is
// dense, f_s(c) = 1 + s * size_x - c, up to its own size limit
// (2c - 2) / size_x, and c beyond. smin / smax are the least and the largest of
// those limits: for s <= smin all heavy entries are dense, for s > smax none.
// Sizes in between (rows with several heavy entries of different limits) read
// the row.
constexpr int kHeavyFew = 4;
struct __align__(64) RowSums {
  long long before;    // sum of BC(size_r, size_x, c)
  long long light;     // sum of c over the light entries
  long long heavy_sx;  // over the heavy entries: sum of size_x
  long long heavy_c;   //                         sum of c
  int smin, smax;      //                         least / largest size limit
  long long internal;  // internal edges of the supernode
  int size, len;
  int nheavy;          // heavy entries
  int sbad;            // a size below this holds fewer edges than some entry counts (0: none does)
};
static_assert(sizeof(RowSums) == 64, "two sectors per row");

__device__ __forceinline__ bool HeavyEntry(long long size_r, long long size_x, long long c) {
  return 1 + (size_r + 1) * size_x < 2 * c;
}

__device__ __forceinline__ int HeavyLimit(long long size_x, long long c) {
  if (c < (1ll << 30)) return static_cast<int>(static_cast<unsigned>(2 * c - 2) / static_cast<unsigned>(size_x));
  const long long l = (2 * c - 2) / size_x;
  return l > 0x7fffffffll ? 0x7fffffff : static_cast<int>(l);
}

// Least size whose block with a target of size_x holds cnt edges. An entry
// beyond its own block's capacity is always heavy.
__device__ __forceinline__ int HeavyNeed(long long size_x, long long cnt) {
  if (cnt < (1ll << 30)) {
    const unsigned x = static_cast<unsigned>(size_x);
    return static_cast<int>((static_cast<unsigned>(cnt) + x - 1u) / x);
  }
  const long long n = (cnt + size_x - 1) / size_x;
  return n > 0x7fffffffll ? 0x7fffffff : static_cast<int>(n);
}

// The heavy part of a row's sums; one lane's share, then the warp's.
struct HeavyAcc {
  long long sx = 0, c = 0;
  int smin = 0x7fffffff, smax = 0, n = 0, sbad = 0;
  __device__ __forceinline__ void Add(long long size_x, long long cnt) {
    const int l = HeavyLimit(size_x, cnt);
    const int need = HeavyNeed(size_x, cnt);
    sbad = need > sbad ? need : sbad;
    sx += size_x;
    c += cnt;
    smin = l < smin ? l : smin;
    smax = l > smax ? l : smax;
    ++n;
  }
  __device__ __forceinline__ void Merge(const HeavyAcc& o) {
    sx += o.sx;
    c += o.c;
    smin = o.smin < smin ? o.smin : smin;
    smax = o.smax > smax ? o.smax : smax;
    sbad = o.sbad > sbad ? o.sbad : sbad;
    n += o.n;
  }
  __device__ __forceinline__ void WarpReduce() {
    n = WarpSumInt(n);
    if (n == 0) return;
    sx = WarpSum(sx);
    c = WarpSum(c);
    smin = __reduce_min_sync(0xffffffffu, smin);
    smax = __reduce_max_sync(0xffffffffu, smax);
    sbad = __reduce_max_sync(0xffffffffu, sbad);
  }
};

__device__ __forceinline__ void StoreRowSums(RowSums* out, long long before, long long light, const HeavyAcc& h,
                                             long long internal, int size, int len) {
  RowSums r;
  r.before = before;
  r.light = light;
  r.heavy_sx = h.sx;
  r.heavy_c = h.c;
  r.smin = h.smin;
  r.smax = h.smax;
  r.internal = internal;
  r.size = size;
  r.len = len;
  r.nheavy = h.n;
  r.sbad = h.sbad;
  *out = r;
}

__device__ __forceinline__ bool RowAfterKnown(const RowSums& r, long long s) {
  return r.nheavy == 0 || s <= r.smin || s > r.smax;
}

// F_r(s) from the sums; false: the row has to be read (WarpRowAfter); *out is its light part then.
__device__ __forceinline__ bool RowAfter(const RowSums& r, long long s, long long* out) {
  *out = r.light;
  if (r.nheavy == 0) return true;
  if (s <= r.smin) {
    *out += r.nheavy + s * r.heavy_sx - r.heavy_c;
    return true;
  }
  if (s > r.smax) {
    *out += r.heavy_c;
    return true;
  }
  return false;
}

// Sum of f_s(c) over row r, by a warp.
__device__ long long WarpRowAfter(const QuotientView& Q, int r, long long s) {
  const int lane = threadIdx.x & 31;
  const Entry* row = Q.ent + Q.off[r];
  const int len = Q.len[r];
  long long sum = 0;
  for (int k = lane; k < len; k += 32) {
    const Entry e = row[k];
    const long long c = EntCnt(e);
    const long long alt = 1 + s * Q.size[EntNb(e)] - c;
    sum += c < alt ? c : alt;
  }
  return WarpSum(sum);
}

// The shared part of a candidate pair.
struct __align__(16) PairInfo {
  long long shared;  // sum over the shared targets (see above)
  unsigned ovl;      // shared targets (low 30 bits) and the flags below
  unsigned eab;      // edges between the two
};
constexpr unsigned kPairBad = 1u << 31;   // a shared target's count exceeds its block capacity
constexpr unsigned kPairAsym = 1u << 30;  // the two rows disagree about e(a, b)

// The pair tables of a big group (g x g words, row-major). Word (i, j), i < j:
// the EA proxy in the low kProxyBits, the number of shared targets above it,
// bit 62 set when row i lists j, bit 63 when row j lists i. Word (j, i): the
// shared part plus the proxy's own (shared = that word - proxy of the targets),
// zero unless a target of the pair is dense in one of the rows; a target whose
// count exceeds the merged block adds kCorrBad instead. A proxy is at most the
// two rows' counts plus the direct edges, below 2^34 (edges < 2^32); shared
// targets are counted only with row sums, on graphs of fewer than 2^30 arcs:
// two rows share fewer than 2^28 targets there.
constexpr int kProxyBits = 34;
constexpr unsigned long long kProxyMask = (1ull << kProxyBits) - 1;
constexpr unsigned long long kOvlOne = 1ull << kProxyBits;
constexpr unsigned long long kOvlMask = (1ull << (62 - kProxyBits)) - 1;
constexpr unsigned long long kRowILists = 1ull << 62;
constexpr unsigned long long kRowJLists = 1ull << 63;
constexpr long long kCorrBad = 1ll << 36;
constexpr long long kFusedMaxArcs = 1ll << 30;

// One target of size st shared by members of sizes sa and sb with counts ca
// and cb: the EA proxy's term max(0, old - new) (src/sweg.cpp:1598-1727) and
// corr = f(ca + cb) - f(ca) - f(cb) + that term.
struct SharedTerm {
  long long delta, corr;
};

__device__ __forceinline__ SharedTerm TermOf(long long sa, long long sb, long long st, long long ca, long long cb,
                                             bool* bad) {
  auto mn = [](long long x, long long y) { return x < y ? x : y; };
  const long long cap_a = sa * st, cap_b = sb * st, cap = cap_a + cap_b, c = ca + cb;
  const long long ga = mn(ca, 1 + cap_a - ca), gb = mn(cb, 1 + cap_b - cb), f = mn(c, 1 + cap - c);
  const long long d = ga + gb - f;
  SharedTerm t;
  t.delta = d > 0 ? d : 0;
  t.corr = f - mn(ca, 1 + cap - ca) - mn(cb, 1 + cap - cb) + t.delta;
  *bad = c > cap;
  return t;
}

// The last index i of [lo, hi) with a[i] <= x, for a non-decreasing array
// with a[lo] <= x, found by the whole warp (warp-uniform arguments): each
// round probes 32 points of the remaining span, so the search takes about
// log32 of the span in dependent loads instead of log2.
__device__ __forceinline__ int WarpLastLE(const long long* __restrict__ a, int lo, int hi, long long x) {
  const int lane = threadIdx.x & 31;
  while (hi - lo > 1) {
    // lo < p, p <= hi - 1, non-decreasing over the lanes
    const int p = lo + 1 + static_cast<int>((static_cast<long long>(hi - lo - 1) * lane) >> 5);
    const int k = __popc(__ballot_sync(0xffffffffu, a[p] <= x));  // lanes 0..k-1 hold
    const int p_lo = __shfl_sync(0xffffffffu, p, k > 0 ? k - 1 : 0);
    const int p_hi = __shfl_sync(0xffffffffu, p, k < 32 ? k : 31);
    if (k > 0) lo = p_lo;
    if (k < 32) hi = p_hi;
  }
  return lo;
}

// ------------------------------------------------------------ prepare

// Per-group arrays of the merge kernels (cand_off, cand_cnt, mat_off,
// sel_off, sel_cnt) are indexed by the group's position in the iteration's
// list of groups with at least two members ("real" groups); real[ri] is the
// Divide group id. A block covers the real groups [rg0, rg0 + nrg).
// A big group with more than kSmemMaxGroup members, or whose row entries
// (counted at Divide time, an upper bound for the rest of the iteration: rows
// of supernodes not yet merged only shrink) exceed the shared-memory bucket
// table, is deferred. PrepareKernel stages its row offsets and member scalars
// in block scratch; PrepareFillKernel writes one (group, target) key and one
// (member, count) value per row entry into the group's sort slots, a radix
// sort brings the entries of every (group, target) together, and
// PrepareAccumKernel pairs the entries of each run, a warp per 32 sorted
// slots. No group is bound to one SM.
// Scratch layout: eoff int32[g+1] | mq int32[g] | msz int32[g].
struct BigDesc {
  unsigned char* base;  // nullptr: not deferred
  int E;
  int pad;
};

struct DeferredView {
  int* eoff;
  int* mq;
  int* msz;
};

__host__ __device__ __forceinline__ unsigned long long DeferredBytes(int g) {
  return 4ull * (3ull * static_cast<unsigned long long>(g) + 1);
}

__device__ __forceinline__ DeferredView Deferred(unsigned char* base, int g) {
  DeferredView V;
  V.eoff = reinterpret_cast<int*>(base);
  V.mq = V.eoff + g + 1;
  V.msz = V.mq + g;
  return V;
}

// Sort key of a deferred group's entry, from the top: low bits of the
// launch-local group index, its other bits, the target. Fill writes the slots
// in the order of the groups and the sort is stable, so it needs the lower two
// fields only: entries of one (group, target) come out side by side, the
// targets of 2^low neighbouring groups interleaved. Low bits are left out where
// that saves a digit of the sort, a pass bound by its ranking and not by bytes
// (keys and values in one word were no faster), up to kSlotGroupBits of them:
// the pair tables of 32 groups of 512 members are 64 MB, half the L2. RMAT-23,
// 23 + 14 bits in 4 passes for 5: sorts 152 -> 117 ms of a run, the adding up
// 136.5 -> 137.7; RMAT-20 with the ranker 135.7 -> 130 ms in all.
constexpr unsigned long long kSlotPad = ~0ull;  // an unused sort slot
constexpr int kSlotGroupBits = 5;
constexpr int kSortDigit = 8;

struct SlotBits {
  int target;  // bits of a target
  int group;   // bits of a group index that are sorted
  int low;     // bits of a group index that are not
  __host__ __device__ int sorted() const { return target + group; }
  __device__ unsigned long long Key(int k, int t) const {
    const unsigned long long high = static_cast<unsigned long long>(k >> low) << target | static_cast<unsigned>(t);
    return static_cast<unsigned long long>(k & ((1 << low) - 1)) << sorted() | high;
  }
  __device__ int Target(unsigned long long key) const { return static_cast<int>(key & ((1ull << target) - 1ull)); }
  __device__ int Group(unsigned long long key) const {
    return static_cast<int>(key >> target & ((1ull << group) - 1ull)) << low | static_cast<int>(key >> sorted());
  }
};

// No sorted field of a key has the padding's bits: the group index's upper
// part stays below all ones.
SlotBits SlotLayout(int n, int groups) {
  SlotBits b{1, 1, 0};
  while ((1ll << b.target) < n) ++b.target;
  auto sorted_bits = [&](int low) {
    int bits = 1;
    while ((groups - 1) >> low >= (1 << bits) - 1) ++bits;
    return bits;
  };
  b.group = sorted_bits(0);
  // the fewest low bits that save a digit
  const int digits = (b.sorted() + kSortDigit - 1) / kSortDigit;
  for (int low = 1; low <= kSlotGroupBits && b.low == 0; ++low) {
    if (b.target + sorted_bits(low) <= (digits - 1) * kSortDigit) {
      b.group = sorted_bits(low);
      b.low = low;
    }
  }
  return b;
}

// The same in 32 bits: sizes below 2^13, counts below 2^28.
__device__ __forceinline__ void TermOf32(int sa, int sb, int st, int ca, int cb, int* delta, int* corr, bool* bad) {
  const int cap_a = sa * st, cap_b = sb * st, cap = cap_a + cap_b, c = ca + cb;
  const int ga = min(ca, 1 + cap_a - ca), gb = min(cb, 1 + cap_b - cb), f = min(c, 1 + cap - c);
  const int d = max(ga + gb - f, 0);
  *delta = d;
  *corr = f - min(ca, 1 + cap - ca) - min(cb, 1 + cap - cb) + d;
  *bad = c > cap;
}

struct PrepareParams {
  QuotientView Q;
  const int* order;
  const int* gstart;
  const int* glen;
  const int* group_of;
  const int* idx_in_group;
  const int* real;
  const int* list;  // real-group positions handled by this launch
  int list0;
  int nlist;
  const long long* moff;  // member-count prefix over the big-group list
  BigDesc* desc;          // per big-group list entry
  float2* cand_feat;      // per candidate: proxy gain, proxy ratio (ranker features; nullptr: off)
  int2* cand_rep;         // per candidate slot: the pair's supernode ids (unused slots stay -1)
  const long long* soff;  // sort-slot prefix over the big-group list (0 slots: not deferred)
  long long slot0;        // soff of the launch's first entry
  SlotBits bits;             // fields of a sort key
  unsigned long long* skey;  // unsorted keys / values of the launch's slots
  unsigned long long* sval;
  const unsigned long long* skey_sorted;
  const unsigned long long* sval_sorted;
  long long nslots;
  const long long* cand_off;
  int2* cand;
  int* cand_cnt;
  const long long* mat_off;
  unsigned char* mat;
  int mat_zeroed;  // the pair tables were cleared by one memset of the block
  // row sums and pair sums for the scoring pass (nullptr: not needed)
  RowSums* rc;
  PairInfo* info;
  unsigned char* scratch;
  unsigned long long scratch_cap;
  BlockCtl* ctl;
  int top_k;
  unsigned long long* stats;
  DevError* err;
};

// Per big group: pair words u64[g*g] | kept flag u8[g*g] | old cost int64[g];
// the flag table starts at FlagOffset and the old costs at OldCostOffset
// (rounded up to 8-byte alignment).
__host__ __device__ __forceinline__ long long FlagOffset(long long gg) { return 8 * gg; }
__host__ __device__ __forceinline__ long long OldCostOffset(long long gg) { return (9 * gg + 7) & ~7ll; }

// rb: the bits of the candidate's double ratio (the reference's rounded
// quotient, computed once per candidate); positive doubles order like their
// bit patterns, so candidates are compared on the integer pipes (this GPU's
// FP64 rate is a small fraction of its integer rate)
struct RankKey {
  unsigned long long rb;
  long long pg;
  int lo, hi, j;
};

// ranked_better (src/sweg.cpp:1926-1938): ratio desc, proxy gain desc,
// rep_lo asc, rep_hi asc.
__device__ __forceinline__ bool Better(const RankKey& x, const RankKey& y) {
  if (x.rb != y.rb) return x.rb > y.rb;
  if (x.pg != y.pg) return x.pg > y.pg;
  if (x.lo != y.lo) return x.lo < y.lo;
  return x.hi < y.hi;
}

// The same order without a double, for proxies and denominators below
// kExactRatio: two different quotients p / d of such numbers are more than
// 2^-52 apart (relative), so they round to different doubles, and cross products
// order them as the rounded quotients. One double division by a warp holds this
// GPU's FP64 pipe for some 250 cycles; ranked that way, it was what the member
// passes waited for. Between partners of one member, (rep_lo, rep_hi) ascending
// is the partner's id ascending.
constexpr long long kExactRatio = 1ll << 26;

struct RankCand {
  unsigned p, d;  // proxy gain (0: no candidate), denominator
  int q;          // partner
};

// Ranks of a member's candidates, kPer to a lane, by the whole warp: rank[t] is
// the number of candidates better than the lane's t-th (meaningful for a
// candidate; p == 0 is none). Every lane's candidate in turn, four in flight.
template <int kPer>
__device__ __forceinline__ void ExactRanks(const RankCand (&c)[kPer], int (&rank)[kPer]) {
#pragma unroll
  for (int t = 0; t < kPer; ++t) rank[t] = 0;
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
#pragma unroll 4
    for (int o = 0; o < 32; ++o) {
      const unsigned op = __shfl_sync(0xffffffffu, c[u].p, o);
      const unsigned od = __shfl_sync(0xffffffffu, c[u].d, o);
      const int oq = __shfl_sync(0xffffffffu, c[u].q, o);
#pragma unroll
      for (int t = 0; t < kPer; ++t) {
        const unsigned long long l = static_cast<unsigned long long>(op) * c[t].d;
        const unsigned long long r = static_cast<unsigned long long>(c[t].p) * od;
        const bool better = l != r ? l > r : op != c[t].p ? op > c[t].p : oq < c[t].q;  // not better than itself
        rank[t] += better ? 1 : 0;
      }
    }
  }
}

// The reference's threshold test RN(gain / before) >= threshold (doubles, gain
// and before > 0) on the integer pipes, with threshold = m * 2^-e exactly
// (split on the host; e < 0: no split). Rounding is monotonic, so a quotient
// at or above the threshold passes, and one more than 2^-51 (relative) below
// it rounds below it and fails; only the band in between, and counts of 2^53
// or more (which the double conversion rounds), take the double division.
struct ThresholdBits {
  unsigned long long m;
  int e;
};

__host__ inline ThresholdBits SplitThreshold(double threshold) {
  ThresholdBits t{0, -1};
  if (threshold > 0.0 && std::isfinite(threshold)) {
    int ex = 0;
    const double f = std::frexp(threshold, &ex);  // threshold = f * 2^ex, f in [0.5, 1)
    t.m = static_cast<unsigned long long>(std::ldexp(f, 53));
    t.e = 53 - ex;
  }
  return t;
}

__device__ __forceinline__ bool RatioAtLeast(long long gain, long long before, double threshold, ThresholdBits t) {
  if (t.e >= 0 && t.e <= 63 && gain < (1ll << 53) && before < (1ll << 53)) {
    const unsigned __int128 l = static_cast<unsigned __int128>(static_cast<unsigned long long>(gain)) << t.e;
    const unsigned __int128 r = static_cast<unsigned __int128>(t.m) * static_cast<unsigned long long>(before);
    if (l >= r) return true;
    if (l + (r >> 51) < r) return false;
  }
  return static_cast<double>(gain) / static_cast<double>(before) >= threshold;
}

__device__ __forceinline__ unsigned BucketHash(int t, unsigned mask) {
  return (static_cast<unsigned>(t) * 0x9E3779B1u) >> 7 & mask;
}

// Adds a shared target (size st; counts ca, cb in the rows of members i, j) to
// the pair's words: one atomic, and a second one where a dense entry is part
// of it. counted: the shared part of the gain is wanted too.
__device__ __forceinline__ void AddShared(unsigned long long* pmat, int g, int i, int j, long long si, long long sj,
                                          long long st, long long ca, long long cb, bool counted) {
  bool bad;
  const SharedTerm t = TermOf(si, sj, st, ca, cb, &bad);
  const long long lo = i < j ? i : j;
  const long long hi = i < j ? j : i;
  const unsigned long long add = static_cast<unsigned long long>(t.delta) + (counted ? kOvlOne : 0ull);
  if (add != 0) atomicAdd(&pmat[lo * g + hi], add);
  if (counted && (t.corr != 0 || bad)) {
    atomicAdd(&pmat[hi * g + lo], static_cast<unsigned long long>(bad ? kCorrBad : t.corr));
  }
}

// Member i's row lists member j with c edges: counted once, from the lower
// index; the other side leaves its mark.
__device__ __forceinline__ void AddDirect(unsigned long long* pmat, int g, int i, int j, long long c) {
  if (i < j) {
    atomicAdd(&pmat[static_cast<long long>(i) * g + j], static_cast<unsigned long long>(c) | kRowILists);
  } else {
    atomicAdd(&pmat[static_cast<long long>(j) * g + i], kRowJLists);
  }
}

__device__ __forceinline__ unsigned long long PairWord(const unsigned long long* pmat, int g, int i, int j) {
  return i < j ? pmat[static_cast<long long>(i) * g + j] : pmat[static_cast<long long>(j) * g + i];
}

__device__ __forceinline__ long long ProxyOf(unsigned long long word) {
  return static_cast<long long>(word & kProxyMask);
}

struct PrepSmem {
  int q[kMaxGroup];
  int sz[kMaxGroup];
  int len[kMaxGroup];
  long long off[kMaxGroup];
  long long old[kMaxGroup];
  int eoff[kMaxGroup + 1];
  int heads[kSmemHeads];
  int et[kSmemEntries];
  int ei[kSmemEntries];
  unsigned ee[kSmemEntries];
  int enx[kSmemEntries];
  unsigned long long examined;
  int total;
};

__global__ void __launch_bounds__(kPrepThreads) PrepareKernel(PrepareParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PrepSmem& S = *reinterpret_cast<PrepSmem*>(smem_raw);
  using BlockScan = cub::BlockScan<int, kPrepThreads>;
  __shared__ typename BlockScan::TempStorage scan_tmp;
  __shared__ int carry;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nwarps = kPrepThreads / 32;
  const int ri = P.list[P.list0 + blockIdx.x];
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  BigDesc* desc = P.desc + P.list0 + blockIdx.x;
  if (tid == 0) {
    desc->base = nullptr;
    desc->E = 0;
  }
  // sort slots of a deferred group start as padding, so that every exit
  // below leaves them well-defined for the sort and the accumulate pass
  const long long slot_beg = P.soff[P.list0 + blockIdx.x];
  const long long slots = P.soff[P.list0 + blockIdx.x + 1] - slot_beg;
  {
    unsigned long long* key = P.skey + (slot_beg - P.slot0);
    for (long long k = tid; k < slots; k += kPrepThreads) key[k] = kSlotPad;
  }
  if (g < 2) {
    if (tid == 0) P.cand_cnt[ri] = 0;
    return;
  }
  if (g > kMaxGroup) {
    if (tid == 0) {
      RaiseError(P.err, kErrGroupTooLarge, gid, g, 0);
      P.cand_cnt[ri] = 0;
    }
    return;
  }
  const QuotientView& Q = P.Q;
  const int start = P.gstart[gid];
  for (int i = tid; i < g; i += kPrepThreads) {
    const int rep = P.order[start + i];
    S.q[i] = rep;
    S.sz[i] = Q.size[rep];
    S.len[i] = Q.len[rep];
    S.off[i] = Q.off[rep];
  }
  if (tid == 0) {
    S.examined = 0;
    carry = 0;
  }
  __syncthreads();
  // exclusive scan of row lengths -> entry offsets
  for (int base = 0; base < g; base += kPrepThreads) {
    const int i = base + tid;
    const int v = i < g ? S.len[i] : 0;
    int ex = 0, agg = 0;
    BlockScan(scan_tmp).ExclusiveSum(v, ex, agg);
    if (i < g) S.eoff[i] = carry + ex;
    __syncthreads();
    if (tid == 0) carry += agg;
    __syncthreads();
  }
  const int E = carry;
  if (tid == 0) S.eoff[g] = E;
  const long long gg = static_cast<long long>(g) * g;
  unsigned char* mat = P.mat + P.mat_off[ri];
  unsigned long long* pmat = reinterpret_cast<unsigned long long*>(mat);
  unsigned char* fmat = mat + FlagOffset(gg);
  if (slots > 0) {
    // deferred group: row offsets and member scalars in block scratch, pair
    // tables zeroed, unused sort slots padded; fill / sort / accumulate follow
    if (E > slots) {
      if (tid == 0) {
        RaiseError(P.err, kErrSlots, gid, E, static_cast<int>(slots));
        P.cand_cnt[ri] = 0;
      }
      return;
    }
    __shared__ unsigned char* dbase;
    if (tid == 0) {
      dbase = reinterpret_cast<unsigned char*>(ScratchAlloc(P.scratch, P.scratch_cap, P.ctl, DeferredBytes(g), P.err));
    }
    __syncthreads();
    if (dbase == nullptr) {
      if (tid == 0) P.cand_cnt[ri] = 0;
      return;
    }
    const DeferredView V = Deferred(dbase, g);
    long long* old_out = reinterpret_cast<long long*>(mat + OldCostOffset(gg));
    for (int i = tid; i < g; i += kPrepThreads) {
      V.eoff[i] = S.eoff[i];
      V.mq[i] = S.q[i];
      V.msz[i] = S.sz[i];
      // the fill pass adds the row terms of the approximate old cost
      const long long si = S.sz[i];
      const long long internal = Q.internal[S.q[i]];
      old_out[i] = internal > 0 ? EncodeCostForPair(S.q[i], si, S.q[i], si, 2 * internal) : 0;
      // the fill pass adds the row's entries
      if (P.rc) StoreRowSums(&P.rc[S.q[i]], 0, 0, HeavyAcc(), internal, S.sz[i], S.len[i]);
    }
    if (tid == 0) V.eoff[g] = E;
    if (!P.mat_zeroed) {
      for (long long k = tid; k < gg; k += kPrepThreads) {
        pmat[k] = 0;
        fmat[k] = 0;
      }
    }
    if (tid == 0) {
      desc->base = dbase;
      desc->E = E;
      atomicAdd(&P.stats[kStGroupCount], 1ull);
      atomicMax(&P.stats[kStGroupMaxSize], static_cast<unsigned long long>(g));
      atomicAdd(&P.stats[kStRawPairCount], static_cast<unsigned long long>(g) * (g - 1) / 2);
      atomicAdd(&P.stats[kStPrepareBytes], 12ull * static_cast<unsigned long long>(E));
    }
    return;
  }
  if (E > kSmemEntries) {
    if (tid == 0) {
      RaiseError(P.err, kErrSlots, gid, E, 0);
      P.cand_cnt[ri] = 0;
    }
    return;
  }
  // bucket table in shared memory
  int* heads = S.heads;
  int* et = S.et;
  int* ei = S.ei;
  unsigned* ee = S.ee;
  int* enx = S.enx;
  const unsigned hmask = kSmemHeads - 1;
  for (unsigned h = tid; h <= hmask; h += kPrepThreads) heads[h] = -1;
  // per-group tables: proxy int64[g*g] | kept flag u8[g*g] | old cost int64[g]
  if (!P.mat_zeroed) {
    for (long long k = tid; k < gg; k += kPrepThreads) {
      pmat[k] = 0;
      fmat[k] = 0;
    }
  }
  __syncthreads();
  // entries, approximate old costs and direct in-group edges
  for (int i = warp; i < g; i += nwarps) {
    const int rep = S.q[i];
    const long long si = S.sz[i];
    const Entry* row = Q.ent + S.off[i];
    const int len = S.len[i];
    const int eo = S.eoff[i];
    long long old = 0, light = 0;
    HeavyAcc heavy;
    for (int k = lane; k < len; k += 32) {
      const Entry e = row[k];
      const int t = EntNb(e);
      const long long c = EntCnt(e);
      const long long st = Q.size[t];
      old += EncodeCostForPair(rep, si, t, st, c);
      if (HeavyEntry(si, st, c)) heavy.Add(st, c); else light += c;
      et[eo + k] = t;
      ei[eo + k] = i;
      ee[eo + k] = static_cast<unsigned>(c);
      enx[eo + k] = atomicExch(&heads[BucketHash(t, hmask)], eo + k);
      if (P.group_of[t] == gid) AddDirect(pmat, g, i, P.idx_in_group[t], c);
    }
    old = WarpSum(old);
    if (P.rc) {
      light = WarpSum(light);
      heavy.WarpReduce();
    }
    if (lane == 0) {
      const long long internal = Q.internal[rep];
      if (P.rc) StoreRowSums(&P.rc[rep], old, light, heavy, internal, S.sz[i], len);
      if (internal > 0) old += EncodeCostForPair(rep, si, rep, si, 2 * internal);
      S.old[i] = old;
    }
  }
  __syncthreads();
  // every two members sharing a target: proxy += max(0, old - new)
  unsigned long long examined = 0;
  for (int idx = tid; idx < E; idx += kPrepThreads) {
    const int t = et[idx];
    const int i = ei[idx];
    const long long c = ee[idx];
    long long st = -1;
    for (int k = enx[idx]; k != -1; k = enx[k]) {
      if (et[k] != t) continue;
      if (st < 0) st = Q.size[t];
      const int j = ei[k];
      ++examined;
      AddShared(pmat, g, i, j, S.sz[i], S.sz[j], st, c, static_cast<long long>(ee[k]), P.rc != nullptr);
    }
  }
  examined = WarpSum(static_cast<long long>(examined));
  if (lane == 0 && examined) atomicAdd(&S.examined, examined);
  __syncthreads();
  // old costs for the member pass, counters of the group
  long long* old_out = reinterpret_cast<long long*>(mat + OldCostOffset(gg));
  for (int i = tid; i < g; i += kPrepThreads) old_out[i] = S.old[i];
  if (tid == 0) {
    atomicAdd(&P.stats[kStGroupCount], 1ull);
    atomicMax(&P.stats[kStGroupMaxSize], static_cast<unsigned long long>(g));
    atomicAdd(&P.stats[kStRawPairCount], static_cast<unsigned long long>(g) * (g - 1) / 2);
    atomicAdd(&P.stats[kStProxyExamined], S.examined);
    // algorithmic bytes: member rows (8 B/entry) + target size gathers (4 B/entry)
    atomicAdd(&P.stats[kStPrepareBytes], 12ull * static_cast<unsigned long long>(E));
  }
}

// Fill pass of the deferred groups: one thread per sort slot of the launch
// (the groups' slot ranges, soff, laid end to end), CTAs striding over windows
// of kFillWindow slots, so the grid follows the total row entries and a hub
// member's long row is spread over many warps. A window's first group is
// found by a binary search of soff; each lane walks forward from it, and
// finds its member by a binary search of the group's row offsets (entries of
// one member are contiguous). Per entry: its sort key (launch-local group
// index, target) and value (member, count), the entry's approximate-old-cost
// term (summed per member run by a segmented warp scan, one atomic per run),
// and direct in-group edges, which go to both halves of the pair table (row i
// holds j and row j holds i with the same count), so no mirror pass is
// needed. Slots past a group's entries keep the padding key.
constexpr int kFillThreads = 256;
constexpr int kFillWindow = 2048;
constexpr int kAccumThreads = 256;

__global__ void __launch_bounds__(kFillThreads) PrepareFillKernel(PrepareParams P) {
  FollowsOn();
  __shared__ int first_group;
  const int lane = threadIdx.x & 31;
  const QuotientView& Q = P.Q;
  const long long windows = (P.nslots + kFillWindow - 1) / kFillWindow;
  for (long long w = blockIdx.x; w < windows; w += gridDim.x) {
    const long long w0 = w * kFillWindow;
    if (threadIdx.x == 0) {
      int lo = 0, hi = P.nlist;  // last group whose slot range starts at or before w0
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.soff[P.list0 + mid] - P.slot0 <= w0) lo = mid; else hi = mid;
      }
      first_group = lo;
    }
    __syncthreads();
    int k = first_group;
    int i = -1;  // member of the previous slot (same group), -1 none
    for (int off = threadIdx.x; off < kFillWindow; off += kFillThreads) {
      const long long s = w0 + off;
      long long run = -1;  // (group, member) of this lane's entry, -1 none
      long long cost = 0, light = 0;
      int rep = -1;
      HeavyAcc heavy;
      if (s < P.nslots) {
        const int k0 = k;
        while (k + 1 < P.nlist && P.soff[P.list0 + k + 1] - P.slot0 <= s) ++k;
        if (k != k0) i = -1;
        const BigDesc d = P.desc[P.list0 + k];
        const long long idx = s - (P.soff[P.list0 + k] - P.slot0);
        if (d.base != nullptr && idx < d.E) {
          const int ri = P.list[P.list0 + k];
          const int gid = P.real[ri];
          const int g = P.glen[gid];
          const DeferredView V = Deferred(d.base, g);
          if (i < 0 || idx >= V.eoff[i + 1] || idx < V.eoff[i]) {
            int lo = 0, hi = g;  // last member with eoff <= idx
            while (hi - lo > 1) {
              const int mid = (lo + hi) >> 1;
              if (V.eoff[mid] <= idx) lo = mid; else hi = mid;
            }
            i = lo;
          }
          rep = V.mq[i];
          const int e0 = V.eoff[i];
          const Entry e = Q.ent[Q.off[rep] + (idx - e0)];
          const int t = EntNb(e);
          const long long c = EntCnt(e);
          const long long st = Q.size[t];
          cost = EncodeCostForPair(rep, V.msz[i], t, st, c);
          if (P.rc) {
            if (HeavyEntry(V.msz[i], st, c)) heavy.Add(st, c); else light = c;
          }
          const long long slot = P.soff[P.list0 + k] - P.slot0 + idx;
          P.skey[slot] = P.bits.Key(k, t);
          P.sval[slot] = static_cast<unsigned long long>(i) << 32 | static_cast<unsigned long long>(c);
          if (P.group_of[t] == gid) {
            AddDirect(reinterpret_cast<unsigned long long*>(P.mat + P.mat_off[ri]), g, i, P.idx_in_group[t], c);
          }
          run = (static_cast<long long>(k) << 11) | i;
        }
      }
      // segmented inclusive scan over runs of equal (group, member)
      for (int o = 1; o < 32; o <<= 1) {
        const long long vc = __shfl_up_sync(0xffffffffu, cost, o);
        const long long vl = __shfl_up_sync(0xffffffffu, light, o);
        const long long vr = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o && vr == run) {
          cost += vc;
          light += vl;
        }
      }
      const long long next_run = __shfl_down_sync(0xffffffffu, run, 1);
      if (run >= 0 && (lane == 31 || next_run != run)) {
        const int ri = P.list[P.list0 + k];
        const int g = P.glen[P.real[ri]];
        unsigned long long* old_out =
            reinterpret_cast<unsigned long long*>(P.mat + P.mat_off[ri] + OldCostOffset(static_cast<long long>(g) * g));
        if (cost != 0) atomicAdd(&old_out[i], static_cast<unsigned long long>(cost));
        if (P.rc) {
          if (cost != 0) atomicAdd(reinterpret_cast<unsigned long long*>(&P.rc[rep].before), static_cast<unsigned long long>(cost));
          if (light != 0) atomicAdd(reinterpret_cast<unsigned long long*>(&P.rc[rep].light), static_cast<unsigned long long>(light));
        }
      }
      // heavy entries: the run's lanes by segmented scans too, where there are any
      if (__any_sync(0xffffffffu, heavy.n != 0)) {
        for (int o = 1; o < 32; o <<= 1) {
          const long long vr = __shfl_up_sync(0xffffffffu, run, o);
          HeavyAcc v;
          v.sx = __shfl_up_sync(0xffffffffu, heavy.sx, o);
          v.c = __shfl_up_sync(0xffffffffu, heavy.c, o);
          v.smin = __shfl_up_sync(0xffffffffu, heavy.smin, o);
          v.smax = __shfl_up_sync(0xffffffffu, heavy.smax, o);
          v.sbad = __shfl_up_sync(0xffffffffu, heavy.sbad, o);
          v.n = __shfl_up_sync(0xffffffffu, heavy.n, o);
          if (lane >= o && vr == run) heavy.Merge(v);
        }
        if (run >= 0 && (lane == 31 || next_run != run) && heavy.n != 0) {
          RowSums* r = &P.rc[rep];
          atomicAdd(reinterpret_cast<unsigned long long*>(&r->heavy_sx), static_cast<unsigned long long>(heavy.sx));
          atomicAdd(reinterpret_cast<unsigned long long*>(&r->heavy_c), static_cast<unsigned long long>(heavy.c));
          atomicMin(&r->smin, heavy.smin);
          atomicMax(&r->smax, heavy.smax);
          atomicMax(&r->sbad, heavy.sbad);
          atomicAdd(&r->nheavy, heavy.n);
        }
      }
    }
    __syncthreads();  // first_group is rewritten by the next window
  }
}

// Accumulate pass of the deferred groups over the sorted slots, a warp per
// 32 consecutive slots. The entries of one (group, target) are a contiguous
// run; each lane pairs its entry with the earlier entries of its run: those
// in its own chunk by shuffles, and, for the run that reaches back past the
// chunk's start, those of the earlier chunks, 32 at a time. Every member pair
// sharing a target is visited once and added to the pair's words (AddShared).
struct RunEntry {
  unsigned long long key;
  long long c;  // edge count to the target
  int i, s;     // member index, member size
};

__device__ __forceinline__ RunEntry LoadRunEntry(const PrepareParams& P, long long p, const DeferredView& V) {
  RunEntry r;
  const unsigned long long v = P.sval_sorted[p];
  r.i = static_cast<int>(v >> 32);
  r.c = static_cast<long long>(v & 0xffffffffu);
  r.s = V.msz[r.i];
  return r;
}

__device__ __forceinline__ RunEntry ShflRunEntry(const RunEntry& r, int src) {
  RunEntry o;
  o.key = __shfl_sync(0xffffffffu, r.key, src);
  o.c = __shfl_sync(0xffffffffu, r.c, src);
  o.s = __shfl_sync(0xffffffffu, r.s, src);
  o.i = __shfl_sync(0xffffffffu, r.i, src);
  return o;
}

// kAccumSplit warps share a chunk: warp y pairs the chunk with the earlier
// chunks y + 1, y + 1 + kAccumSplit, ... of its run (warp 0 also within the
// chunk), so a chunk deep in a long run is not one warp's long loop.
constexpr int kAccumSplit = 4;
// Work items are fetched from a queue, kAccumFetch at a time: a run over a
// hub target makes some chunks far longer than others, so a static stride
// leaves most warps idle behind a few. A fetch unit is one y of kAccumFetch
// chunks spread over the whole slot range (chunk g, g + G, g + 2G, ... with G
// fetch groups), so the consecutive chunks of one long run land on different
// warps, and so do the split warps of one chunk.
constexpr int kAccumFetch = 8;

__global__ void __launch_bounds__(kAccumThreads, 6) PrepareAccumKernel(PrepareParams P) {
  FollowsOn();
  const int lane = threadIdx.x & 31;
  unsigned long long examined = 0;
  const bool counted = P.rc != nullptr;
  const long long nchunks = (P.nslots + 31) >> 5;
  const long long ngroups8 = (nchunks + kAccumFetch - 1) / kAccumFetch;
  const long long nfetch = ngroups8 * kAccumSplit;
  long long fetched = -1, left = 0;
  for (;;) {
    if (left == 0) {
      long long f = 0;
      if (lane == 0) f = static_cast<long long>(atomicAdd(&P.ctl->work_next[0], 1ull));
      fetched = __shfl_sync(0xffffffffu, f, 0);
      if (fetched >= nfetch) break;
      left = kAccumFetch;
    }
    --left;
    // fetch unit u = (chunk group g, y): chunks g + k * ngroups8, k < kAccumFetch
    const int y = static_cast<int>(fetched % kAccumSplit);
    const long long ch = (fetched / kAccumSplit) + (kAccumFetch - 1 - left) * ngroups8;
    if (ch >= nchunks) continue;
    const long long p0 = ch << 5;
    if (y > 0) {
      // nothing unless the chunk's first run reaches back at least y + 1 chunks
      if (p0 < 32ll * (y + 1)) continue;
      const unsigned long long f = P.skey_sorted[p0];
      if (f == kSlotPad || P.skey_sorted[p0 - 32ll * y - 1] != f) continue;
    }
    const long long p = p0 + lane;
    RunEntry me;
    me.key = p < P.nslots ? P.skey_sorted[p] : kSlotPad;
    me.c = 0;
    me.s = me.i = 0;
    const bool valid = me.key != kSlotPad;
    int g = 0;
    long long st = 0;
    unsigned long long* pmat = nullptr;
    if (valid) {
      const int bl = P.bits.Group(me.key);
      const int t = P.bits.Target(me.key);
      const int ri = P.list[P.list0 + bl];
      g = P.glen[P.real[ri]];
      pmat = reinterpret_cast<unsigned long long*>(P.mat + P.mat_off[ri]);
      const RunEntry r = LoadRunEntry(P, p, Deferred(P.desc[P.list0 + bl].base, g));
      me.c = r.c;
      me.s = r.s;
      me.i = r.i;
      st = P.Q.size[t];
    }
    // pairs inside the chunk: each lane visits the earlier lanes holding its
    // key, one per round (a chunk whose targets are all distinct, the common
    // case, takes no round)
    if (y == 0) {
      unsigned earlier = __match_any_sync(0xffffffffu, me.key) & ((1u << lane) - 1u);
      if (!valid) earlier = 0u;
      const int rounds = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(__popc(earlier))));
      for (int r = 0; r < rounds; ++r) {
        const int src = earlier != 0u ? __ffs(earlier) - 1 : lane;
        const RunEntry o = ShflRunEntry(me, src);
        if (earlier != 0u) {
          ++examined;
          AddShared(pmat, g, me.i, o.i, me.s, o.s, st, me.c, o.c, counted);
          earlier &= earlier - 1u;
        }
      }
    }
    // the run holding the chunk's first slot may start in earlier chunks
    const unsigned long long first = __shfl_sync(0xffffffffu, me.key, 0);
    if (first == kSlotPad || p0 == 0 || P.skey_sorted[p0 - 1] != first) continue;
    const int fbl = P.bits.Group(first);
    const int fg = P.glen[P.real[P.list[P.list0 + fbl]]];
    const DeferredView FV = Deferred(P.desc[P.list0 + fbl].base, fg);
    const bool mine = valid && me.key == first;
    for (long long c0 = p0 - 32ll * (y + 1);; c0 -= 32ll * kAccumSplit) {
      // c0 >= 0; the chunk holds run entries iff its last slot is in the run
      if (P.skey_sorted[c0 + 31] != first) break;
      RunEntry o;
      o.key = P.skey_sorted[c0 + lane];
      o.c = 0;
      o.s = o.i = 0;
      if (o.key == first) o = [&] { RunEntry r = LoadRunEntry(P, c0 + lane, FV); r.key = first; return r; }();
      for (int src = 0; src < 32; ++src) {
        const RunEntry b = ShflRunEntry(o, src);
        if (mine && b.key == first) {
          ++examined;
          AddShared(pmat, g, me.i, b.i, me.s, b.s, st, me.c, b.c, counted);
        }
      }
      // the run continues below this chunk iff its first slot is in the run
      if (c0 < 32ll * kAccumSplit || __shfl_sync(0xffffffffu, o.key, 0) != first) break;
    }
  }
  examined = static_cast<unsigned long long>(WarpSum(static_cast<long long>(examined)));
  if (lane == 0 && examined) atomicAdd(&P.stats[kStProxyExamined], examined);
}

// Top-k partners of member i of a big group whose partners fill NT slots of
// 32 (the fp32 prescreen branch of PrepareMembersKernel).
template <int NT, typename ProxyFn, typename KeepFn>
__device__ __forceinline__ void MembersTopK(int lane, int g, int i, int qi, int top_k, int cnt,
                                            ProxyFn proxy, const long long* old, long long old_i, const int* q, int* cj,
                                            KeepFn keep) {
  auto ratio_of = [&](int j, long long pg) {
    long long denom = old_i + old[j];
    if (denom < 1) denom = 1;
    return static_cast<unsigned long long>(
        __double_as_longlong(static_cast<double>(pg) / static_cast<double>(denom)));
  };
  // fp32 prescreen: the exact (double) ratio is only computed for the
  // candidates that can be in the member's top_k. The fp32 ratio of a
  // candidate is within relative 3 * 2^-24 of its double ratio, so every
  // candidate of the exact top_k has an fp32 ratio >= tau * (1 - 2^-20),
  // where tau is the top_k-th largest fp32 ratio (bounded by bisection on the
  // float bit patterns, which order like the positive values).
  float rf[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int j = lane + 32 * t;
    float v = 0.0f;  // not a candidate
    if (j < g && j != i) {
      const long long pg = proxy(i, j);
      if (pg > 0) {
        long long denom = old_i + old[j];
        if (denom < 1) denom = 1;
        v = __fdiv_rn(static_cast<float>(pg), static_cast<float>(denom));
      }
    }
    rf[t] = v;
  }
  float cut = 0.0f;
  if (cnt > top_k + 16) {
    // count(bits >= lo) >= top_k > count(bits >= hi), starting from the
    // smallest and one past the largest positive ratio (the cnt candidates)
    unsigned lo = 0x7f800000u, hi = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const unsigned b = __float_as_uint(rf[t]);
      if (rf[t] > 0.0f) {
        lo = b < lo ? b : lo;
        hi = b > hi ? b : hi;
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi) + 1u;
    // (any lo with a lane's worth of candidates left will do: a few steps
    // instead of the two dozen that single out tau)
    int left = cnt;
    while (hi - lo > 1 && left > 30) {
      const unsigned mid = lo + ((hi - lo) >> 1);
      int c = 0;
#pragma unroll
      for (int t = 0; t < NT; ++t) c += __float_as_uint(rf[t]) >= mid ? 1 : 0;
      c = WarpSumInt(c);
      if (c >= top_k) {
        lo = mid;
        left = c;
      } else {
        hi = mid;
      }
    }
    cut = __uint_as_float(lo) * (1.0f - 9.5367431640625e-7f);
  }
  int npass = 0;
#pragma unroll
  for (int t = 0; t < NT; ++t) npass += (rf[t] > 0.0f && rf[t] >= cut) ? 1 : 0;
  npass = WarpSumInt(npass);
  if (npass <= 32) {
    // one surviving candidate per lane; its rank is the number of
    // candidates better than it under the strict order, and the top_k
    // ranks are kept
    int base = 0;
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const bool pass = rf[t] > 0.0f && rf[t] >= cut;
      const unsigned ball = __ballot_sync(0xffffffffu, pass);
      if (pass) cj[base + __popc(ball & ((1u << lane) - 1u))] = lane + 32 * t;
      base += __popc(ball);
    }
    __syncwarp();
    const bool have = lane < npass;
    RankKey mine;
    mine.rb = 0;
    mine.pg = 0;
    mine.lo = 0;
    mine.hi = 0;
    mine.j = -1;
    long long denom = 1;
    if (have) {
      const int j = cj[lane];
      const long long pg = proxy(i, j);
      const int qj = q[j];
      denom = old_i + old[j];
      if (denom < 1) denom = 1;
      mine.j = j;
      mine.pg = pg;
      mine.lo = qi < qj ? qi : qj;
      mine.hi = qi < qj ? qj : qi;
    }
    int rank = 0;
    if (!__any_sync(0xffffffffu, mine.pg >= kExactRatio || denom >= kExactRatio)) {
      const RankCand c[1] = {{static_cast<unsigned>(mine.pg), static_cast<unsigned>(denom),
                              have ? q[mine.j] : 0}};
      int r[1];
      ExactRanks(c, r);
      rank = r[0];
    } else {
      if (have) mine.rb = ratio_of(mine.j, mine.pg);
      for (int o = 0; o < npass; ++o) {
        RankKey other;
        other.rb = __shfl_sync(0xffffffffu, mine.rb, o);
        other.pg = __shfl_sync(0xffffffffu, mine.pg, o);
        other.lo = __shfl_sync(0xffffffffu, mine.lo, o);
        other.hi = __shfl_sync(0xffffffffu, mine.hi, o);
        if (have && o != lane && Better(other, mine)) ++rank;
      }
    }
    if (have && rank < top_k) {
      const int a = i < mine.j ? i : mine.j;
      const int b = i < mine.j ? mine.j : i;
      keep(a, b);
    }
  } else {
    // each lane keeps its best top_k candidates sorted, then the warp merges
    // the 32 lists head by head (candidates are distinct, so no key ties)
    RankKey lst[kLaneTopK];
    int nl = 0;
  #pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int j = lane + 32 * t;
      if (rf[t] <= 0.0f || rf[t] < cut) continue;
      const long long pg = proxy(i, j);
      RankKey k;
      k.j = j;
      k.rb = ratio_of(j, pg);
      k.pg = pg;
      const int qj = q[j];
      k.lo = qi < qj ? qi : qj;
      k.hi = qi < qj ? qj : qi;
      if (nl == top_k && !Better(k, lst[nl - 1])) continue;
      int pos = nl < top_k ? nl : top_k - 1;
      while (pos > 0 && Better(k, lst[pos - 1])) {
        lst[pos] = lst[pos - 1];
        --pos;
      }
      lst[pos] = k;
      if (nl < top_k) ++nl;
    }
    int head = 0;
    for (int r = 0; r < top_k; ++r) {
      RankKey best;
      bool have = head < nl;
      if (have) best = lst[head];
      int src = lane;
      for (int o = 16; o > 0; o >>= 1) {
        RankKey other;
        other.rb = __shfl_xor_sync(0xffffffffu, best.rb, o);
        other.pg = __shfl_xor_sync(0xffffffffu, best.pg, o);
        other.lo = __shfl_xor_sync(0xffffffffu, best.lo, o);
        other.hi = __shfl_xor_sync(0xffffffffu, best.hi, o);
        other.j = __shfl_xor_sync(0xffffffffu, best.j, o);
        const int osrc = __shfl_xor_sync(0xffffffffu, src, o);
        const int ohave = __shfl_xor_sync(0xffffffffu, have ? 1 : 0, o);
        if (ohave && (!have || Better(other, best))) {
          best = other;
          have = true;
          src = osrc;
        }
      }
      if (!have) break;
      if (src == lane) ++head;
      if (lane == 0) {
        const int a = i < best.j ? i : best.j;
        const int b = i < best.j ? best.j : i;
        keep(a, b);
      }
    }
  }
}

// Member i of a group (members q, old costs, proxy(i, j)) by one warp: keep(a, b) is called for the pair of each of its top_k partners, by
// some lane. cj: 32 words of the warp's own.
template <typename ProxyFn, typename KeepFn>
__device__ __forceinline__ void RankMember(int g, int i, const int* q, const long long* old, int top_k_max, int* cj,
                                           ProxyFn proxy, KeepFn keep) {
  const int lane = threadIdx.x & 31;
  // candidates with positive proxy, ratio, top-k (the ratio is recomputed where
  // it is needed instead of being stored)
  int top_k = top_k_max < g - 1 ? top_k_max : g - 1;
  if (top_k < 1) top_k = 1;
  const long long old_i = old[i];
  auto ratio_of = [&](int j, long long pg) {
    long long denom = old_i + old[j];
    if (denom < 1) denom = 1;
    return static_cast<unsigned long long>(
        __double_as_longlong(static_cast<double>(pg) / static_cast<double>(denom)));
  };
  int cnt = 0;
  for (int base = 0; base < g; base += 32) {
    const int j = base + lane;
    const bool pred = j < g && j != i && proxy(i, j) > 0;
    cnt += __popc(__ballot_sync(0xffffffffu, pred));
  }
  const int qi = q[i];
  if (cnt <= top_k) {
    for (int j = lane; j < g; j += 32) {
      if (j == i || proxy(i, j) <= 0) continue;
      const int a = i < j ? i : j;
      const int b = i < j ? j : i;
      keep(a, b);
    }
  } else if (top_k <= kLaneTopK) {
    const int nt = (g + 31) >> 5;
    if (nt <= 1) {
      MembersTopK<1>(lane, g, i, qi, top_k, cnt, proxy, old, old_i, q, cj, keep);
    } else if (nt <= 2) {
      MembersTopK<2>(lane, g, i, qi, top_k, cnt, proxy, old, old_i, q, cj, keep);
    } else if (nt <= 4) {
      MembersTopK<4>(lane, g, i, qi, top_k, cnt, proxy, old, old_i, q, cj, keep);
    } else if (nt <= 8) {
      MembersTopK<8>(lane, g, i, qi, top_k, cnt, proxy, old, old_i, q, cj, keep);
    } else {
      MembersTopK<kMaxGroup / 32>(lane, g, i, qi, top_k, cnt, proxy, old, old_i, q, cj, keep);
    }
  } else {
    RankKey prev;
    bool have_prev = false;
    for (int r = 0; r < top_k; ++r) {
      RankKey best;
      bool have = false;
      for (int j = lane; j < g; j += 32) {
        if (j == i) continue;
        const long long pg = proxy(i, j);
        if (pg <= 0) continue;
        RankKey k;
        k.j = j;
        k.rb = ratio_of(j, pg);
        k.pg = pg;
        const int qj = q[j];
        k.lo = qi < qj ? qi : qj;
        k.hi = qi < qj ? qj : qi;
        if (have_prev && !Better(prev, k)) continue;
        if (!have || Better(k, best)) {
          best = k;
          have = true;
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        RankKey other;
        other.rb = __shfl_xor_sync(0xffffffffu, best.rb, o);
        other.pg = __shfl_xor_sync(0xffffffffu, best.pg, o);
        other.lo = __shfl_xor_sync(0xffffffffu, best.lo, o);
        other.hi = __shfl_xor_sync(0xffffffffu, best.hi, o);
        other.j = __shfl_xor_sync(0xffffffffu, best.j, o);
        const int ohave = __shfl_xor_sync(0xffffffffu, have ? 1 : 0, o);
        if (ohave && (!have || Better(other, best))) {
          best = other;
          have = true;
        }
      }
      if (!have) break;
      if (lane == 0) {
        const int a = i < best.j ? i : best.j;
        const int b = i < best.j ? best.j : i;
        keep(a, b);
      }
      prev = best;
      have_prev = true;
    }
  }
}

// Member pass of the big groups: one warp per member of every group in the
// launch's big-group list (moff = prefix of the member counts), so a large
// group's members are ranked by the whole GPU instead of one CTA.
__global__ void __launch_bounds__(256) PrepareMembersKernel(PrepareParams P) {
  FollowsOn();
  __shared__ int cand_j[8][32];  // per warp: the candidates that survive the prescreen
  const long long wg = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long total = P.moff[P.list0 + P.nlist] - P.moff[P.list0];
  if (wg >= total) return;
  const long long target = P.moff[P.list0] + wg;
  const int lo = WarpLastLE(P.moff, P.list0, P.list0 + P.nlist, target);  // last entry with moff <= target
  const int ri = P.list[lo];
  const int i = static_cast<int>(target - P.moff[lo]);
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  const int* q = P.order + P.gstart[gid];
  unsigned char* fmat = P.mat + P.mat_off[ri] + FlagOffset(static_cast<long long>(g) * g);
  const unsigned long long* pmat = reinterpret_cast<const unsigned long long*>(P.mat + P.mat_off[ri]);
  const long long* old =
      reinterpret_cast<const long long*>(P.mat + P.mat_off[ri] + OldCostOffset(static_cast<long long>(g) * g));
  RankMember(g, i, q, old, P.top_k, cand_j[threadIdx.x >> 5],
                        [&](int x, int j) { return ProxyOf(PairWord(pmat, g, x, j)); },
                        [&](int a, int b) { fmat[static_cast<long long>(a) * g + b] = 1; });
}

// Flag bytes (0 or 1) of table word w that lie in [beg, end), as a bit set
// with one bit per set flag (bit 8k for byte k).
__device__ __forceinline__ unsigned long long RowFlagBits(const unsigned long long* fw, long long w, long long beg,
                                                          long long end) {
  const long long lo = beg - w * 8;  // first byte of the range in this word
  const long long hi = end - w * 8;  // one past the last
  unsigned long long m = 0x0101010101010101ull;
  if (lo > 0) m &= ~0ull << (8 * lo);
  if (hi < 8) m &= (1ull << (8 * hi)) - 1ull;
  return fw[w] & m;
}

// The shared part of pair (a, b) from its two words.
__device__ __forceinline__ PairInfo PairInfoOf(const QuotientView& Q, int a, int b, unsigned long long word,
                                               long long corr) {
  PairInfo p;
  p.ovl = static_cast<unsigned>((word >> kProxyBits) & kOvlMask);
  p.eab = 0;
  if (word & (kRowILists | kRowJLists)) {
    const long long ea = RowLookup(Q.ent + Q.off[a], Q.len[a], b);
    const long long eb = RowLookup(Q.ent + Q.off[b], Q.len[b], a);
    if (ea != eb) p.ovl |= kPairAsym;
    p.eab = static_cast<unsigned>(ea);
  }
  if (corr >= kCorrBad / 2 || corr <= -kCorrBad / 2) p.ovl |= kPairBad;
  // the proxy holds the direct edges as listed by row a
  p.shared = corr - (ProxyOf(word) - static_cast<long long>(p.eab));
  return p;
}

// Output pass of the big groups: the union of kept pairs in (a_idx, b_idx)
// order, one CTA per group.
__global__ void __launch_bounds__(kPrepThreads) PrepareOutputKernel(PrepareParams P) {
  FollowsOn();
  using BlockScan = cub::BlockScan<int, kPrepThreads>;
  __shared__ typename BlockScan::TempStorage scan_tmp;
  __shared__ int carry;
  __shared__ int eoff[kMaxGroup + 1];
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nwarps = kPrepThreads / 32;
  const int ri = P.list[P.list0 + blockIdx.x];
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  const long long gg = static_cast<long long>(g) * g;
  const unsigned char* fmat = P.mat + P.mat_off[ri] + FlagOffset(gg);
  const unsigned long long* pmat = reinterpret_cast<const unsigned long long*>(P.mat + P.mat_off[ri]);
  const long long* old = reinterpret_cast<const long long*>(P.mat + P.mat_off[ri] + OldCostOffset(gg));
  const int* q = P.order + P.gstart[gid];
  // union of kept pairs in (a_idx, b_idx) order. The flags of row a,
  // bytes [a*g + a + 1, a*g + g) of the table, are read as 8-byte words
  // (the table starts 8-byte aligned; the masked bytes past its end lie in
  // the group's old-cost array).
  const unsigned long long* fw = reinterpret_cast<const unsigned long long*>(fmat);
  for (int a = warp; a < g; a += nwarps) {
    const long long beg = static_cast<long long>(a) * g + a + 1;
    const long long end = static_cast<long long>(a) * g + g;
    int cnt = 0;
    for (long long w = (beg >> 3) + lane; w < (end + 7) >> 3; w += 32) cnt += __popcll(RowFlagBits(fw, w, beg, end));
    cnt = WarpSumInt(cnt);
    if (lane == 0) eoff[a] = cnt;
  }
  __syncthreads();
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < g; base += kPrepThreads) {
    const int i = base + tid;
    const int v = i < g ? eoff[i] : 0;
    int ex = 0, agg = 0;
    BlockScan(scan_tmp).ExclusiveSum(v, ex, agg);
    __syncthreads();
    if (i < g) eoff[i] = carry + ex;
    __syncthreads();
    if (tid == 0) carry += agg;
    __syncthreads();
  }
  const int nc = carry;
  int2* out = P.cand + P.cand_off[ri];
  for (int a = warp; a < g; a += nwarps) {
    const long long beg = static_cast<long long>(a) * g + a + 1;
    const long long end = static_cast<long long>(a) * g + g;
    const long long row0 = static_cast<long long>(a) * g;
    int pos = eoff[a];
    for (long long w0 = beg >> 3; w0 < (end + 7) >> 3; w0 += 32) {
      const long long w = w0 + lane;
      unsigned long long bits = w < (end + 7) >> 3 ? RowFlagBits(fw, w, beg, end) : 0ull;
      const int c = __popcll(bits);
      int incl = c;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      long long at = pos + incl - c;
      while (bits) {
        const int k = (__ffsll(static_cast<long long>(bits)) - 1) >> 3;
        bits &= bits - 1;
        const int b = static_cast<int>(w * 8 + k - row0);
        out[at] = make_int2(a, b);
        P.cand_rep[P.cand_off[ri] + at] = make_int2(q[a], q[b]);
        const unsigned long long word = pmat[static_cast<long long>(a) * g + b];
        if (P.info) {
          P.info[P.cand_off[ri] + at] =
              PairInfoOf(P.Q, q[a], q[b], word, static_cast<long long>(pmat[static_cast<long long>(b) * g + a]));
        }
        if (P.cand_feat) {
          const long long pg = ProxyOf(word);
          long long denom = old[a] + old[b];
          if (denom < 1) denom = 1;
          // a ranker feature, not a decision: single precision is enough
          P.cand_feat[P.cand_off[ri] + at] =
              make_float2(static_cast<float>(pg), __fdividef(static_cast<float>(pg), static_cast<float>(denom)));
        }
        ++at;
      }
      pos += __shfl_sync(0xffffffffu, incl, 31);
    }
  }
  if (tid == 0) {
    P.cand_cnt[ri] = nc;
    atomicAdd(&P.stats[kStCandAfterPrune], static_cast<unsigned long long>(nc));
  }
}

// ------------------------------------------------------------ prepare, small groups

// Groups of at most kSmallGroup members whose rows hold at most kSmallStage
// entries (99% of the real groups on R-MAT workloads): one warp per group, no
// block-wide barrier. The group's rows and their target sizes are staged in
// shared memory in one coalesced pass; the EA-proxy sum over targets shared by
// two members then equals, per member pair, the sum over the intersection of
// their two sorted rows (a row never holds its own rep, so the reference's
// own-rep exclusion is implied). One lane per staged entry looks its target up
// in the rows of the later members and adds what it finds to the pair's sums in
// shared memory: the lanes' work is even, where a lane per pair merging two
// rows made the group wait for its longest row. Output and counters equal
// those of PrepareKernel.
constexpr int kSmallGroup = 32;
constexpr int kSmallWarps = 4;
constexpr int kSmallPairs = kSmallGroup * (kSmallGroup - 1) / 2;
constexpr int kSmallStage = 256;  // staged row entries per group
// Sums are kept in 32 bits where the group's counts sum to less than this
// (every term is at most 4 counts); the other groups, and those with a count
// beyond its block's capacity, merge a pair's rows again whenever they need
// its sums.
constexpr long long kSmallNarrow = 1ll << 28;

struct SmallRowsSmem {
  long long old[kSmallGroup];
  long long off[kSmallGroup];
  Entry ent[kSmallStage];
  HeavyAcc heavy[kSmallGroup];
  int tsz[kSmallStage];
  unsigned light[kSmallGroup];
  unsigned char row[kSmallStage];  // member of the entry
  int q[kSmallGroup];
  int sz[kSmallGroup];
  int start[kSmallGroup + 1];
  unsigned fmask[kSmallGroup];
};

// Pair sums, upper triangle by TriIndex(a, b): proxy << 32 | corr, and the
// number of shared targets (at most kSmallStage / 2 of them: a byte each).
template <int kPairs>
struct SmallPairsSmem {
  unsigned long long pc[kPairs];
  unsigned ovl[(kPairs + 3) / 4];
};
static_assert(kSmallStage / 2 < 1 << 8, "two rows share at most half of the staged entries");

struct SmallWarpSmem {
  SmallRowsSmem rows;
  SmallPairsSmem<kSmallPairs> pairs;
};

struct SmallSmem {
  SmallWarpSmem w[kSmallWarps];
};

__device__ __forceinline__ int TriIndex(int a, int b, int g) { return a * (2 * g - a - 1) / 2 + (b - a - 1); }

// The pair at a position of the upper triangle.
__device__ __forceinline__ void TriPair(int pidx, int g, int* a, int* b) {
  int x = 0, rem = pidx;
  if (g > kSmallGroup) {
    // a is near the root of a * (2g - a - 1) / 2 = pidx
    const float d = (2.0f * g - 1.0f) * (2.0f * g - 1.0f) - 8.0f * static_cast<float>(pidx);
    x = static_cast<int>((2.0f * g - 1.0f - sqrtf(d > 0.0f ? d : 0.0f)) * 0.5f);
    x = x < 0 ? 0 : x > g - 2 ? g - 2 : x;
    while (x > 0 && TriIndex(x, x + 1, g) > pidx) --x;
    rem = pidx - TriIndex(x, x + 1, g);
  }
  while (rem >= g - 1 - x) {
    rem -= g - 1 - x;
    ++x;
  }
  *a = x;
  *b = x + 1 + rem;
}

// Members a < b of a staged group by one lane.
struct SmallPair {
  long long proxy;  // EA proxy, direct edges included
  long long corr;   // as in the pair tables
  int ovl;
  bool bad;
};

template <typename Rows>
__device__ __forceinline__ SmallPair SmallMerge(const Rows& S, int a, int b) {
  const int qb = S.q[b];
  const long long sa = S.sz[a], sb = S.sz[b];
  int ia = S.start[a], ib = S.start[b];
  const int ea_end = S.start[a + 1], eb_end = S.start[b + 1];
  SmallPair r{0, 0, 0, false};
  while (ia < ea_end && ib < eb_end) {
    const Entry ea = S.ent[ia], eb = S.ent[ib];
    const int ta = EntNb(ea), tb = EntNb(eb);
    if (ta < tb) {
      if (ta == qb) r.proxy += EntCnt(ea);
      ++ia;
    } else if (tb < ta) {
      ++ib;
    } else {
      bool bad;
      const SharedTerm t = TermOf(sa, sb, S.tsz[ia], EntCnt(ea), EntCnt(eb), &bad);
      r.proxy += t.delta;
      r.corr += t.corr;
      r.bad |= bad;
      ++r.ovl;
      ++ia;
      ++ib;
    }
  }
  for (; ia < ea_end; ++ia) {
    if (EntNb(S.ent[ia]) == qb) r.proxy += EntCnt(S.ent[ia]);
  }
  return r;
}

template <typename Rows>
__device__ __forceinline__ long long StagedLookup(const Rows& S, int a, int key) {
  return RowLookup(S.ent + S.start[a], S.start[a + 1] - S.start[a], key);
}

template <typename Rows>
__device__ __forceinline__ PairInfo SmallPairInfo(const Rows& S, int a, int b, const SmallPair& r) {
  const long long ea = StagedLookup(S, a, S.q[b]);
  const long long eb = StagedLookup(S, b, S.q[a]);
  PairInfo pi;
  pi.shared = r.corr - (r.proxy - ea);
  pi.ovl = static_cast<unsigned>(r.ovl) | (r.bad ? kPairBad : 0u) | (ea != eb ? kPairAsym : 0u);
  pi.eab = static_cast<unsigned>(ea);
  return pi;
}

// Stages a group's rows and their target sizes: one flat pass over the entries
// (independent loads), then the sizes. Returns the entries, nothing staged when
// they are more than kSmallStage (not by the plan: row entries counted at
// Divide time only shrink); wide: the group's counts reach kSmallNarrow.
__device__ __forceinline__ int StageSmallRows(const QuotientView& Q, const int* order, int g, SmallRowsSmem& S,
                                              bool* wide) {
  const int lane = threadIdx.x & 31;
  int len = 0;
  if (lane < g) {
    const int rep = order[lane];
    S.q[lane] = rep;
    S.sz[lane] = Q.size[rep];
    len = Q.len[rep];
    S.off[lane] = Q.off[rep];
    S.fmask[lane] = 0;
  }
  int incl = len;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int E = __shfl_sync(0xffffffffu, incl, 31);
  if (lane < g) S.start[lane] = incl - len;
  if (lane == 0) S.start[g] = E;
  *wide = false;
  if (E > kSmallStage) return E;
  __syncwarp();
  long long counts = 0;
#pragma unroll 4
  for (int k = lane; k < E; k += 32) {
    int lo = 0, hi = g;  // row of entry k: last i with start[i] <= k
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (S.start[mid] <= k) lo = mid; else hi = mid;
    }
    const Entry e = Q.ent[S.off[lo] + (k - S.start[lo])];
    S.ent[k] = e;
    S.row[k] = static_cast<unsigned char>(lo);
    counts += EntCnt(e);
  }
  __syncwarp();
#pragma unroll 4
  for (int k = lane; k < E; k += 32) S.tsz[k] = Q.size[EntNb(S.ent[k])];
  *wide = WarpSum(counts) >= kSmallNarrow;
  __syncwarp();
  return E;
}

// One entry (count c, target size st) into member i's sums, in the low words: the
// counts sum to less than kSmallNarrow. Old costs are signed there (a count
// beyond its block's capacity has a negative one, above -c) until SmallFinishRow.
template <typename Rows>
__device__ __forceinline__ void AddRowEntry(Rows& S, int i, long long c, long long st) {
  const long long si = S.sz[i];
  const long long alt = 1 + si * st - c;
  atomicAdd(reinterpret_cast<unsigned*>(&S.old[i]), static_cast<unsigned>(c < alt ? c : alt));
  if (HeavyEntry(si, st, c)) {
    HeavyAcc h;
    h.Add(st, c);
    HeavyAcc* a = &S.heavy[i];
    atomicAdd(reinterpret_cast<unsigned long long*>(&a->sx), static_cast<unsigned long long>(h.sx));
    atomicAdd(reinterpret_cast<unsigned long long*>(&a->c), static_cast<unsigned long long>(h.c));
    atomicMin(&a->smin, h.smin);
    atomicMax(&a->smax, h.smax);
    atomicMax(&a->sbad, h.sbad);
    atomicAdd(&a->n, 1);
  } else {
    atomicAdd(&S.light[i], static_cast<unsigned>(c));
  }
}

// Old cost and heavy sums of member i, by one thread (counts too large for
// AddRowEntry).
template <typename Rows>
__device__ __forceinline__ void WideRow(Rows& S, int i) {
  long long old = 0;
  for (int k = S.start[i]; k < S.start[i + 1]; ++k) {
    const long long c = EntCnt(S.ent[k]), st = S.tsz[k];
    old += EncodeCostForPair(S.q[i], S.sz[i], EntNb(S.ent[k]), st, c);
    if (HeavyEntry(S.sz[i], st, c)) S.heavy[i].Add(st, c);
  }
  S.old[i] = old;
}

// The staged group's row sums and pair sums, by a warp: S.old (with the
// internal term), S.light and S.heavy per member, and the pair sums. Returns
// the shared targets visited; *slow: the 32-bit sums do not hold, SmallMerge
// gives the pairs'.
template <int kPairs>
__device__ __forceinline__ unsigned SmallSums(const QuotientView& Q, SmallRowsSmem& S, SmallPairsSmem<kPairs>& T, int g,
                                              int E, bool wide, bool* slow) {
  const int lane = threadIdx.x & 31;
  const int npairs = g * (g - 1) / 2;
  for (int k = lane; k < npairs; k += 32) T.pc[k] = 0;
  for (int k = lane; k < (npairs + 3) / 4; k += 32) T.ovl[k] = 0;
  unsigned examined = 0;
  bool any_bad = false;
  if (lane < g) {
    S.heavy[lane] = HeavyAcc();
    S.old[lane] = 0;
    S.light[lane] = 0;
  }
  __syncwarp();
  if (!wide) {
    for (int k0 = 0; k0 < E; k0 += 32) {
      const int k = k0 + lane;
      if (k >= E) continue;
      const Entry e = S.ent[k];
      const int t = EntNb(e), i = S.row[k];
      const long long c = EntCnt(e), st = S.tsz[k], si = S.sz[i];
      AddRowEntry(S, i, c, st);
      for (int j = i + 1; j < g; ++j) {
        const int b = TriIndex(i, j, g);
        if (t == S.q[j]) {  // a row does not list itself: no search needed
          atomicAdd(reinterpret_cast<unsigned*>(&T.pc[b]) + 1, static_cast<unsigned>(c));
          continue;
        }
        int lo = S.start[j], hi = S.start[j + 1];
        const int end = hi;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (EntNb(S.ent[mid]) < t) lo = mid + 1; else hi = mid;
        }
        if (lo == end || EntNb(S.ent[lo]) != t) continue;
        bool bad;
        const SharedTerm x = TermOf(si, S.sz[j], st, c, EntCnt(S.ent[lo]), &bad);
        ++examined;
        any_bad |= bad;
        if (x.delta != 0) atomicAdd(reinterpret_cast<unsigned*>(&T.pc[b]) + 1, static_cast<unsigned>(x.delta));
        if (x.corr != 0) atomicAdd(reinterpret_cast<int*>(&T.pc[b]), static_cast<int>(x.corr));
        atomicAdd(&T.ovl[b >> 2], 1u << (8 * (b & 3)));
      }
    }
  }
  *slow = __any_sync(0xffffffffu, any_bad) || wide;
  __syncwarp();
  if (wide) {
    // too large for 32 bits: a lane per member, a lane per pair
    if (lane < g) WideRow(S, lane);
    for (int pidx = lane; pidx < npairs; pidx += 32) {
      int a, b;
      TriPair(pidx, g, &a, &b);
      examined += static_cast<unsigned>(SmallMerge(S, a, b).ovl);
    }
  }
  return examined;
}

// Member i's record and its old cost's internal term, by one lane.
template <typename Rows>
__device__ __forceinline__ void SmallFinishRow(const QuotientView& Q, Rows& S, int i, bool wide,
                                               RowSums* out) {
  const int rep = S.q[i];
  const long long si = S.sz[i];
  const long long internal = Q.internal[rep];
  if (!wide) S.old[i] = static_cast<int>(static_cast<unsigned>(S.old[i]));
  if (out) {
    long long light = S.light[i];
    if (wide) {
      for (int k = S.start[i]; k < S.start[i + 1]; ++k) {
        const long long c = EntCnt(S.ent[k]);
        if (!HeavyEntry(si, S.tsz[k], c)) light += c;
      }
    }
    StoreRowSums(out, S.old[i], light, S.heavy[i], internal, S.sz[i], S.start[i + 1] - S.start[i]);
  }
  if (internal > 0) S.old[i] += EncodeCostForPair(rep, si, rep, si, 2 * internal);
}

// Pair (a, b) at position t of the pair sums.
template <int kPairs>
__device__ __forceinline__ SmallPair SmallPairAt(const SmallRowsSmem& S, const SmallPairsSmem<kPairs>& T, int t, int a,
                                                 int b, bool slow) {
  if (slow) return SmallMerge(S, a, b);
  SmallPair r;
  r.proxy = static_cast<long long>(T.pc[t] >> 32);
  r.corr = static_cast<int>(T.pc[t] & 0xffffffffull);
  r.ovl = (T.ovl[t >> 2] >> (8 * (t & 3))) & 0xff;
  r.bad = false;
  return r;
}

// Sum of f_s(c) over staged row i, by one lane.
template <typename Rows>
__device__ __forceinline__ long long StagedRowAfter(const Rows& S, int i, long long s) {
  long long sum = 0;
  for (int k = S.start[i]; k < S.start[i + 1]; ++k) {
    const long long c = EntCnt(S.ent[k]);
    const long long alt = 1 + s * S.tsz[k] - c;
    sum += c < alt ? c : alt;
  }
  return sum;
}

// Marks every member's top_k partners in fmask (bit b of word a, a < b), by a
// warp; proxy_of(a, b), a < b.
template <typename ProxyFn>
__device__ __forceinline__ void SmallTopK(SmallRowsSmem& S, int g, int top_k_max, ProxyFn proxy_of) {
  const int lane = threadIdx.x & 31;
  int top_k = top_k_max < g - 1 ? top_k_max : g - 1;
  if (top_k < 1) top_k = 1;
  if (lane < g && g - 1 <= top_k_max) {
    // every member has at most top_k partners: all positive ones are kept
    const int i = lane;
    for (int j = i + 1; j < g; ++j) {
      if (proxy_of(i, j) > 0) atomicOr(&S.fmask[i], 1u << j);
    }
  } else if (g - 1 > top_k_max) {
    // ranking, one member at a time by the whole warp, lane j holding
    // partner j: a partner's rank is the number of partners better than it
    // under ranked_better (ratio desc, proxy gain desc, rep_lo asc, rep_hi
    // asc), and the top_k ranks are kept. The ratio is the same correctly
    // rounded double as the reference's; positive doubles order like their
    // bit patterns, so every comparison is an integer one.
    const int j = lane;
    for (int i = 0; i < g; ++i) {
      long long pg = 0;
      if (j < g && j != i) pg = i < j ? proxy_of(i, j) : proxy_of(j, i);
      const bool valid = pg > 0;
      const unsigned vm = __ballot_sync(0xffffffffu, valid);
      const int cnt = __popc(vm);
      if (cnt <= top_k) {
        if (valid) atomicOr(&S.fmask[i < j ? i : j], 1u << (i < j ? j : i));
        continue;
      }
      long long denom = 1;
      if (valid) {
        denom = S.old[i] + S.old[j];
        if (denom < 1) denom = 1;
      }
      if (!__any_sync(0xffffffffu, pg >= kExactRatio || denom >= kExactRatio)) {
        const RankCand c[1] = {{static_cast<unsigned>(pg), static_cast<unsigned>(denom), valid ? S.q[j] : 0}};
        int r[1];
        ExactRanks(c, r);
        if (valid && r[0] < top_k) atomicOr(&S.fmask[i < j ? i : j], 1u << (i < j ? j : i));
        continue;
      }
      long long rbits = 0;
      int lo = 0, hi = 0;
      if (valid) {
        rbits = __double_as_longlong(static_cast<double>(pg) / static_cast<double>(denom));
        const int qi = S.q[i];
        const int qj = S.q[j];
        lo = qi < qj ? qi : qj;
        hi = qi < qj ? qj : qi;
      }
      int rank = 0;
      for (unsigned rest = vm; rest; rest &= rest - 1) {
        const int o = __ffs(rest) - 1;
        const long long orb = __shfl_sync(0xffffffffu, rbits, o);
        const long long opg = __shfl_sync(0xffffffffu, pg, o);
        const int olo = __shfl_sync(0xffffffffu, lo, o);
        const int ohi = __shfl_sync(0xffffffffu, hi, o);
        const bool better =
            orb != rbits ? orb > rbits : opg != pg ? opg > pg : olo != lo ? olo < lo : ohi < hi;
        rank += (valid && o != j && better) ? 1 : 0;
      }
      if (valid && rank < top_k) atomicOr(&S.fmask[i < j ? i : j], 1u << (i < j ? j : i));
    }
  }
  __syncwarp();
}

__global__ void __launch_bounds__(kSmallWarps * 32) PrepareSmallKernel(PrepareParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmallWarpSmem& W = reinterpret_cast<SmallSmem*>(smem_raw)->w[threadIdx.x >> 5];
  SmallRowsSmem& S = W.rows;
  const int lane = threadIdx.x & 31;
  const int li = blockIdx.x * kSmallWarps + (threadIdx.x >> 5);
  if (li >= P.nlist) return;
  const int ri = P.list[P.list0 + li];
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  bool wide;
  const int E = StageSmallRows(P.Q, P.order + P.gstart[gid], g, S, &wide);
  if (E > kSmallStage) {
    if (lane == 0) {
      RaiseError(P.err, kErrSlots, gid, E, 0);
      P.cand_cnt[ri] = 0;
    }
    return;
  }
  bool slow;
  unsigned examined = SmallSums(P.Q, S, W.pairs, g, E, wide, &slow);
  if (lane < g) SmallFinishRow(P.Q, S, lane, wide, P.rc ? &P.rc[S.q[lane]] : nullptr);
  __syncwarp();
  SmallTopK(S, g, P.top_k, [&](int a, int b) {
    return slow ? SmallMerge(S, a, b).proxy : static_cast<long long>(W.pairs.pc[TriIndex(a, b, g)] >> 32);
  });
  // union of kept pairs in (a_idx, b_idx) order
  const unsigned mine = lane < g ? S.fmask[lane] : 0u;
  const int cnt = __popc(mine);
  int ex = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, ex, o);
    if (lane >= o) ex += y;
  }
  const int total = __shfl_sync(0xffffffffu, ex, 31);
  ex -= cnt;
  int2* out = P.cand + P.cand_off[ri];
  float2* feat = P.cand_feat ? P.cand_feat + P.cand_off[ri] : nullptr;
  PairInfo* info = P.info ? P.info + P.cand_off[ri] : nullptr;
  unsigned bits = mine;
  while (bits) {
    const int b = __ffs(bits) - 1;
    bits &= bits - 1;
    if (feat || info) {
      const SmallPair r = SmallPairAt(S, W.pairs, TriIndex(lane, b, g), lane, b, slow);
      if (feat) {
        long long denom = S.old[lane] + S.old[b];
        if (denom < 1) denom = 1;
        feat[ex] =
            make_float2(static_cast<float>(r.proxy), __fdividef(static_cast<float>(r.proxy), static_cast<float>(denom)));
      }
      if (info) info[ex] = SmallPairInfo(S, lane, b, r);
    }
    P.cand_rep[P.cand_off[ri] + ex] = make_int2(S.q[lane], S.q[b]);
    out[ex++] = make_int2(lane, b);
  }
  examined = __reduce_add_sync(0xffffffffu, examined);
  if (lane == 0) {
    P.cand_cnt[ri] = total;
    atomicAdd(&P.stats[kStGroupCount], 1ull);
    atomicMax(&P.stats[kStGroupMaxSize], static_cast<unsigned long long>(g));
    atomicAdd(&P.stats[kStRawPairCount], static_cast<unsigned long long>(g) * (g - 1) / 2);
    atomicAdd(&P.stats[kStCandAfterPrune], static_cast<unsigned long long>(total));
    atomicAdd(&P.stats[kStProxyExamined], static_cast<unsigned long long>(examined));
    atomicAdd(&P.stats[kStPrepareBytes], 12ull * static_cast<unsigned long long>(E));
  }
}

// ------------------------------------------------------------ score

struct ScoreParams {
  QuotientView Q;
  BlockCtl* ctl;  // work queues of the scoring passes
  const int* order;
  const int* gstart;
  const int* real;
  int rg0;
  int nrg;
  const long long* cand_off;
  const int2* cand;
  const int* cand_cnt;
  const int2* cand_rep;  // the pair's supernode ids, -1 for unused slots
  longlong2* res;
  // learned ranker (phase 0: off, every slot scored). keep[slot]: 1 =
  // exploration slot, scored in phase 1; 2 = scored in phase 2 iff its logit
  // zbuf[slot] >= *cutoff (the cutoff comes from phase 1's passing pairs)
  int phase;
  const unsigned char* keep;
  const float* zbuf;
  float* zpos;        // phase 1: logits of the exploration pairs passing the filter
  long long* zgain;   // phase 1: their exact gains
  unsigned* npos;
  unsigned zcap;
  const float* cutoff;
  int audit;          // phase 2: score pruned slots aside and count the ones the filter passes
  double threshold;
  ThresholdBits thr;  // threshold split for the integer test
  int use_threshold;
  const RowSums* rc;     // row sums of the block-start state (nullptr: full merge of the two rows)
  const PairInfo* info;  // per candidate slot (with rc)
  int strict;            // check every entry of both rows against its block's capacity (as the full merge does)
  unsigned long long* stats;
  DevError* err;
};

// The exact gain of candidate (a, b) from the row sums and the pair's shared
// part, by one lane; false: a row's heavy entries are neither all dense nor
// all light at this size, and have to be read.
struct GainParts {
  long long gain, before;
  int uni, ovl;
  int err;  // ErrCode of an invalid pair
};

__device__ __forceinline__ bool GainFromSums(const RowSums& A, const RowSums& B, const PairInfo& p, int strict,
                                             GainParts* out) {
  const long long sa = A.size, sb = B.size, s = sa + sb;
  const long long eab = p.eab;
  long long fa, fb;
  const bool have_a = RowAfter(A, s, &fa);
  const bool have_b = RowAfter(B, s, &fb);
  // counts beyond their block's capacity: at the merged size, and at the
  // row's own size where asked for or with more than a few heavy entries
  int bad = (p.ovl & kPairBad) != 0 || s < A.sbad || s < B.sbad;
  if (strict || A.nheavy > kHeavyFew || B.nheavy > kHeavyFew) bad |= sa < A.sbad || sb < B.sbad;
  const long long before = A.before + B.before - BlockCost(sb, sa, eab, false, bad) +
                           BlockCost(sa, sa, A.internal, true, bad) + BlockCost(sb, sb, B.internal, true, bad);
  const long long after = fa + fb - BlockCost(s, sb, eab, false, bad) - BlockCost(s, sa, eab, false, bad) + p.shared +
                          BlockCost(s, s, A.internal + B.internal + eab, true, bad);
  out->err = (p.ovl & kPairAsym) ? kErrAsymmetric : bad ? kErrBlockCost : kErrNone;
  out->gain = before - after;  // without the F of a row that has to be read
  out->before = before;
  out->ovl = static_cast<int>(p.ovl & ((1u << 30) - 1u));
  const int e = eab > 0 ? 1 : 0;
  out->uni = (A.len - e) + (B.len - e) - out->ovl;
  return have_a && have_b;
}

// The same, by a warp, for the pairs GainFromSums leaves.
__device__ GainParts WarpGainReadingRows(const QuotientView& Q, const RowSums& A, const RowSums& B, const PairInfo& p,
                                         int a, int b, int strict) {
  const long long s = static_cast<long long>(A.size) + B.size;
  GainParts g;
  GainFromSums(A, B, p, strict, &g);
  long long part;
  if (!RowAfter(A, s, &part)) g.gain += part - WarpRowAfter(Q, a, s);
  if (!RowAfter(B, s, &part)) g.gain += part - WarpRowAfter(Q, b, s);
  return g;
}

__device__ __forceinline__ bool PassesFilter(long long gain, long long before, double threshold, ThresholdBits thr,
                                             int use_threshold) {
  if (gain <= 0) return false;
  if (!use_threshold) return true;
  return before > 0 && RatioAtLeast(gain, before, threshold, thr);
}

__device__ __forceinline__ void FlushScoreStats(unsigned long long* stats, const GainWork& w, long long pairs,
                                                long long view_nnz) {
  if (pairs == 0) return;
  atomicAdd(&stats[kStExactCalls], static_cast<unsigned long long>(pairs));
  atomicAdd(&stats[kStInputNnz], static_cast<unsigned long long>(view_nnz));
  atomicAdd(&stats[kStRawA], static_cast<unsigned long long>(w.raw_a));
  atomicAdd(&stats[kStRawB], static_cast<unsigned long long>(w.raw_b));
  atomicAdd(&stats[kStUnion], static_cast<unsigned long long>(w.uni));
  atomicAdd(&stats[kStOverlap], static_cast<unsigned long long>(w.ovl));
  // algorithmic bytes: the gain computations' own, 8 B pair + 16 B result per pair
  atomicAdd(&stats[kStScoreBytes], static_cast<unsigned long long>(w.bytes + 24 * pairs));
}

// Candidate slots of a block are the concatenated per-group capacities; slots
// past a group's candidate count hold -1 and are skipped. A warp takes
// kScoreFetch slots at a time from the block's queue; fetch f holds the slots
// f, f + F, f + 2F, ... (F = the number of fetches): the candidates of one
// member are consecutive slots, and a hub member's pairs, where they have to
// read rows, must not all land on one warp.
//
// With row sums each lane scores its own pair from two 64-byte row records and
// one 16-byte pair record, the pairs that still have to read a row follow one
// by one by the whole warp. Before, every pair merged its two rows here
// (8-byte entries, 32 of each per step), although the prepare kernels had
// already visited every shared target: at R-MAT scale 23 that was 330 ms of a
// 1,291 ms run, and is 30 ms here. Without row sums (graphs beyond kFusedMaxArcs) a warp merges
// one pair's rows at a time, and fetches fewer of them.
constexpr int kScoreFetch = 32;
constexpr int kScoreFetchMerge = 8;

__global__ void __launch_bounds__(kScoreThreads, 4) ScoreKernel(ScoreParams P) {
  FollowsOn();
  constexpr unsigned kFull = 0xffffffffu;
  const long long s0 = P.cand_off[P.rg0];
  const long long s1 = P.cand_off[P.rg0 + P.nrg];
  const int lane = threadIdx.x & 31;
  GainWork w = {0, 0, 0, 0, 0};
  long long pairs = 0, view_nnz = 0;
  unsigned long long pruned = 0;
  const float cutoff = P.phase == 2 ? *P.cutoff : 0.0f;
  unsigned long long* queue = &P.ctl->work_next[P.phase == 2 ? 2 : 1];
  const int fetch = P.rc ? kScoreFetch : kScoreFetchMerge;
  const long long nfetch = (s1 - s0 + fetch - 1) / fetch;
  for (;;) {
    long long f = 0;
    if (lane == 0) f = static_cast<long long>(atomicAdd(queue, 1ull));
    f = __shfl_sync(kFull, f, 0);
    if (f >= nfetch) break;
    // what to do with this lane's slot: 0 nothing, 1 score, 2 pruned by the
    // ranker (scored aside by the audit)
    const long long slot = s0 + f + static_cast<long long>(lane) * nfetch;
    int2 ab = make_int2(-1, -1);
    int todo = 0;
    if (lane < fetch && slot < s1) {
      ab = P.cand_rep[slot];
      if (ab.x >= 0) {
        todo = 1;
        if (P.phase == 1 && P.keep[slot] != 1) todo = 0;  // phase 1 scores the exploration slots
        if (P.phase == 2) {
          if (P.keep[slot] == 1) {
            todo = 0;  // exploration slot, scored in phase 1
          } else if (P.zbuf[slot] < cutoff) {
            todo = 2;
          }
        }
      }
    }
    const bool score = todo == 1 || (todo == 2 && P.audit);
    GainParts g = {0, 0, 0, 0, 0};
    RowSums A, B;
    PairInfo p;
    bool by_warp = score;
    if (score && P.rc) {
      A = P.rc[ab.x];
      B = P.rc[ab.y];
      p = P.info[slot];
      by_warp = !GainFromSums(A, B, p, P.strict, &g);
      if (g.err) RaiseError(P.err, g.err, ab.x, ab.y, 0);
    }
    for (unsigned rest = __ballot_sync(kFull, by_warp); rest != 0u; rest &= rest - 1u) {
      const int j = __ffs(rest) - 1;
      const int a = __shfl_sync(kFull, ab.x, j);
      const int b = __shfl_sync(kFull, ab.y, j);
      GainParts r = {0, 0, 0, 0, 0};
      if (P.rc) {
        const long long sj = __shfl_sync(kFull, slot, j);
        r = WarpGainReadingRows(P.Q, P.rc[a], P.rc[b], P.info[sj], a, b, P.strict);
      } else {
        GainWork one = {0, 0, 0, 0, 0};
        WarpExactGain(P.Q, a, b, &r.gain, &r.before, &one, P.err);
        r.uni = static_cast<int>(one.uni);
        r.ovl = static_cast<int>(one.ovl);
      }
      if (lane == j) g = r;
    }
    if (todo == 0) continue;
    const bool passes = score && PassesFilter(g.gain, g.before, P.threshold, P.thr, P.use_threshold);
    if (todo == 2) {
      if (P.audit && passes) {
        atomicAdd(&P.stats[kStRkAuditPassing], 1ull);
        atomicAdd(&P.stats[kStRkAuditLost], 1ull);
      }
      P.res[slot] = make_longlong2(0, -1);
      ++pruned;
      continue;
    }
    if (P.phase != 0 && passes) {
      if (P.audit) atomicAdd(&P.stats[kStRkAuditPassing], 1ull);
      if (P.phase == 1) {
        const unsigned at = atomicAdd(P.npos, 1u);
        if (at < P.zcap) {
          P.zpos[at] = P.zbuf[slot];
          P.zgain[at] = g.gain;
        }
      }
    }
    P.res[slot] = make_longlong2(g.gain, g.before);
    ++pairs;
    const int la = P.rc ? A.len : P.Q.len[ab.x];
    const int lb = P.rc ? B.len : P.Q.len[ab.y];
    const long long ia = P.rc ? A.internal : P.Q.internal[ab.x];
    const long long ib = P.rc ? B.internal : P.Q.internal[ab.y];
    view_nnz += la + (ia > 0 ? 1 : 0) + lb + (ib > 0 ? 1 : 0);
    w.raw_a += la;
    w.raw_b += lb;
    w.uni += g.uni;
    w.ovl += g.ovl;
    // with row sums: two row records and a pair record; a pair that reads rows
    // (or merges them) 8 B per entry and 4 B per size
    w.bytes += P.rc ? 2ll * sizeof(RowSums) + sizeof(PairInfo) : 0ll;
    if (by_warp) {
      w.bytes += P.rc ? 12ll * ((RowAfterKnown(A, A.size + B.size) ? 0 : la) +
                                (RowAfterKnown(B, A.size + B.size) ? 0 : lb))
                      : 8ll * (la + lb) + 4ll * g.uni;
    }
  }
  __syncwarp();
  pairs = WarpSum(pairs);
  view_nnz = WarpSum(view_nnz);
  w.raw_a = WarpSum(w.raw_a);
  w.raw_b = WarpSum(w.raw_b);
  w.uni = WarpSum(w.uni);
  w.ovl = WarpSum(w.ovl);
  w.bytes = WarpSum(w.bytes);
  pruned = static_cast<unsigned long long>(WarpSum(static_cast<long long>(pruned)));
  if (lane == 0) {
    FlushScoreStats(P.stats, w, pairs, view_nnz);
    if (pruned) atomicAdd(&P.stats[kStRkPruned], pruned);
  }
}

// Scoring service over an explicit pair list (ScoreCandidatesCuda's role), a
// warp per pair. Pairs whose rows hold more than kPairLong entries together are
// left to ScoreLongPairsKernel in units of kPairUnit entries of the longer row
// and the part of the other that these ids span: a hub pair of 100,000 entries
// is a chain of thousands of steps for one warp, and was the kernel's tail
// (1.16 ms for 262,144 pairs at R-MAT 20, a tenth of it work).
constexpr int kPairLong = 2048;
constexpr int kPairUnit = 1024;

struct PairUnit {
  long long pair;
  int at;  // first entry of the longer row
  int pad;
};

// The terms of e(a, b) and of the two supernodes themselves.
__device__ __forceinline__ void PairOwnTerms(const QuotientView& Q, int a, int b, long long eab, long long* before,
                                             long long* after, int* bad) {
  const long long sa = Q.size[a], sb = Q.size[b], ia = Q.internal[a], ib = Q.internal[b];
  *before = BlockCost(sa, sa, ia, true, *bad) + BlockCost(sb, sb, ib, true, *bad) + BlockCost(sa, sb, eab, false, *bad);
  *after = BlockCost(sa + sb, sa + sb, ia + ib + eab, true, *bad);
}

__global__ void __launch_bounds__(kScoreThreads) ScorePairsKernel(QuotientView Q, const int* rep_a,
                                                                  const int* rep_b, long long count,
                                                                  long long* gain_out, long long* before_out,
                                                                  PairUnit* units, unsigned long long* nunits,
                                                                  unsigned long long max_units, DevError* err) {
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nw = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (long long p = warp; p < count; p += nw) {
    const int a = rep_a[p];
    const int b = rep_b[p];
    if (a == b || Q.size[a] <= 0 || Q.size[b] <= 0) {
      if (lane == 0) {
        RaiseError(err, kErrInactive, a, b, 0);
        gain_out[p] = 0;
        before_out[p] = 0;
      }
      continue;
    }
    const int la = Q.len[a], lb = Q.len[b];
    if (la + lb > kPairLong) {
      const int longer = la > lb ? la : lb;
      const unsigned n = static_cast<unsigned>((longer + kPairUnit - 1) / kPairUnit);
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(nunits, static_cast<unsigned long long>(n));
      at = __shfl_sync(0xffffffffu, at, 0);
      for (unsigned k = lane; k < n && at + k < max_units; k += 32) {
        units[at + k] = PairUnit{at + n <= max_units ? p : -1, static_cast<int>(k) * kPairUnit, 0};
      }
      if (at + n <= max_units) {
        if (lane == 0) {
          const long long ea = RowLookup(Q.ent + Q.off[a], la, b), eb = RowLookup(Q.ent + Q.off[b], lb, a);
          long long before, after;
          int bad = 0;
          PairOwnTerms(Q, a, b, ea, &before, &after, &bad);
          if (ea != eb) RaiseError(err, kErrAsymmetric, a, b, 0);
          if (bad) RaiseError(err, kErrBlockCost, a, b, 0);
          gain_out[p] = before - after;  // the units add theirs
          before_out[p] = before;
        }
        continue;
      }
    }
    long long gain = 0, before = 0;
    WarpExactGain(Q, a, b, &gain, &before, nullptr, err);
    if (lane == 0) {
      gain_out[p] = gain;
      before_out[p] = before;
    }
  }
}

__global__ void __launch_bounds__(kScoreThreads) ScoreLongPairsKernel(QuotientView Q, const int* rep_a,
                                                                      const int* rep_b, long long* gain_out,
                                                                      long long* before_out, const PairUnit* units,
                                                                      const unsigned long long* nunits,
                                                                      unsigned long long max_units, DevError* err) {
  const unsigned long long total = *nunits < max_units ? *nunits : max_units;
  const unsigned long long nw = (static_cast<unsigned long long>(gridDim.x) * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (unsigned long long t = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < total;
       t += nw) {
    const PairUnit u = units[t];
    if (u.pair < 0) continue;
    const int a = rep_a[u.pair], b = rep_b[u.pair];
    const bool a_long = Q.len[a] >= Q.len[b];
    const int x = a_long ? a : b, y = a_long ? b : a;
    const Entry* rx = Q.ent + Q.off[x];
    const Entry* ry = Q.ent + Q.off[y];
    const int lx = Q.len[x], ly = Q.len[y];
    const int end = u.at + kPairUnit < lx ? u.at + kPairUnit : lx;
    // ids from the unit's first (the first unit: from the start) up to the
    // next unit's first (the last unit: to the end)
    int edge = 0;
    if (lane == 0 && u.at > 0) edge = RowLowerBound(ry, ly, EntNb(rx[u.at]));
    if (lane == 1) edge = end < lx ? RowLowerBound(ry, ly, EntNb(rx[end])) : ly;
    const int y0 = __shfl_sync(0xffffffffu, edge, 0), y1 = __shfl_sync(0xffffffffu, edge, 1);
    MergeTerms T;
    WarpMergeTerms(Q, x, y, Q.size[x], Q.size[y], rx + u.at, end - u.at, ry + y0, y1 - y0, &T);
    const long long before = WarpSum(T.before), after = WarpSum(T.after);
    const bool bad = __any_sync(0xffffffffu, T.bad);
    if (lane == 0) {
      atomicAdd(reinterpret_cast<unsigned long long*>(&gain_out[u.pair]), static_cast<unsigned long long>(before - after));
      atomicAdd(reinterpret_cast<unsigned long long*>(&before_out[u.pair]), static_cast<unsigned long long>(before));
      if (bad) RaiseError(err, kErrBlockCost, a, b, 0);
    }
  }
}

// ------------------------------------------------------------ select

struct SelectParams {
  const int* order;
  const int* gstart;
  const int* glen;
  const int* real;
  int rg0;
  const long long* cand_off;
  const int2* cand;
  const int* cand_cnt;
  const longlong2* res;
  const long long* sel_off;
  int* sel_keep;
  int* sel_rem;
  long long* sel_gain;
  int* sel_cnt;
  const int* qlen;
  int* stamp;
  int* partner;
  int* seq;
  int block_stamp;
  double threshold;
  ThresholdBits thr;  // threshold split for the integer test
  int use_threshold;
  unsigned char* scratch;
  unsigned long long scratch_cap;
  BlockCtl* ctl;
  unsigned long long* stats;
  DevError* err;
  const int* list;  // real-group positions handled by this launch
  int list0;
  int nlist;
  int* sel_list;    // selection slots of the selected pairs, appended (count: ctl->sel_total)
};

// In-place ascending bitonic sort of n (power of two) keys by one CTA.
__device__ void CtaBitonicSort(unsigned long long* keys, int n) {
  for (int k = 2; k <= n; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const unsigned long long a = keys[i];
          const unsigned long long b = keys[ixj];
          const bool up = (i & k) == 0;
          if ((a > b) == up) {
            keys[i] = b;
            keys[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Threshold filter, g0 order (gain desc, a_idx asc, b_idx asc) by a bitonic
// sort of packed keys, greedy endpoint-disjoint pass. The selected pairs are
// the block's commit list: the reference validates each against the same
// block-start state its score came from (gain > 0 by the filter), so every
// one is accepted; their endpoints are marked here (stamp, partner, commit
// order) for the commit kernel.
template <int kThreads, int kSmemKeys>
__global__ void __launch_bounds__(kThreads) SelectKernel(SelectParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* skeys = reinterpret_cast<unsigned long long*>(smem_raw);
  __shared__ unsigned char used[kMaxGroup];
  __shared__ int nkeys;
  __shared__ unsigned long long* gkeys;
  __shared__ unsigned long long rej_thr, positive;
  const int tid = threadIdx.x;
  const int ri = P.list[P.list0 + blockIdx.x];
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  const int cnt = g >= 2 && g <= kMaxGroup ? P.cand_cnt[ri] : 0;
  if (cnt == 0) {
    if (tid == 0) P.sel_cnt[ri] = 0;
    return;
  }
  int cap = 1;
  while (cap < cnt) cap <<= 1;
  if (tid == 0) {
    nkeys = 0;
    rej_thr = 0;
    positive = 0;
    gkeys = cap <= kSmemKeys ? skeys
                                   : ScratchAlloc(P.scratch, P.scratch_cap, P.ctl, 8ull * cap, P.err);
  }
  for (int i = tid; i < g; i += kThreads) used[i] = 0;
  __syncthreads();
  unsigned long long* keys = gkeys;
  if (keys == nullptr) {
    if (tid == 0) P.sel_cnt[ri] = 0;
    return;
  }
  const long long base = P.cand_off[ri];
  unsigned long long my_rej = 0, my_pos = 0;
  for (int c = tid; c < cnt; c += kThreads) {
    const longlong2 r = P.res[base + c];
    const long long gain = r.x;
    const long long before = r.y;
    if (before < 0) continue;  // pruned by the ranker before scoring
    if (gain <= 0) {
      ++my_rej;
      continue;
    }
    if (P.use_threshold) {
      if (before <= 0) {
        ++my_rej;
        continue;
      }
      if (!RatioAtLeast(gain, before, P.threshold, P.thr)) {
        ++my_rej;
        continue;
      }
    }
    ++my_pos;
    if (gain > kKeyGainMax) RaiseError(P.err, kErrKeyRange, gid, c, 0);
    const int2 ab = P.cand[base + c];
    const unsigned long long key = (static_cast<unsigned long long>(kKeyGainMax - gain) << (2 * kKeyIdxBits)) |
                                   (static_cast<unsigned long long>(ab.x) << kKeyIdxBits) |
                                   static_cast<unsigned long long>(ab.y);
    keys[atomicAdd(&nkeys, 1)] = key;
  }
  if (my_rej) atomicAdd(&rej_thr, my_rej);
  if (my_pos) atomicAdd(&positive, my_pos);
  __syncthreads();
  const int m = nkeys;
  int pow2 = 1;
  while (pow2 < m) pow2 <<= 1;
  for (int i = m + tid; i < pow2; i += kThreads) keys[i] = ~0ull;
  __syncthreads();
  if (m > 1) CtaBitonicSort(keys, pow2);
  if (tid == 0) {
    const int* q = P.order + P.gstart[gid];
    const long long so = P.sel_off[ri];
    int ns = 0;
    long long total = 0;
    unsigned long long overlap = 0, work = 0;
    const unsigned long long idx_mask = (1ull << kKeyIdxBits) - 1;
    for (int k = 0; k < m; ++k) {
      const unsigned long long key = keys[k];
      const int b = static_cast<int>(key & idx_mask);
      const int a = static_cast<int>((key >> kKeyIdxBits) & idx_mask);
      const long long gain = kKeyGainMax - static_cast<long long>(key >> (2 * kKeyIdxBits));
      if (used[a] || used[b]) {
        ++overlap;
        continue;
      }
      used[a] = 1;
      used[b] = 1;
      const int keep = q[a];
      const int rem = q[b];
      P.sel_keep[so + ns] = keep;
      P.sel_rem[so + ns] = rem;
      P.sel_gain[so + ns] = gain;
      P.stamp[keep] = 2 * P.block_stamp;
      P.stamp[rem] = 2 * P.block_stamp + 1;
      P.partner[keep] = rem;
      P.partner[rem] = keep;
      P.seq[rem] = static_cast<int>(so + ns);
      P.sel_list[atomicAdd(&P.ctl->sel_total, 1u)] = static_cast<int>(so + ns);
      work += static_cast<unsigned long long>(P.qlen[keep] + P.qlen[rem]);
      ++ns;
      total += gain;
    }
    P.sel_cnt[ri] = ns;
    atomicAdd(&P.stats[kStRejThreshold], rej_thr);
    atomicAdd(&P.stats[kStPositive], positive);
    atomicAdd(&P.stats[kStRejOverlap], overlap);
    atomicAdd(&P.stats[kStCandPairs], static_cast<unsigned long long>(m));
    atomicAdd(&P.stats[kStSelected], static_cast<unsigned long long>(ns));
    atomicAdd(&P.stats[kStLocalGain], static_cast<unsigned long long>(total));
    // CommitSelectedPairs validation counters (src/sweg.cpp:2683-2719): one
    // exact-gain call per selected pair, reading both rows, all accepted.
    atomicAdd(&P.stats[kStValidationCalls], static_cast<unsigned long long>(ns));
    atomicAdd(&P.stats[kStValidationWork], work);
    atomicAdd(&P.stats[kStIsolatedGain], static_cast<unsigned long long>(total));
  }
}

// Groups of more than kSelectMidGroup members: the g0 greedy pass over keys
// in ascending order selects exactly the edges that are, in some round of
// the following loop, the smallest live key at both of their endpoints
// (keys are distinct): per round every live key bids for its two endpoints
// (shared-memory atomicMin), keys that win both are selected, keys touching
// a selected endpoint die. Only the selected keys (at most g/2) are then
// sorted, which gives the greedy order of the commit list; a key is skipped
// by the greedy pass exactly when it is not selected, so the overlap count
// is the number of keys minus the selected ones.
constexpr int kMatchThreads = 512;
constexpr int kMatchSmemKeys = 8192;

template <int kGroup>
struct MatchSmem {
  unsigned long long best[kGroup];
  unsigned long long chosen[kGroup / 2];
  unsigned char matched[kGroup];
  int nchosen, live_any;
};

// The greedy choice among m keys of a group of g members by a CTA of
// kThreads (kin, kout: two buffers of m keys, the first holds them);
// chosen[] gets the selected keys in ascending order, their number is
// returned. Ends with a barrier.
template <int kThreads, int kGroup>
__device__ int MatchKeys(MatchSmem<kGroup>& M, unsigned long long* kin, unsigned long long* kout, int m, int g) {
  const int tid = threadIdx.x;
  if (tid == 0) M.nchosen = 0;
  for (int i = tid; i < g; i += kThreads) M.matched[i] = 0;
  // rounds of locally dominant keys (each round selects at least the
  // smallest live key, so at most g/2 rounds); the keys still live after a
  // round move to the other buffer (the matching depends on the key values
  // only, not on their order)
  int nlive = m;
  for (int round = 0; round <= kGroup / 2 && nlive > 0; ++round) {
    for (int i = tid; i < g; i += kThreads) M.best[i] = ~0ull;
    if (tid == 0) M.live_any = 0;
    __syncthreads();
    for (int k = tid; k < nlive; k += kThreads) {
      const unsigned long long key = kin[k];
      atomicMin(&M.best[(key >> kKeyIdxBits) & kKeyIdxMask], key);
      atomicMin(&M.best[key & kKeyIdxMask], key);
    }
    __syncthreads();
    for (int k = tid; k < nlive; k += kThreads) {
      const unsigned long long key = kin[k];
      const int a = static_cast<int>((key >> kKeyIdxBits) & kKeyIdxMask);
      const int b = static_cast<int>(key & kKeyIdxMask);
      if (M.best[a] == key && M.best[b] == key) {
        M.matched[a] = 1;
        M.matched[b] = 1;
        M.chosen[atomicAdd(&M.nchosen, 1)] = key;
      }
    }
    __syncthreads();
    for (int k = tid; k < nlive; k += kThreads) {
      const unsigned long long key = kin[k];
      if (!M.matched[(key >> kKeyIdxBits) & kKeyIdxMask] && !M.matched[key & kKeyIdxMask]) {
        kout[atomicAdd(&M.live_any, 1)] = key;
      }
    }
    __syncthreads();
    nlive = M.live_any;
    unsigned long long* t = kin;
    kin = kout;
    kout = t;
    __syncthreads();  // every thread has read live_any before the next round resets it
  }
  __syncthreads();
  const int ns = M.nchosen;
  int pow2 = 1;
  while (pow2 < ns) pow2 <<= 1;
  for (int i = ns + tid; i < pow2; i += kThreads) M.chosen[i] = ~0ull;
  __syncthreads();
  if (ns > 1) CtaBitonicSort(M.chosen, pow2);
  return ns;
}

__device__ __forceinline__ void SelectMatchGroup(const SelectParams& P, int ri) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* skeys = reinterpret_cast<unsigned long long*>(smem_raw);
  __shared__ MatchSmem<kMaxGroup> M;
  __shared__ int nkeys;
  __shared__ unsigned long long* gkeys;
  __shared__ unsigned long long rej_thr;
  const int tid = threadIdx.x;
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  const int cnt = g >= 2 && g <= kMaxGroup ? P.cand_cnt[ri] : 0;
  if (cnt == 0) {
    if (tid == 0) P.sel_cnt[ri] = 0;
    return;
  }
  if (tid == 0) {
    nkeys = 0;
    rej_thr = 0;
    // two key buffers of cnt entries: the live keys are compacted from one
    // into the other every round
    gkeys = 2 * cnt <= kMatchSmemKeys ? skeys
                                      : ScratchAlloc(P.scratch, P.scratch_cap, P.ctl, 16ull * cnt, P.err);
  }
  __syncthreads();
  unsigned long long* keys = gkeys;
  if (keys == nullptr) {
    if (tid == 0) P.sel_cnt[ri] = 0;
    return;
  }
  const long long base = P.cand_off[ri];
  unsigned long long my_rej = 0;
  for (int c = tid; c < cnt; c += kMatchThreads) {
    const longlong2 r = P.res[base + c];
    const long long gain = r.x;
    const long long before = r.y;
    if (before < 0) continue;  // pruned by the ranker before scoring
    bool ok = gain > 0;
    if (ok && P.use_threshold) {
      ok = before > 0 && RatioAtLeast(gain, before, P.threshold, P.thr);
    }
    if (!ok) {
      ++my_rej;
      continue;
    }
    if (gain > kKeyGainMax) RaiseError(P.err, kErrKeyRange, gid, c, 0);
    const int2 ab = P.cand[base + c];
    keys[atomicAdd(&nkeys, 1)] = PackKey(gain, ab.x, ab.y);
  }
  if (my_rej) atomicAdd(&rej_thr, my_rej);
  __syncthreads();
  const int m = nkeys;
  // the selected keys in greedy (ascending key) order
  const int ns = MatchKeys<kMatchThreads>(M, keys, keys + cnt, m, g);
  const int* q = P.order + P.gstart[gid];
  const long long so = P.sel_off[ri];
  long long my_total = 0;
  unsigned long long my_work = 0;
  for (int i = tid; i < ns; i += kMatchThreads) {
    const unsigned long long key = M.chosen[i];
    const int a = static_cast<int>((key >> kKeyIdxBits) & kKeyIdxMask);
    const int b = static_cast<int>(key & kKeyIdxMask);
    const long long gain = kKeyGainMax - static_cast<long long>(key >> (2 * kKeyIdxBits));
    const int keep = q[a];
    const int rem = q[b];
    P.sel_keep[so + i] = keep;
    P.sel_rem[so + i] = rem;
    P.sel_gain[so + i] = gain;
    P.stamp[keep] = 2 * P.block_stamp;
    P.stamp[rem] = 2 * P.block_stamp + 1;
    P.partner[keep] = rem;
    P.partner[rem] = keep;
    P.seq[rem] = static_cast<int>(so + i);
    P.sel_list[atomicAdd(&P.ctl->sel_total, 1u)] = static_cast<int>(so + i);
    my_work += static_cast<unsigned long long>(P.qlen[keep] + P.qlen[rem]);
    my_total += gain;
  }
  // chosen[] is no longer needed: reuse best[] for the two sums
  __syncthreads();
  if (tid == 0) {
    M.best[0] = 0;
    M.best[1] = 0;
  }
  __syncthreads();
  my_total = WarpSum(my_total);
  my_work = static_cast<unsigned long long>(WarpSum(static_cast<long long>(my_work)));
  if ((tid & 31) == 0) {
    if (my_total) atomicAdd(&M.best[0], static_cast<unsigned long long>(my_total));
    if (my_work) atomicAdd(&M.best[1], my_work);
  }
  __syncthreads();
  if (tid == 0) {
    const unsigned long long total = M.best[0];
    P.sel_cnt[ri] = ns;
    atomicAdd(&P.stats[kStRejThreshold], rej_thr);
    atomicAdd(&P.stats[kStPositive], static_cast<unsigned long long>(m));
    atomicAdd(&P.stats[kStRejOverlap], static_cast<unsigned long long>(m - ns));
    atomicAdd(&P.stats[kStCandPairs], static_cast<unsigned long long>(m));
    atomicAdd(&P.stats[kStSelected], static_cast<unsigned long long>(ns));
    atomicAdd(&P.stats[kStLocalGain], total);
    atomicAdd(&P.stats[kStValidationCalls], static_cast<unsigned long long>(ns));
    atomicAdd(&P.stats[kStValidationWork], M.best[1]);
    atomicAdd(&P.stats[kStIsolatedGain], total);
  }
}

__global__ void __launch_bounds__(kMatchThreads) SelectMatchKernel(SelectParams P) {
  FollowsOn();
  // list == nullptr: the real groups list0, list0 + 1, ... (a whole block)
  SelectMatchGroup(P, P.list ? P.list[P.list0 + blockIdx.x] : P.list0 + static_cast<int>(blockIdx.x));
}

// Groups of at most kSelectSmallGroup members (at most 28 candidates): one
// warp per group, one candidate per lane, a register bitonic sort across the
// lanes and the greedy pass over shuffled keys; counters are summed per CTA.
// Output and counters equal those of SelectKernel.
constexpr int kSelectSmallGroup = 8;
constexpr int kSelectSmallWarps = 8;

__device__ __forceinline__ unsigned long long WarpBitonicSortAsc(unsigned long long key, int lane) {
  for (int k = 2; k <= 32; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, j);
      const bool up = (lane & k) == 0;
      const bool lower = (lane & j) == 0;
      // the lower lane of a pair keeps the smaller key in an ascending run
      const bool take_min = lower == up;
      key = take_min ? (other < key ? other : key) : (other > key ? other : key);
    }
  }
  return key;
}

__global__ void __launch_bounds__(kSelectSmallWarps * 32) SelectSmallKernel(SelectParams P) {
  FollowsOn();
  __shared__ unsigned long long acc[9];
  const int lane = threadIdx.x & 31;
  const int li = blockIdx.x * kSelectSmallWarps + (threadIdx.x >> 5);
  if (threadIdx.x < 9) acc[threadIdx.x] = 0;
  __syncthreads();
  if (li < P.nlist) {
    const int ri = P.list[P.list0 + li];
    const int gid = P.real[ri];
    const int g = P.glen[gid];
    const int cnt = P.cand_cnt[ri];
    const long long base = P.cand_off[ri];
    unsigned long long key = ~0ull;
    int rej = 0, pos = 0;
    if (lane < cnt) {
      const longlong2 r = P.res[base + lane];
      const long long gain = r.x;
      const long long before = r.y;
      if (before >= 0) {  // negative: pruned by the ranker before scoring
        bool ok = gain > 0;
        if (ok && P.use_threshold) {
          ok = before > 0 && RatioAtLeast(gain, before, P.threshold, P.thr);
        }
        if (!ok) {
          rej = 1;
        } else {
          pos = 1;
          if (gain > kKeyGainMax) RaiseError(P.err, kErrKeyRange, gid, lane, 0);
          const int2 ab = P.cand[base + lane];
          key = (static_cast<unsigned long long>(kKeyGainMax - gain) << (2 * kKeyIdxBits)) |
                (static_cast<unsigned long long>(ab.x) << kKeyIdxBits) | static_cast<unsigned long long>(ab.y);
        }
      }
    }
    const int m = __popc(__ballot_sync(0xffffffffu, pos != 0));
    const int nrej = __popc(__ballot_sync(0xffffffffu, rej != 0));
    key = WarpBitonicSortAsc(key, lane);
    const int* q = P.order + P.gstart[gid];
    const long long so = P.sel_off[ri];
    const unsigned long long idx_mask = (1ull << kKeyIdxBits) - 1;
    unsigned used = 0;
    int ns = 0;
    long long total = 0;
    unsigned long long overlap = 0, work = 0;
    for (int k = 0; k < m; ++k) {
      const unsigned long long kk = __shfl_sync(0xffffffffu, key, k);
      const int b = static_cast<int>(kk & idx_mask);
      const int a = static_cast<int>((kk >> kKeyIdxBits) & idx_mask);
      if ((used >> a & 1u) || (used >> b & 1u)) {
        ++overlap;
        continue;
      }
      used |= (1u << a) | (1u << b);
      const long long gain = kKeyGainMax - static_cast<long long>(kk >> (2 * kKeyIdxBits));
      if (lane == 0) {
        const int keep = q[a];
        const int rem = q[b];
        P.sel_keep[so + ns] = keep;
        P.sel_rem[so + ns] = rem;
        P.sel_gain[so + ns] = gain;
        P.stamp[keep] = 2 * P.block_stamp;
        P.stamp[rem] = 2 * P.block_stamp + 1;
        P.partner[keep] = rem;
        P.partner[rem] = keep;
        P.seq[rem] = static_cast<int>(so + ns);
        P.sel_list[atomicAdd(&P.ctl->sel_total, 1u)] = static_cast<int>(so + ns);
        work += static_cast<unsigned long long>(P.qlen[keep] + P.qlen[rem]);
      }
      ++ns;
      total += gain;
    }
    (void)g;
    if (lane == 0) {
      P.sel_cnt[ri] = ns;
      atomicAdd(&acc[0], static_cast<unsigned long long>(nrej));
      atomicAdd(&acc[1], static_cast<unsigned long long>(m));
      atomicAdd(&acc[2], overlap);
      atomicAdd(&acc[3], static_cast<unsigned long long>(m));
      atomicAdd(&acc[4], static_cast<unsigned long long>(ns));
      atomicAdd(&acc[5], static_cast<unsigned long long>(total));
      atomicAdd(&acc[6], work);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (acc[0]) atomicAdd(&P.stats[kStRejThreshold], acc[0]);
    if (acc[1]) atomicAdd(&P.stats[kStPositive], acc[1]);
    if (acc[2]) atomicAdd(&P.stats[kStRejOverlap], acc[2]);
    if (acc[3]) atomicAdd(&P.stats[kStCandPairs], acc[3]);
    if (acc[4]) {
      atomicAdd(&P.stats[kStSelected], acc[4]);
      atomicAdd(&P.stats[kStValidationCalls], acc[4]);
    }
    if (acc[5]) {
      atomicAdd(&P.stats[kStLocalGain], acc[5]);
      atomicAdd(&P.stats[kStIsolatedGain], acc[5]);
    }
    if (acc[6]) atomicAdd(&P.stats[kStValidationWork], acc[6]);
  }
}

#include "medium.cuh"
#include "window.cuh"

// ------------------------------------------------------------ commit

// A claimed neighbour row of more than kRowSmem entries and its block scratch:
// one mask bit per entry (renamed or not), the entries to insert (room for a
// power of two of at least the row's length), a copy of the row where needed.
struct HugeRow {
  int x;
  int len;
  int nins;  // entries to insert
  int pad;
  unsigned* mask;
  Entry* ins;
  Entry* copy;
};

struct CommitParams {
  QuotientView Q;
  int rg0;
  int nrg;
  const long long* sel_off;
  const int* sel_keep;
  const int* sel_rem;
  const long long* sel_gain;
  const int* sel_cnt;
  // Update_S state
  int* head;
  int* next;
  int* tail;
  int* fwd;
  int* stamp;
  int* partner;
  int* seq;
  int* claim;
  int block_stamp;
  unsigned long long* pool_top;
  unsigned long long pool_cap;
  unsigned char* scratch;
  unsigned long long scratch_cap;
  BlockCtl* ctl;
  unsigned long long* stats;
  DevError* err;
  int* rows_short;  // claimed neighbour rows of at most kWarpRowMax entries (count: ctl->short_cnt)
  int* rows_long;   // those of at most kRowSmem (count: ctl->long_cnt)
  HugeRow* rows_huge;  // the other claimed neighbour rows (count: ctl->huge_cnt)
  int2* huge_units;    // {index into rows_huge, first entry} of their scan units (count: ctl->huge_units)
  unsigned* ticket; // last-CTA counter of the long-row rewrite kernel, left at 0
  const int* sel_list;  // selection slots of the block's selected pairs (count: ctl->sel_total)
  int warp_pairs;       // 1: pairs with at most kWarpRow row entries go to CommitShortKernel
  int windowed;         // 1: the batch of a window of blocks (W): the groups it touches are listed
  WindowParams W;
};

// Optional re-validation (--verify-cuda-gain): recomputes the exact gain of
// every selected pair against the block-start state and checks it equals
// the scored gain and is positive.
__global__ void __launch_bounds__(256) VerifyKernel(CommitParams P) {
  const int lane = threadIdx.x & 31;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nw = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const unsigned total = P.ctl->sel_total;
  for (long long idx = warp; idx < total; idx += nw) {
    const long long slot = P.sel_list[idx];
    const int k = P.sel_keep[slot];
    const int r = P.sel_rem[slot];
    long long gain = 0, before = 0;
    WarpExactGain(P.Q, k, r, &gain, &before, nullptr, P.err);
    if (lane == 0 && (gain != P.sel_gain[slot] || gain <= 0)) RaiseError(P.err, kErrValidation, k, r, 0);
  }
}

// Marks the endpoints of an explicit merge batch (no selection step).
__global__ void MarkKernel(const int* keep, const int* rem, int count, int* stamp, int* partner, int* seq,
                           int block_stamp, int* sel_list, BlockCtl* ctl) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) {
    stamp[keep[i]] = 2 * block_stamp;
    stamp[rem[i]] = 2 * block_stamp + 1;
    partner[keep[i]] = rem[i];
    partner[rem[i]] = keep[i];
    seq[rem[i]] = i;
    sel_list[i] = i;
  }
  if (i == 0) ctl->sel_total = static_cast<unsigned>(count);
}

struct RowsSmem {
  Entry s[kRowSmem];
  int d[kRowSmem + 1];
  Entry ins[kRowSmem];
};
// every warp of a rewrite CTA has a kWarpRowMax slice of s and of ins
static_assert(kWarpRowMax * (kRowsThreads / 32) <= kRowSmem, "warp slices of the rewrite buffers");

// Rewrites a staged sorted row S[0..L) (adjacent equal ids allowed: the keep
// row is staged as the merge of two rows) into out: duplicates are summed,
// ids sk / sr are dropped, entries of supernodes removed in this block move
// to their keep partner (summed into its entry, or inserted at its sorted
// position). Returns the new length.
__device__ int RewriteRow(const CommitParams& P, Entry* S, int L, int* D, Entry* INS, int sk, int sr, Entry* out) {
  using BlockScan = cub::BlockScan<int, kRowsThreads>;
  __shared__ typename BlockScan::TempStorage scan_tmp;
  __shared__ int nins, carry;
  const int tid = threadIdx.x;
  const int remove_stamp = 2 * P.block_stamp + 1;
  if (tid == 0) {
    nins = 0;
    carry = 0;
  }
  if (sk >= 0) {
    // a keep row staged as the merge of two rows: equal neighbours are adjacent
    for (int i = tid; i < L; i += kRowsThreads) {
      int drop = 0;
      if (i > 0 && EntNb(S[i]) == EntNb(S[i - 1])) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&S[i - 1]), static_cast<unsigned long long>(EntCnt(S[i])));
        drop = 1;
      }
      D[i] = drop;
    }
  } else {
    // a neighbour row is canonical
    for (int i = tid; i < L; i += kRowsThreads) D[i] = 0;
  }
  __syncthreads();
  // entries of supernodes removed in this block: four lookups in flight per
  // thread
  for (int i0 = tid; i0 < L; i0 += 4 * kRowsThreads) {
    int id[4], st[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * kRowsThreads;
      id[u] = i < L && !D[i] ? EntNb(S[i]) : -1;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) st[u] = id[u] >= 0 && id[u] != sk && id[u] != sr ? P.stamp[id[u]] : 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * kRowsThreads;
      if (id[u] < 0) continue;
      if (id[u] == sk || id[u] == sr) {
        D[i] = 1;
        continue;
      }
      if (st[u] == remove_stamp) {
        const int kp = P.partner[id[u]];
        D[i] = 1;
        if (kp == sk) continue;
        const int p = RowLowerBound(S, L, kp);
        const long long c = EntCnt(S[i]);
        if (p < L && EntNb(S[p]) == kp) {
          atomicAdd(reinterpret_cast<unsigned long long*>(&S[p]), static_cast<unsigned long long>(c));
        } else {
          INS[atomicAdd(&nins, 1)] = MakeEnt(kp, c);
        }
      }
    }
  }
  __syncthreads();
  // exclusive scan of drop flags (D[L] = total), four flags per thread a step
  for (int base = 0; base < L; base += 4 * kRowsThreads) {
    const int i0 = base + 4 * tid;
    int v[4], sum = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      v[u] = i0 + u < L ? D[i0 + u] : 0;
      sum += v[u];
    }
    int ex = 0, agg = 0;
    BlockScan(scan_tmp).ExclusiveSum(sum, ex, agg);
    __syncthreads();
    int run = carry + ex;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i0 + u < L) D[i0 + u] = run;
      run += v[u];
    }
    __syncthreads();
    if (tid == 0) carry += agg;
    __syncthreads();
  }
  if (tid == 0) D[L] = carry;
  const int m = nins;
  int pow2 = 1;
  while (pow2 < m) pow2 <<= 1;
  for (int i = m + tid; i < pow2; i += kRowsThreads) INS[i] = ~0ull;
  __syncthreads();
  if (m > 1) CtaBitonicSort(INS, pow2);
  for (int i = tid; i < L; i += kRowsThreads) {
    if (D[i + 1] != D[i]) continue;  // dropped
    const Entry e = S[i];
    const int pos = i - D[i] + RowLowerBound(INS, m, EntNb(e));
    out[pos] = e;
  }
  for (int j = tid; j < m; j += kRowsThreads) {
    const Entry e = INS[j];
    const int p = RowLowerBound(S, L, EntNb(e));
    out[j + p - D[p]] = e;
  }
  __syncthreads();
  return L - D[L] + m;
}

// Staging buffers for a row of L entries: shared memory when it fits,
// block scratch otherwise. Returns false (error raised) when scratch is out.
__device__ bool StageBuffers(const CommitParams& P, RowsSmem& R, int L, Entry** S, int** D, Entry** INS) {
  __shared__ Entry* gbuf;
  if (L <= kRowSmem) {
    *S = R.s;
    *D = R.d;
    *INS = R.ins;
    return true;
  }
  int pow2 = 1;
  while (pow2 < L) pow2 <<= 1;
  if (threadIdx.x == 0) {
    gbuf = reinterpret_cast<Entry*>(ScratchAlloc(P.scratch, P.scratch_cap, P.ctl,
                                                 8ull * L + 4ull * (L + 1) + 8ull * pow2 + 512ull, P.err));
  }
  __syncthreads();
  if (gbuf == nullptr) return false;
  *S = gbuf;
  *INS = gbuf + L;
  *D = reinterpret_cast<int*>(gbuf + L + pow2);
  return true;
}

// Row x holds an entry of a supernode removed in this block: listed once for
// the rewrite, by its length.
__device__ __forceinline__ void ClaimRow(const CommitParams& P, int x) {
  if (atomicExch(&P.claim[x], P.block_stamp) == P.block_stamp) return;
  const int len = P.Q.len[x];
  if (len <= kWarpRowMax) {
    P.rows_short[atomicAdd(&P.ctl->short_cnt, 1u)] = x;
  } else if (len <= (P.windowed ? kWindowRow : kRowSmem)) {
    P.rows_long[atomicAdd(&P.ctl->long_cnt, 1u)] = x;
  } else {
    int pow2 = 1;
    while (pow2 < len) pow2 <<= 1;
    const unsigned long long mask_bytes = ((static_cast<unsigned long long>(len) + 31) / 32 * 4 + 15) & ~15ull;
    unsigned char* mem = reinterpret_cast<unsigned char*>(
        ScratchAlloc(P.scratch, P.scratch_cap, P.ctl, mask_bytes + 8ull * pow2 + 8ull * len, P.err));
    if (mem == nullptr) return;
    HugeRow h;
    h.x = x;
    h.len = len;
    h.nins = 0;
    h.pad = 0;
    h.mask = reinterpret_cast<unsigned*>(mem);
    h.ins = reinterpret_cast<Entry*>(mem + mask_bytes);
    h.copy = h.ins + pow2;
    const unsigned at = atomicAdd(&P.ctl->huge_cnt, 1u);
    P.rows_huge[at] = h;
    const unsigned units = static_cast<unsigned>((len + kHugeUnit - 1) / kHugeUnit);
    const unsigned u0 = atomicAdd(&P.ctl->huge_units, units);
    for (unsigned u = 0; u < units; ++u) P.huge_units[u0 + u] = make_int2(static_cast<int>(at), static_cast<int>(u) * kHugeUnit);
  }
}

// A neighbour x of a merged pair: its group has to be evaluated again if it has
// been already ([p, e): evaluated, not committed).
__device__ __forceinline__ void MarkTouched(const CommitParams& P, int x, int p, int e) {
  const int ri = P.W.node_ri[x];
  if (ri < p || ri >= e) return;
  if (P.W.dirty[ri] != 0 || atomicExch(&P.W.dirty[ri], 1) != 0) return;
  P.W.list_dirty[atomicAdd(&P.W.ctl->ndirty, 1)] = ri;
}

// One CTA per selected pair of the block (persistent grid over the block's
// selection slots). Per pair:
//   Update_S bookkeeping: size, internal count, member list, forwarding, and
//     QuotientGraph::Merge's touched-entry count replayed in commit order
//   keep row <- merge(row keep, row remove) with the block's removes folded
//     into their keeps, written to fresh pool space
//   every neighbour row of remove that is not a keep/remove of this block is
//     claimed once per block and rewritten in place (remove -> its keep)
// Rows of keeps and removes are only read (the keep row goes to new space),
// and a claimed neighbour row is touched by its claimant alone, so the CTAs
// need no ordering among themselves.
__global__ void __launch_bounds__(kRowsThreads) CommitKernel(CommitParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RowsSmem& R = *reinterpret_cast<RowsSmem*>(smem_raw);
  __shared__ long long new_off;
  __shared__ int folded_sum;
  const QuotientView& Q = P.Q;
  const int tid = threadIdx.x;
  const int remove_stamp = 2 * P.block_stamp + 1;
  const unsigned total = P.ctl->sel_total;
  const int win_p = P.windowed ? P.W.ctl->p : 0;
  const int win_e = P.windowed ? P.W.ctl->e : 0;
  for (unsigned idx = blockIdx.x; idx < total; idx += gridDim.x) {
    const long long slot = P.sel_list[idx];
    const int k = P.sel_keep[slot];
    const int r = P.sel_rem[slot];
    const int lr = Q.len[r];
    const int lk = Q.len[k];
    if (P.warp_pairs && lk + lr <= kWarpRow) continue;  // CommitShortKernel's pair
    const Entry* rr = Q.ent + Q.off[r];
    const Entry* rk = Q.ent + Q.off[k];
    const int my_seq = static_cast<int>(slot);
    if (tid == 0) folded_sum = 0;
    __syncthreads();
    // touched count and neighbour-row claims (block-start row of remove); a
    // claimed row goes to the short or long rewrite list
    int folded = 0;
    for (int i = tid; i < lr; i += kRowsThreads) {
      const int x = EntNb(rr[i]);
      if (x == k) continue;
      if (P.windowed) MarkTouched(P, x, win_p, win_e);
      const int sx = P.stamp[x];
      if (sx == remove_stamp && P.seq[x] < my_seq && RowLookup(rr, lr, P.partner[x]) != 0) ++folded;
      if ((sx >> 1) == P.block_stamp) continue;  // keep/remove rows are rebuilt by their own pair
      ClaimRow(P, x);
    }
    folded = WarpSumInt(folded);
    if ((tid & 31) == 0 && folded) atomicAdd(&folded_sum, folded);
    __syncthreads();
    // keep row <- merge(row k, row r), staged with keep entries first on ties
    const int L = lk + lr;
    Entry *S, *INS;
    int* D;
    if (!StageBuffers(P, R, L, &S, &D, &INS)) return;
    for (int i = tid; i < lk; i += kRowsThreads) {
      const Entry e = rk[i];
      if (P.windowed && EntNb(e) != r) MarkTouched(P, EntNb(e), win_p, win_e);
      S[i + RowLowerBound(rr, lr, EntNb(e))] = e;
    }
    for (int j = tid; j < lr; j += kRowsThreads) {
      const Entry e = rr[j];
      const int key = EntNb(e);
      int lo = 0, hi = lk;  // upper bound in row k
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (EntNb(rk[mid]) <= key) lo = mid + 1; else hi = mid;
      }
      S[j + lo] = e;
    }
    if (tid == 0) {
      const unsigned long long want = static_cast<unsigned long long>(L > 0 ? L : 1);
      const unsigned long long at = atomicAdd(P.pool_top, want);
      if (at + want > P.pool_cap) {
        RaiseError(P.err, kErrPool, k, L, 0);
        new_off = -1;
      } else {
        new_off = static_cast<long long>(at);
      }
    }
    __syncthreads();
    if (new_off < 0) return;
    const long long ekr = RowLookup(rk, lk, r);
    const int nl = RewriteRow(P, S, L, D, INS, k, r, Q.ent + new_off);
    if (tid == 0) {
      Q.internal[k] += Q.internal[r] + ekr;
      Q.internal[r] = 0;
      Q.size[k] += Q.size[r];
      Q.size[r] = 0;
      P.next[P.tail[k]] = P.head[r];
      P.tail[k] = P.tail[r];
      P.head[r] = -1;
      P.fwd[r] = k;
      Q.off[k] = new_off;
      Q.len[k] = nl;
      Q.cap[k] = L > 0 ? L : 1;
      Q.len[r] = 0;
      atomicAdd(&P.stats[kStAccepted], 1ull);
      atomicAdd(&P.stats[kStTouched],
                static_cast<unsigned long long>(2 + 3 * (lr - (ekr > 0 ? 1 : 0) - folded_sum)));
      atomicAdd(&P.stats[kStUpdateBytes], 8ull * (2ull * L + nl));
    }
    __syncthreads();
  }
}

// Selected pairs whose keep and remove rows hold at most kWarpRow entries
// together, one warp per pair: the same work as CommitKernel (claims,
// touched-entry replay, keep row = the two rows with this block's removes
// renamed to their keeps, ids k and r dropped, equal neighbours summed,
// Update_S bookkeeping), with the keep row built in registers (bitonic sort
// across the lanes, segmented sum, compaction).
__global__ void __launch_bounds__(256) CommitShortKernel(CommitParams P) {
  FollowsOn();
  const QuotientView& Q = P.Q;
  const int lane = threadIdx.x & 31;
  const int remove_stamp = 2 * P.block_stamp + 1;
  const unsigned total = P.ctl->sel_total;
  const long long nw = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; idx < total;
       idx += nw) {
    const long long slot = P.sel_list[idx];
    const int k = P.sel_keep[slot];
    const int r = P.sel_rem[slot];
    const int lr = Q.len[r];
    const int lk = Q.len[k];
    if (lk + lr > kWarpRow) continue;  // CommitKernel's pair
    const Entry* rr = Q.ent + Q.off[r];
    const Entry* rk = Q.ent + Q.off[k];
    const int my_seq = static_cast<int>(slot);
    // touched count and neighbour-row claims (lanes over the remove row)
    int folded = 0;
    if (lane < lr) {
      const int x = EntNb(rr[lane]);
      if (x != k) {
        const int sx = P.stamp[x];
        if (sx == remove_stamp && P.seq[x] < my_seq && RowLookup(rr, lr, P.partner[x]) != 0) folded = 1;
        if ((sx >> 1) != P.block_stamp) ClaimRow(P, x);
      }
    }
    const int folded_sum = __popc(__ballot_sync(0xffffffffu, folded != 0));
    // the keep row: lane i < lk holds row k's entry i, lane lk + j row r's entry j
    unsigned long long key = ~0ull;
    long long ekr = 0;
    if (lane < lk + lr) {
      const Entry e = lane < lk ? rk[lane] : rr[lane - lk];
      int id = EntNb(e);
      if (lane < lk && id == r) ekr = EntCnt(e);
      if (id != k && id != r) {
        if (P.stamp[id] == remove_stamp) id = P.partner[id];
        key = static_cast<unsigned long long>(id) << 32 | static_cast<unsigned long long>(EntCnt(e));
      }
    }
    ekr = WarpMax(ekr);
    key = WarpBitonicSortAsc(key, lane);
    const bool valid = key != ~0ull;
    const int id = static_cast<int>(key >> 32);
    const long long c = valid ? static_cast<long long>(key & 0xffffffffull) : 0;
    const int prev = __shfl_up_sync(0xffffffffu, id, 1);
    const bool head = valid && (lane == 0 || prev != id);
    long long sum = c;
    bool more = head;
    for (int j = 1; j < 32; ++j) {
      const int idj = __shfl_down_sync(0xffffffffu, id, j);
      const long long cj = __shfl_down_sync(0xffffffffu, c, j);
      if (more && lane + j < 32 && idj == id) {
        sum += cj;
      } else {
        more = false;
      }
      if (!__any_sync(0xffffffffu, more)) break;
    }
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int nl = __popc(heads);
    const int L = lk + lr;
    long long new_off = 0;
    if (lane == 0) {
      const unsigned long long want = static_cast<unsigned long long>(L > 0 ? L : 1);
      const unsigned long long at = atomicAdd(P.pool_top, want);
      if (at + want > P.pool_cap) {
        RaiseError(P.err, kErrPool, k, L, 0);
        new_off = -1;
      } else {
        new_off = static_cast<long long>(at);
      }
    }
    new_off = __shfl_sync(0xffffffffu, new_off, 0);
    if (new_off < 0) continue;
    if (head) Q.ent[new_off + __popc(heads & ((1u << lane) - 1u))] = MakeEnt(id, sum);
    if (lane == 0) {
      Q.internal[k] += Q.internal[r] + ekr;
      Q.internal[r] = 0;
      Q.size[k] += Q.size[r];
      Q.size[r] = 0;
      P.next[P.tail[k]] = P.head[r];
      P.tail[k] = P.tail[r];
      P.head[r] = -1;
      P.fwd[r] = k;
      Q.off[k] = new_off;
      Q.len[k] = nl;
      Q.cap[k] = L > 0 ? L : 1;
      Q.len[r] = 0;
      atomicAdd(&P.stats[kStAccepted], 1ull);
      atomicAdd(&P.stats[kStTouched],
                static_cast<unsigned long long>(2 + 3 * (lr - (ekr > 0 ? 1 : 0) - folded_sum)));
      atomicAdd(&P.stats[kStUpdateBytes], 8ull * (2ull * L + nl));
    }
  }
}

// A claimed neighbour row of kWarpRow < L <= kWarpRowMax entries, one warp,
// staged in the warp's slice S of shared memory. Only the entries of
// supernodes removed in this block change: each is renamed to its keep
// partner and summed into the partner's entry when the row has one, else
// inserted (INS, sorted). Every other entry keeps its order, so its new
// position is its old one less the renamed entries before it plus the
// inserted entries below it: no sort of the row. Returns the new length.
__device__ int RewriteMediumRow(const CommitParams& P, Entry* row, int L, Entry* S, Entry* INS) {
  constexpr int kChunks = kWarpRowMax / 32;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int remove_stamp = 2 * P.block_stamp + 1;
  for (int j = lane; j < L; j += 32) S[j] = row[j];
  __syncwarp();
  unsigned rm[kChunks];  // renamed entries of each 32-entry chunk (warp-uniform)
  int m = 0;             // inserted entries so far
#pragma unroll
  for (int t = 0; t < kChunks; ++t) {
    const int j = lane + 32 * t;
    bool renamed = false, insert = false;
    Entry ins = 0;
    if (j < L) {
      const Entry e = S[j];
      const int id = EntNb(e);
      if (P.stamp[id] == remove_stamp) {
        renamed = true;
        const int kp = P.partner[id];
        const long long c = EntCnt(e);
        int lo = 0, hi = L;  // kp among the staged ids (only counts change meanwhile)
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (EntNb(S[mid]) < kp) lo = mid + 1; else hi = mid;
        }
        if (lo < L && EntNb(S[lo]) == kp) {
          atomicAdd(reinterpret_cast<unsigned long long*>(&S[lo]), static_cast<unsigned long long>(c));
        } else {
          insert = true;
          ins = MakeEnt(kp, c);
        }
      }
    }
    rm[t] = __ballot_sync(0xffffffffu, renamed);
    const unsigned im = __ballot_sync(0xffffffffu, insert);
    if (insert) INS[m + __popc(im & lt)] = ins;
    m += __popc(im);
  }
  // the inserted entries in id order (distinct ids: one remove per keep)
  int pow2 = 1;
  while (pow2 < m) pow2 <<= 1;
  for (int i = m + lane; i < pow2; i += 32) INS[i] = ~0ull;
  __syncwarp();
  for (int k = 2; k <= pow2; k <<= 1) {
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int i = lane; i < pow2; i += 32) {
        const int ixj = i ^ jj;
        if (ixj > i) {
          const Entry a = INS[i];
          const Entry b = INS[ixj];
          if ((a > b) == ((i & k) == 0)) {
            INS[i] = b;
            INS[ixj] = a;
          }
        }
      }
      __syncwarp();
    }
  }
  // renamed entries before position q of the staged row
  auto dropped_before = [&](int q) {
    int d = 0;
#pragma unroll
    for (int t = 0; t < kChunks; ++t) {
      if (32 * t + 32 <= q) d += __popc(rm[t]);
      else if (32 * t < q) d += __popc(rm[t] & ((1u << (q - 32 * t)) - 1u));
    }
    return d;
  };
  int k_total = 0;
#pragma unroll
  for (int t = 0; t < kChunks; ++t) k_total += __popc(rm[t]);
#pragma unroll
  for (int t = 0; t < kChunks; ++t) {
    const int j = lane + 32 * t;
    if (j < L && !((rm[t] >> lane) & 1u)) {
      const Entry e = S[j];
      int lo = 0, hi = m;  // inserted entries below this id
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (EntNb(INS[mid]) < EntNb(e)) lo = mid + 1; else hi = mid;
      }
      row[j - dropped_before(j) + lo] = e;
    }
  }
  for (int i = lane; i < m; i += 32) {
    const Entry e = INS[i];
    int lo = 0, hi = L;  // staged entries below the inserted id
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (EntNb(S[mid]) < EntNb(e)) lo = mid + 1; else hi = mid;
    }
    row[lo - dropped_before(lo) + i] = e;
  }
  __syncwarp();
  return L - k_total + m;
}

// Claimed neighbour rows of at most kWarpRowMax entries, one warp per row.
// Rows of at most kWarpRow entries: each entry of a supernode removed in this
// block is renamed to its keep partner, the row is sorted by neighbour
// (register bitonic sort), equal neighbours are summed and the row is
// compacted in place (it can only shrink). Longer ones: RewriteMediumRow with
// the warp's slice of the CTA's shared memory.
__device__ void RewriteShortRows(const CommitParams& P, RowsSmem& R) {
  const QuotientView& Q = P.Q;
  const int lane = threadIdx.x & 31;
  const int warp_in_cta = threadIdx.x >> 5;
  const unsigned cnt = P.ctl->short_cnt;
  const int remove_stamp = 2 * P.block_stamp + 1;
  const long long nw = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  unsigned long long rows = 0, entries = 0, bytes = 0;
  for (long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; idx < cnt; idx += nw) {
    const int x = P.rows_short[idx];
    Entry* row = Q.ent + Q.off[x];
    const int lx = Q.len[x];
    if (lx > kWarpRow) {
      const int nl = RewriteMediumRow(P, row, lx, R.s + warp_in_cta * kWarpRowMax, R.ins + warp_in_cta * kWarpRowMax);
      if (lane == 0) {
        Q.len[x] = nl;
        ++rows;
        entries += static_cast<unsigned long long>(lx);
        bytes += 8ull * static_cast<unsigned long long>(lx + nl);
      }
      continue;
    }
    unsigned long long key = ~0ull;
    if (lane < lx) {
      const Entry e = row[lane];
      int id = EntNb(e);
      if (P.stamp[id] == remove_stamp) id = P.partner[id];
      key = static_cast<unsigned long long>(id) << 32 | static_cast<unsigned long long>(EntCnt(e));
    }
    key = WarpBitonicSortAsc(key, lane);
    const bool valid = key != ~0ull;
    const int id = static_cast<int>(key >> 32);
    const long long c = valid ? static_cast<long long>(key & 0xffffffffull) : 0;
    const int prev = __shfl_up_sync(0xffffffffu, id, 1);
    const bool head = valid && (lane == 0 || prev != id);
    long long total = c;
    bool more = head;
    for (int j = 1; j < 32; ++j) {
      const int idj = __shfl_down_sync(0xffffffffu, id, j);
      const long long cj = __shfl_down_sync(0xffffffffu, c, j);
      if (more && lane + j < 32 && idj == id) {
        total += cj;
      } else {
        more = false;
      }
      if (!__any_sync(0xffffffffu, more)) break;
    }
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    if (head) row[__popc(heads & ((1u << lane) - 1u))] = MakeEnt(id, total);
    const int nl = __popc(heads);
    if (lane == 0) {
      Q.len[x] = nl;
      ++rows;
      entries += static_cast<unsigned long long>(lx);
      bytes += 8ull * static_cast<unsigned long long>(lx + nl);
    }
  }
  if (lane == 0 && rows) {
    atomicAdd(&P.stats[kStRowsRewritten], rows);
    atomicAdd(&P.stats[kStRowEntriesRewritten], entries);
    atomicAdd(&P.stats[kStUpdateBytes], bytes);
  }
}

// Claimed neighbour rows of kWarpRowMax < L <= kRowSmem entries, one CTA per
// row, staged in shared memory.
__device__ void RewriteLongRows(const CommitParams& P, RowsSmem& R) {
  const QuotientView& Q = P.Q;
  const unsigned cnt = P.ctl->long_cnt;
  for (unsigned idx = blockIdx.x; idx < cnt; idx += gridDim.x) {
    const int x = P.rows_long[idx];
    Entry* rowp = Q.ent + Q.off[x];
    const int lx = Q.len[x];
    for (int i = threadIdx.x; i < lx; i += kRowsThreads) R.s[i] = rowp[i];
    __syncthreads();
    const int nlx = RewriteRow(P, R.s, lx, R.d, R.ins, -1, -1, rowp);
    if (threadIdx.x == 0) {
      Q.len[x] = nlx;
      atomicAdd(&P.stats[kStRowsRewritten], 1ull);
      atomicAdd(&P.stats[kStRowEntriesRewritten], static_cast<unsigned long long>(lx));
      atomicAdd(&P.stats[kStUpdateBytes], 8ull * (lx + nlx));
    }
    __syncthreads();
  }
}

// First position of a sorted row whose neighbour is >= x, by the whole warp.
__device__ __forceinline__ int WarpRowLowerBound(const Entry* row, int len, int x) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = len;  // the answer lies in [lo, hi]
  while (lo < hi) {
    // 32 probes of [lo, hi), non-decreasing over the lanes
    const int p = lo + static_cast<int>((static_cast<long long>(hi - lo) * lane) >> 5);
    const int k = __popc(__ballot_sync(0xffffffffu, EntNb(row[p]) < x));  // lanes 0..k-1 are below
    const int below = __shfl_sync(0xffffffffu, p, k > 0 ? k - 1 : 0);
    const int above = __shfl_sync(0xffffffffu, p, k < 32 ? k : 31);
    if (k < 32) hi = above;
    if (k > 0) lo = below + 1; else hi = lo;
  }
  return lo;
}

// First step of the longer rows, a warp per kHugeUnit entries: marks the
// entries of supernodes removed in this block, adds each one's count to its
// keep's entry in the row (ids stay in place, so the row stays searchable) or
// lists it for insertion.
__device__ void ScanHugeRows(const CommitParams& P) {
  constexpr int kDeep = 8;
  const QuotientView& Q = P.Q;
  const int lane = threadIdx.x & 31;
  const unsigned units = P.ctl->huge_units;
  const int remove_stamp = 2 * P.block_stamp + 1;
  const unsigned nw = (gridDim.x * blockDim.x) >> 5;
  for (unsigned u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < units; u += nw) {
    const int2 unit = P.huge_units[u];
    HugeRow* h = P.rows_huge + unit.x;
    const int x = h->x, len = h->len;
    unsigned* mask = h->mask;
    Entry* row = Q.ent + Q.off[x];
    const int end = unit.y + kHugeUnit < len ? unit.y + kHugeUnit : len;
    for (int i0 = unit.y; i0 < end; i0 += 32 * kDeep) {
      Entry e[kDeep];
      int st[kDeep];
#pragma unroll
      for (int d = 0; d < kDeep; ++d) {
        const int i = i0 + 32 * d + lane;
        e[d] = i < end ? row[i] : 0;
      }
#pragma unroll
      for (int d = 0; d < kDeep; ++d) {
        const int i = i0 + 32 * d + lane;
        st[d] = i < end ? P.stamp[EntNb(e[d])] : 0;
      }
#pragma unroll
      for (int d = 0; d < kDeep; ++d) {
        const bool renamed = st[d] == remove_stamp;
        const unsigned m = __ballot_sync(0xffffffffu, renamed);
        if (lane == 0 && i0 + 32 * d < end) mask[(i0 >> 5) + d] = m;
        // the keep's place in the row: by the whole warp for one or two of them
        // (three rounds of loads instead of a dozen), else each lane its own
        int at = 0;
        const int kp = renamed ? P.partner[EntNb(e[d])] : 0;
        if (__popc(m) <= 2) {
          for (unsigned rest = m; rest; rest &= rest - 1) {
            const int src = __ffs(rest) - 1;
            const int x = WarpRowLowerBound(row, len, __shfl_sync(0xffffffffu, kp, src));
            if (lane == src) at = x;
          }
        } else if (renamed) {
          at = RowLowerBound(row, len, kp);
        }
        if (renamed) {
          const long long c = EntCnt(e[d]);
          const int p = at;
          if (p < len && EntNb(row[p]) == kp) {
            atomicAdd(&row[p], static_cast<unsigned long long>(c));
          } else {
            h->ins[atomicAdd(&h->nins, 1)] = MakeEnt(kp, c);
          }
        }
      }
    }
  }
}

// All claimed neighbour rows of a block: the long ones by whole CTAs, then the
// first step of the longest, then the short ones by single warps.
__global__ void __launch_bounds__(kRowsThreads) RewriteRowsKernel(CommitParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RowsSmem& R = *reinterpret_cast<RowsSmem*>(smem_raw);
  ScanHugeRows(P);
  RewriteLongRows(P, R);
  __syncthreads();  // the shared buffers pass from the CTA's long rows to its warps
  RewriteShortRows(P, R);
}

struct HugeSmem {
  Entry ins[kHugeChunk];
  int at[kHugeChunk];  // per inserted entry: first staying or renamed entry above it
  unsigned word[kHugeChunk / 32];
  int before[kHugeChunk / 32];  // renamed entries of the chunk before each mask word
  int deleted;                  // renamed entries of the chunk
};

// Renamed entries before position p of the row: `base` of them before the
// chunk, whose mask words are staged.
__device__ __forceinline__ int RenamedBefore(const HugeSmem& H, int base, int p_in_chunk) {
  const int w = p_in_chunk >> 5;
  return base + H.before[w] + __popc(H.word[w] & ((1u << (p_in_chunk & 31)) - 1u));
}

// Stages a chunk's mask words and their running counts; all threads, with
// barriers (words past the row read as zero).
__device__ void StageMask(HugeSmem& H, const unsigned* mask, int base, int len) {
  constexpr int kWords = kHugeChunk / 32;
  const int words = (len + 31) / 32;
  for (int w = threadIdx.x; w < kWords; w += kHugeThreads) {
    H.word[w] = base / 32 + w < words ? mask[base / 32 + w] : 0u;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    constexpr int kPer = kWords / 32;
    int v[kPer], sum = 0;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      v[u] = __popc(H.word[threadIdx.x * kPer + u]);
      sum += v[u];
    }
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (static_cast<int>(threadIdx.x) >= o) incl += y;
    }
    int run = incl - sum;
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      H.before[threadIdx.x * kPer + u] = run;
      run += v[u];
    }
    if (threadIdx.x == 31) H.deleted = incl;
  }
  __syncthreads();
}

// Second step of the longest rows, a CTA per row: without its renamed entries
// and with the inserted ones, in place. An entry moves left by the renamed
// entries before it and right by the inserted ones below it, at most
// kHugeChunk of them: every chunk is in registers before the one before it is
// written, so nothing unread is overwritten. (A row with more to insert
// goes through a copy.) One CTA with everything
// staged in global memory took 431 us for a row of 27,500 entries, most of it
// in dependent loads; the split takes the loads of the scan off that chain.
// The last CTA clears the block control words for the next block: all their
// readers are done by then.
__global__ void __launch_bounds__(kHugeThreads) RewriteHugeKernel(CommitParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  HugeSmem& H = *reinterpret_cast<HugeSmem*>(smem_raw);
  __shared__ bool last;
  const QuotientView& Q = P.Q;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const unsigned cnt = P.ctl->huge_cnt;
  for (unsigned idx = blockIdx.x; idx < cnt; idx += gridDim.x) {
    const HugeRow h = P.rows_huge[idx];
    const int len = h.len, m = h.nins;
    Entry* row = Q.ent + Q.off[h.x];
    int pow2 = 1;
    while (pow2 < m) pow2 <<= 1;
    const bool in_place = m <= kHugeChunk;
    Entry* ins = in_place ? H.ins : h.ins;
    if (in_place) {
      for (int j = tid; j < m; j += kHugeThreads) ins[j] = h.ins[j];
    }
    for (int j = m + tid; j < pow2; j += kHugeThreads) ins[j] = ~0ull;
    __syncthreads();
    if (m > 1) CtaBitonicSort(ins, pow2);
    int deleted = 0;  // renamed entries before the chunk
    if (in_place) {
      for (int j = tid; j < m; j += kHugeThreads) H.at[j] = RowLowerBound(row, len, EntNb(ins[j]));
      Entry cur[kHugePer], nxt[kHugePer];
#pragma unroll
      for (int d = 0; d < kHugePer; ++d) {
        const int i = d * kHugeThreads + tid;
        cur[d] = i < len ? row[i] : 0;
      }
      for (int base = 0; base < len; base += kHugeChunk) {
#pragma unroll
        for (int d = 0; d < kHugePer; ++d) {
          const int i = base + kHugeChunk + d * kHugeThreads + tid;
          nxt[d] = i < len ? row[i] : 0;
        }
        StageMask(H, h.mask, base, len);
        // ends with a barrier: the next chunk is in registers everywhere
#pragma unroll
        for (int d = 0; d < kHugePer; ++d) {
          const int in = d * kHugeThreads + tid;
          const int i = base + in;
          if (i < len && !((H.word[in >> 5] >> lane) & 1u)) {
            int lo = 0, hi = m;  // inserted entries at or before this position
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              if (H.at[mid] <= i) lo = mid + 1; else hi = mid;
            }
            const int to = i - RenamedBefore(H, deleted, in) + lo;
            if (to != i) row[to] = cur[d];
          }
        }
        const bool last_chunk = base + kHugeChunk >= len;
        for (int j = tid; j < m; j += kHugeThreads) {
          const int p = H.at[j];
          if (p < base || (p >= base + kHugeChunk && !last_chunk)) continue;
          // p == len: past the last word of a full last chunk
          const int before = p - base < kHugeChunk ? RenamedBefore(H, deleted, p - base) : deleted + H.deleted;
          row[j + p - before] = ins[j];
        }
        deleted += H.deleted;
        __syncthreads();  // the staged words are replaced
#pragma unroll
        for (int d = 0; d < kHugePer; ++d) cur[d] = nxt[d];
      }
    } else {
      for (int i = tid; i < len; i += kHugeThreads) h.copy[i] = row[i];
      __syncthreads();
      for (int base = 0; base < len; base += kHugeChunk) {
        StageMask(H, h.mask, base, len);
        const bool last_chunk = base + kHugeChunk >= len;
        for (int in = tid; in < kHugeChunk && base + in < len; in += kHugeThreads) {
          if ((H.word[in >> 5] >> (in & 31)) & 1u) continue;
          const Entry e = h.copy[base + in];
          row[base + in - RenamedBefore(H, deleted, in) + RowLowerBound(ins, m, EntNb(e))] = e;
        }
        for (int j = tid; j < m; j += kHugeThreads) {
          const int p = RowLowerBound(h.copy, len, EntNb(ins[j]));
          if (p < base || (p >= base + kHugeChunk && !last_chunk)) continue;
          const int before = p - base < kHugeChunk ? RenamedBefore(H, deleted, p - base) : deleted + H.deleted;
          row[j + p - before] = ins[j];
        }
        deleted += H.deleted;
        __syncthreads();
      }
    }
    if (tid == 0) {
      const int nl = len - deleted + m;
      Q.len[h.x] = nl;
      atomicAdd(&P.stats[kStRowsRewritten], 1ull);
      atomicAdd(&P.stats[kStRowEntriesRewritten], static_cast<unsigned long long>(len));
      atomicAdd(&P.stats[kStUpdateBytes], 8ull * (len + nl));
    }
    __syncthreads();
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(P.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (last && tid == 0) {
    P.ctl->scratch_top = 0;
    P.ctl->short_cnt = 0;
    P.ctl->long_cnt = 0;
    P.ctl->huge_cnt = 0;
    P.ctl->huge_units = 0;
    P.ctl->sel_total = 0;
    P.ctl->work_next[0] = 0;
    P.ctl->work_next[1] = 0;
    P.ctl->work_next[2] = 0;
    *P.ticket = 0u;
  }
  if (last && P.windowed) BuildLists(P.W);
}

__global__ void ScatterGroupKernel(const int* __restrict__ q, const int* __restrict__ idx, int g,
                                   int* __restrict__ group_of, int* __restrict__ idx_in_group) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < g) {
    group_of[q[i]] = 0;
    idx_in_group[q[i]] = idx[i];
  }
}

__global__ void RelabelKernel(int* __restrict__ label, const int* __restrict__ fwd, int n) {
  FollowsOn();
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) label[v] = fwd[label[v]];
}

}  // namespace

// --------------------------------------------------------------- host side

void Engine::ConfigureKernels() {
  window_tables_ = kWindowTables;
  row_sum_arcs_ = kFusedMaxArcs;
  CheckCuda(cudaFuncSetAttribute(PrepareKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(PrepSmem))), "prepare smem attribute");
  CheckCuda(cudaFuncSetAttribute(PrepareSmallKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(SmallSmem))), "prepare-small smem attribute");
  CheckCuda(cudaFuncSetAttribute(SelectMatchKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 8 * kMatchSmemKeys), "select smem attribute");
  CheckCuda(cudaFuncSetAttribute(CommitKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(RowsSmem))), "commit smem attribute");
  CheckCuda(cudaFuncSetAttribute(RewriteRowsKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(RowsSmem))), "rewrite smem attribute");
  CheckCuda(cudaFuncSetAttribute(RewriteHugeKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(HugeSmem))), "long-row rewrite smem attribute");
  CheckCuda(cudaFuncSetAttribute(MediumKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(MediumSmem))), "medium smem attribute");
  CheckCuda(cudaFuncSetAttribute(WindowEvalKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(EvalSmem))), "window evaluation smem attribute");
  CheckCuda(cudaFuncSetAttribute(WindowSelectKernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 8 * kMatchSmemKeys), "window selection smem attribute");
  // the queue-fed kernels launch exactly the CTAs that fit on the GPU at once
  int sms = 0, per_sm = 0;
  CheckCuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, cfg_.device), "SM count");
  CheckCuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, PrepareAccumKernel, kAccumThreads, 0),
            "accumulate occupancy");
  accum_grid_ = std::max(1, sms * per_sm);
  CheckCuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ScoreKernel, kScoreThreads, 0), "score occupancy");
  score_grid_ = std::max(1, sms * per_sm);
}

void Engine::SetLimit(int which, int64_t value) {
  const int64_t most = which == kLimitWindowTables ? INT64_MAX : which == kLimitRowSumArcs ? kFusedMaxArcs : 0;
  if (value < 1 || value > most) throw std::invalid_argument("unknown limit or value out of range");
  (which == kLimitWindowTables ? window_tables_ : row_sum_arcs_) = value;
}

// Per-iteration layout: the groups with >= 2 members in Divide order, their
// candidate / selection capacities (min(C(g,2), g*top_k) and g/2) as prefix
// offsets, pair-table offsets restarting at every block, and for every block
// the range of its real groups (empty blocks do no work).
namespace {

// ---- the plan of a one-block iteration, on the device ----
// Per Divide group, the classification and offsets of the host plan
// (PrepareIterationBuffers with one block of every group): tile sums, one
// CTA scanning the tile sums, then every real group's entries scattered into
// the lists in group order.
constexpr int kPlanThreads = 256;
constexpr int kPlanItems = 8;
constexpr int kPlanTile = kPlanThreads * kPlanItems;
enum PlanScalar : int {
  kPlanR = 0, kPlanCand, kPlanSel, kPlanSmall, kPlanBig, kPlanMembers, kPlanSlots, kPlanMat,
  kPlanSelSmall, kPlanSelMid, kPlanSelBig, kPlanMed, kPlanSmallBase, kPlanScalars = kPlanSmallBase + 4
};
// The small-group list is laid out by member count, largest class first
// (more than 24, 17..24, 9..16, at most 8 members): the longest warps start
// first instead of forming the prepare kernel's tail.
constexpr int kPlanSmallClasses = 4;
__device__ __forceinline__ int SmallClass(int g) { return g > 24 ? 0 : g > 16 ? 1 : g > 8 ? 2 : 3; }

// What the medium groups do: candidates for the later passes like the rest
// (the ranker prunes them there), or everything in one kernel (medium.cuh);
// windows of blocks have their own limits.
enum PlanMode : int { kPlanLists = 0, kPlanFused = 1, kPlanWindows = 2 };

struct PlanSums {
  long long cand, sel, moff, soff, mat;
  int real, med, big, ssmall, smid, sbig;
  int small[kPlanSmallClasses];
};

struct PlanSumOp {
  __device__ __forceinline__ PlanSums operator()(const PlanSums& a, const PlanSums& b) const {
    PlanSums r;
    r.cand = a.cand + b.cand;
    r.sel = a.sel + b.sel;
    r.moff = a.moff + b.moff;
    r.soff = a.soff + b.soff;
    r.mat = a.mat + b.mat;
    r.real = a.real + b.real;
#pragma unroll
    for (int c = 0; c < kPlanSmallClasses; ++c) r.small[c] = a.small[c] + b.small[c];
    r.med = a.med + b.med;
    r.big = a.big + b.big;
    r.ssmall = a.ssmall + b.ssmall;
    r.smid = a.smid + b.smid;
    r.sbig = a.sbig + b.sbig;
    return r;
  }
};

__device__ __forceinline__ PlanSums PlanZero() {
  PlanSums z;
  z.cand = z.sel = z.moff = z.soff = z.mat = 0;
  z.real = z.med = z.big = z.ssmall = z.smid = z.sbig = 0;
#pragma unroll
  for (int c = 0; c < kPlanSmallClasses; ++c) z.small[c] = 0;
  return z;
}

// one group's contribution: the same rules as the host plan
__device__ __forceinline__ PlanSums PlanOfGroup(int g, unsigned e, long long k, int mode, int one_class) {
  PlanSums f = PlanZero();
  if (g < 2) return f;
  const long long gl = g;
  f.real = 1;
  f.cand = gl * (gl - 1) / 2 < gl * k ? gl * (gl - 1) / 2 : gl * k;
  f.sel = gl / 2;
  const bool windowed = mode == kPlanWindows;
  if (windowed ? WindowSmall(g, e) : g <= kSmallGroup && e <= static_cast<unsigned>(kSmallStage)) {
    f.small[one_class ? 0 : SmallClass(g)] = 1;
  } else if (mode == kPlanFused && MediumFits(g, e)) {
    f.med = 1;  // with its selection
    return f;
  } else {
    f.big = 1;
    f.moff = gl;
    f.soff = e > static_cast<unsigned>(kSmemEntries) || g > kSmemMaxGroup ? static_cast<long long>(e) : 0;
    f.mat = windowed ? WindowBytes(gl, e) : (OldCostOffset(gl * gl) + 8 * gl + 255) & ~255ll;
  }
  if (g <= kSelectSmallGroup) {
    f.ssmall = 1;
  } else if (g <= kSelectMidGroup) {
    f.smid = 1;
  } else {
    f.sbig = 1;
  }
  return f;
}

struct PlanParams {
  const int* glen;
  const unsigned* gent;
  long long G;
  long long top_k;
  int mode;  // PlanMode
  PlanSums* tile_sums;
  PlanSums* tile_off;
  int tiles;
  long long* scalars;
  int* real;
  long long* cand_off;
  long long* sel_off;
  long long* mat_off;
  int* small;
  int* med;
  int* big;
  long long* big_moff;
  long long* soff;
  int* sel_small;
  int* sel_mid;
  int* sel_big;
  // several blocks: the sums before each block's first group, and the small
  // groups in one class, so that every list is in group order
  PlanSums* block_sums;
  long long batch;
  int one_class;
  int* ri_of;  // per Divide group: its position, -1 for a group of one (nullptr: not needed)
};

__global__ void __launch_bounds__(kPlanThreads) PlanTileKernel(PlanParams P) {
  FollowsOn();
  using Reduce = cub::BlockReduce<PlanSums, kPlanThreads>;
  __shared__ typename Reduce::TempStorage tmp;
  const long long base = static_cast<long long>(blockIdx.x) * kPlanTile + threadIdx.x * kPlanItems;
  PlanSums acc = PlanZero();
  for (int j = 0; j < kPlanItems; ++j) {
    const long long gi = base + j;
    if (gi >= P.G) break;
    const PlanSums f = PlanOfGroup(P.glen[gi], P.gent[gi], P.top_k, P.mode, P.one_class);
    acc = PlanSumOp()(acc, f);
  }
  const PlanSums t = Reduce(tmp).Reduce(acc, PlanSumOp());
  if (threadIdx.x == 0) P.tile_sums[blockIdx.x] = t;
}

// one CTA: exclusive offsets of the tiles, the totals, and the closing
// entries of the offset arrays
__global__ void __launch_bounds__(kPlanThreads) PlanScanKernel(PlanParams P) {
  FollowsOn();
  using Scan = cub::BlockScan<PlanSums, kPlanThreads>;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ PlanSums carry;
  if (threadIdx.x == 0) carry = PlanZero();
  __syncthreads();
  for (int t0 = 0; t0 < P.tiles; t0 += kPlanThreads) {
    const int t = t0 + threadIdx.x;
    const PlanSums v = t < P.tiles ? P.tile_sums[t] : PlanZero();
    PlanSums ex, total;
    Scan(tmp).ExclusiveScan(v, ex, PlanZero(), PlanSumOp(), total);
    const PlanSums c = carry;
    if (t < P.tiles) P.tile_off[t] = PlanSumOp()(c, ex);
    __syncthreads();
    if (threadIdx.x == 0) carry = PlanSumOp()(c, total);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const PlanSums T = carry;
    long long* s = P.scalars;
    s[kPlanR] = T.real;
    s[kPlanCand] = T.cand;
    s[kPlanSel] = T.sel;
    long long sb = 0;
    for (int c = 0; c < kPlanSmallClasses; ++c) {
      s[kPlanSmallBase + c] = sb;
      sb += T.small[c];
    }
    s[kPlanSmall] = sb;
    s[kPlanMed] = T.med;
    s[kPlanBig] = T.big;
    s[kPlanMembers] = T.moff;
    s[kPlanSlots] = T.soff;
    s[kPlanMat] = T.mat;
    s[kPlanSelSmall] = T.ssmall;
    s[kPlanSelMid] = T.smid;
    s[kPlanSelBig] = T.sbig;
    P.cand_off[T.real] = T.cand;
    P.sel_off[T.real] = T.sel;
    P.mat_off[T.real] = T.mat;
    P.big_moff[T.big] = T.moff;
    P.soff[T.big] = T.soff;
  }
}

__global__ void __launch_bounds__(kPlanThreads) PlanScatterKernel(PlanParams P) {
  FollowsOn();
  using Scan = cub::BlockScan<PlanSums, kPlanThreads>;
  __shared__ typename Scan::TempStorage tmp;
  const long long base = static_cast<long long>(blockIdx.x) * kPlanTile + threadIdx.x * kPlanItems;
  int g[kPlanItems];
  unsigned e[kPlanItems];
  PlanSums acc = PlanZero();
#pragma unroll
  for (int j = 0; j < kPlanItems; ++j) {
    const long long gi = base + j;
    g[j] = gi < P.G ? P.glen[gi] : 0;
    e[j] = gi < P.G ? P.gent[gi] : 0u;
    acc = PlanSumOp()(acc, PlanOfGroup(g[j], e[j], P.top_k, P.mode, P.one_class));
  }
  PlanSums off;
  Scan(tmp).ExclusiveScan(acc, off, P.tile_off[blockIdx.x], PlanSumOp());
#pragma unroll
  for (int j = 0; j < kPlanItems; ++j) {
    const PlanSums f = PlanOfGroup(g[j], e[j], P.top_k, P.mode, P.one_class);
    if (P.block_sums && base + j < P.G && (base + j) % P.batch == 0) P.block_sums[(base + j) / P.batch] = off;
    if (P.ri_of && base + j < P.G) P.ri_of[base + j] = f.real ? off.real : -1;
    if (f.real) {
      const int ri = off.real;
      P.real[ri] = static_cast<int>(base + j);
      P.cand_off[ri] = off.cand;
      P.sel_off[ri] = off.sel;
      P.mat_off[ri] = off.mat;
      if (f.med) {
        P.med[off.med] = ri;
      } else if (!f.big) {
        const int c = P.one_class ? 0 : SmallClass(g[j]);
        P.small[P.scalars[kPlanSmallBase + c] + off.small[c]] = ri;
      } else {
        P.big[off.big] = ri;
        P.big_moff[off.big] = off.moff;
        P.soff[off.big] = off.soff;
      }
      if (f.ssmall) {
        P.sel_small[off.ssmall] = ri;
      } else if (f.smid) {
        P.sel_mid[off.smid] = ri;
      } else if (f.sbig) {
        P.sel_big[off.sbig] = ri;
      }
    }
    off = PlanSumOp()(off, f);
  }
}

}  // namespace

// Medium groups go from rows to selected pairs in one kernel where there are
// enough of them, unless something wants to see their candidates (the ranker)
// or the exact gain needs the rows again.
bool Engine::FusedOn() const { return RowSumsOn() && !cfg_.ranker; }

bool Engine::PlanFused() const {
  return FusedOn() && std::min<long long>(cfg_.group_batch_size, n_groups_) >= kMedMinAll;
}

void Engine::PrepareIterationBuffers() {
  const int64_t G = n_groups_;
  h_real_.clear();
  h_block_rg_.clear();
  const int64_t bs = cfg_.group_batch_size;
  const long long k = cfg_.top_k > 0 ? cfg_.top_k : 1;
  for (int64_t b0 = 0; b0 < G; b0 += bs) {
    const int64_t b1 = std::min(G, b0 + bs);
    h_block_rg_.push_back(static_cast<int>(h_real_.size()));
    for (int64_t gi = b0; gi < b1; ++gi) {
      if (h_glen_[static_cast<size_t>(gi)] >= 2) h_real_.push_back(static_cast<int>(gi));
    }
  }
  h_block_rg_.push_back(static_cast<int>(h_real_.size()));
  const size_t R = h_real_.size();
  h_cand_off_.assign(R + 1, 0);
  h_sel_off_.assign(R + 1, 0);
  h_mat_off_.assign(R + 1, 0);
  long long max_mat = 0;
  for (size_t ri = 0; ri < R; ++ri) {
    const long long g = h_glen_[static_cast<size_t>(h_real_[ri])];
    // (a member listed twice ties with itself, and more than k partners are kept)
    h_cand_off_[ri + 1] = h_cand_off_[ri] + (members_repeat_ ? g * (g - 1) / 2 : std::min(g * (g - 1) / 2, g * k));
    h_sel_off_[ri + 1] = h_sel_off_[ri] + g / 2;
  }
  // groups of at most kSmallGroup members whose rows fit the staging buffer
  // go to the warp-per-group kernel; only the others need pair tables in
  // global memory
  h_small_.clear();
  h_big_.clear();
  h_big_moff_.assign(1, 0);
  h_soff_.assign(1, 0);
  h_med_.clear();
  h_block_small_.clear();
  h_block_med_.clear();
  h_block_big_.clear();
  std::vector<long long> block_mat;
  auto is_small = [&](int ri) {
    const size_t gid = static_cast<size_t>(h_real_[static_cast<size_t>(ri)]);
    return h_glen_[gid] <= kSmallGroup && h_gent_[gid] <= static_cast<unsigned>(kSmallStage);
  };
  auto is_medium = [&](int ri) {
    const size_t gid = static_cast<size_t>(h_real_[static_cast<size_t>(ri)]);
    return !is_small(ri) && MediumFits(h_glen_[gid], h_gent_[gid]);
  };
  h_block_fused_.clear();
  for (size_t b = 0; b + 1 < h_block_rg_.size(); ++b) {
    h_block_small_.push_back(static_cast<int>(h_small_.size()));
    h_block_med_.push_back(static_cast<int>(h_med_.size()));
    h_block_big_.push_back(static_cast<int>(h_big_.size()));
    int medium = 0;
    if (FusedOn()) {
      for (int ri = h_block_rg_[b]; ri < h_block_rg_[b + 1]; ++ri) medium += is_medium(ri) ? 1 : 0;
    }
    const bool fused = medium >= kMedMinGroups;
    h_block_fused_.push_back(fused ? 1 : 0);
    // a small block with any big group sends all its groups to the big path
    // (one prepare path, fewer launches; the same candidates)
    bool all_big = false;
    if (h_block_rg_[b + 1] - h_block_rg_[b] <= kFewGroups) {
      for (int ri = h_block_rg_[b]; ri < h_block_rg_[b + 1] && !all_big; ++ri) all_big = !is_small(ri);
    }
    long long off = 0;
    for (int ri = h_block_rg_[b]; ri < h_block_rg_[b + 1]; ++ri) {
      const size_t gid = static_cast<size_t>(h_real_[static_cast<size_t>(ri)]);
      const long long g = h_glen_[gid];
      // rows counted at Divide time (rows of supernodes not merged yet only
      // shrink during an iteration, so the count is an upper bound)
      if (!all_big && is_small(ri)) {
        h_small_.push_back(ri);
        continue;
      }
      if (fused && is_medium(ri)) {
        h_med_.push_back(ri);
        continue;
      }
      h_big_.push_back(ri);
      h_big_moff_.push_back(h_big_moff_.back() + g);
      // groups beyond the shared-memory bucket table get sort slots
      const long long e_ub = h_gent_[gid];
      h_soff_.push_back(h_soff_.back() + (e_ub > kSmemEntries || g > kSmemMaxGroup ? e_ub : 0));
      h_mat_off_[static_cast<size_t>(ri)] = off;
      off += (OldCostOffset(g * g) + 8 * g + 255) & ~255ll;  // pair tables + old costs
    }
    max_mat = std::max(max_mat, off);
    block_mat.push_back(off);
  }
  h_block_small_.push_back(static_cast<int>(h_small_.size()));
  h_block_med_.push_back(static_cast<int>(h_med_.size()));
  h_block_big_.push_back(static_cast<int>(h_big_.size()));
  // selection: groups of at most kSelectSmallGroup members (at most 28
  // candidates) get one warp each, the others one CTA each
  h_sel_small_.clear();
  h_sel_mid_.clear();
  h_sel_big_.clear();
  h_block_sel_small_.clear();
  h_block_sel_mid_.clear();
  h_block_sel_big_.clear();
  for (size_t b = 0; b + 1 < h_block_rg_.size(); ++b) {
    h_block_sel_small_.push_back(static_cast<int>(h_sel_small_.size()));
    h_block_sel_mid_.push_back(static_cast<int>(h_sel_mid_.size()));
    h_block_sel_big_.push_back(static_cast<int>(h_sel_big_.size()));
    for (int ri = h_block_rg_[b]; ri < h_block_rg_[b + 1]; ++ri) {
      const int g = h_glen_[static_cast<size_t>(h_real_[static_cast<size_t>(ri)])];
      if (h_block_fused_[b] && is_medium(ri)) continue;  // selected by its own kernel
      (g <= kSelectSmallGroup ? h_sel_small_ : g <= kSelectMidGroup ? h_sel_mid_ : h_sel_big_).push_back(ri);
    }
  }
  h_block_sel_small_.push_back(static_cast<int>(h_sel_small_.size()));
  h_block_sel_mid_.push_back(static_cast<int>(h_sel_mid_.size()));
  h_block_sel_big_.push_back(static_cast<int>(h_sel_big_.size()));
  d_sel_small_.ensure(h_sel_small_.size() + 1);
  d_sel_mid_.ensure(h_sel_mid_.size() + 1);
  d_sel_big_.ensure(h_sel_big_.size() + 1);
  if (!h_sel_mid_.empty()) {
    CheckCuda(cudaMemcpyAsync(d_sel_mid_.p, h_sel_mid_.data(), sizeof(int) * h_sel_mid_.size(),
                              cudaMemcpyHostToDevice, stream_), "h2d select mid list");
  }
  if (!h_sel_small_.empty()) {
    CheckCuda(cudaMemcpyAsync(d_sel_small_.p, h_sel_small_.data(), sizeof(int) * h_sel_small_.size(),
                              cudaMemcpyHostToDevice, stream_), "h2d select small list");
  }
  if (!h_sel_big_.empty()) {
    CheckCuda(cudaMemcpyAsync(d_sel_big_.p, h_sel_big_.data(), sizeof(int) * h_sel_big_.size(),
                              cudaMemcpyHostToDevice, stream_), "h2d select big list");
  }
  d_med_.ensure(h_med_.size() + 1);
  if (!h_med_.empty()) {
    CheckCuda(cudaMemcpyAsync(d_med_.p, h_med_.data(), sizeof(int) * h_med_.size(), cudaMemcpyHostToDevice, stream_),
              "h2d medium list");
  }
  d_small_.ensure(h_small_.size() + 1);
  d_big_.ensure(h_big_.size() + 1);
  long long max_slots = 1;
  for (size_t b = 0; b + 1 < h_block_big_.size(); ++b) {
    max_slots = std::max(max_slots, h_soff_[static_cast<size_t>(h_block_big_[b + 1])] -
                                        h_soff_[static_cast<size_t>(h_block_big_[b])]);
  }
  d_soff_.ensure(h_soff_.size());
  CheckCuda(cudaMemcpyAsync(d_soff_.p, h_soff_.data(), sizeof(long long) * h_soff_.size(), cudaMemcpyHostToDevice,
                            stream_), "h2d soff");
  if (!h_small_.empty()) {
    CheckCuda(cudaMemcpyAsync(d_small_.p, h_small_.data(), sizeof(int) * h_small_.size(), cudaMemcpyHostToDevice,
                              stream_), "h2d small list");
  }
  d_big_moff_.ensure(h_big_moff_.size());
  if (!h_big_.empty()) {
    CheckCuda(cudaMemcpyAsync(d_big_.p, h_big_.data(), sizeof(int) * h_big_.size(), cudaMemcpyHostToDevice,
                              stream_), "h2d big list");
    CheckCuda(cudaMemcpyAsync(d_big_moff_.p, h_big_moff_.data(), sizeof(long long) * h_big_moff_.size(),
                              cudaMemcpyHostToDevice, stream_), "h2d big member offsets");
  }
  d_real_.ensure(R + 1);
  d_cand_off_.ensure(R + 1);
  d_sel_off_.ensure(R + 1);
  d_mat_off_.ensure(R + 1);
  if (R > 0) {
    CheckCuda(cudaMemcpyAsync(d_real_.p, h_real_.data(), sizeof(int) * R, cudaMemcpyHostToDevice, stream_),
              "h2d real");
    CheckCuda(cudaMemcpyAsync(d_cand_off_.p, h_cand_off_.data(), sizeof(long long) * (R + 1),
                              cudaMemcpyHostToDevice, stream_), "h2d cand_off");
    CheckCuda(cudaMemcpyAsync(d_sel_off_.p, h_sel_off_.data(), sizeof(long long) * (R + 1),
                              cudaMemcpyHostToDevice, stream_), "h2d sel_off");
    CheckCuda(cudaMemcpyAsync(d_mat_off_.p, h_mat_off_.data(), sizeof(long long) * (R + 1),
                              cudaMemcpyHostToDevice, stream_), "h2d mat_off");
  }
  SizeIterationBuffers(R, static_cast<size_t>(h_cand_off_[R]), static_cast<size_t>(h_sel_off_[R]), h_big_.size(),
                       max_mat, max_slots, false);
  plans_.clear();
  for (size_t b = 0; b + 1 < h_block_rg_.size(); ++b) {
    BlockPlan bp;
    bp.rg0 = h_block_rg_[b];
    bp.rg1 = h_block_rg_[b + 1];
    bp.slots = h_cand_off_[static_cast<size_t>(bp.rg1)] - h_cand_off_[static_cast<size_t>(bp.rg0)];
    bp.sel_slots = h_sel_off_[static_cast<size_t>(bp.rg1)] - h_sel_off_[static_cast<size_t>(bp.rg0)];
    bp.s0 = h_block_small_[b];
    bp.s1 = h_block_small_[b + 1];
    bp.m0 = h_block_med_[b];
    bp.m1 = h_block_med_[b + 1];
    bp.by_lists = h_block_fused_[b] != 0;
    bp.b0 = h_block_big_[b];
    bp.b1 = h_block_big_[b + 1];
    bp.members = h_big_moff_[static_cast<size_t>(bp.b1)] - h_big_moff_[static_cast<size_t>(bp.b0)];
    bp.slot0 = h_soff_[static_cast<size_t>(bp.b0)];
    bp.nslots = h_soff_[static_cast<size_t>(bp.b1)] - bp.slot0;
    bp.mat_bytes = block_mat[b];
    bp.ss0 = h_block_sel_small_[b];
    bp.ss1 = h_block_sel_small_[b + 1];
    bp.sm0 = h_block_sel_mid_[b];
    bp.sm1 = h_block_sel_mid_[b + 1];
    bp.sb0 = h_block_sel_big_[b];
    bp.sb1 = h_block_sel_big_[b + 1];
    plans_.push_back(bp);
  }
}

// Buffers whose sizes follow from the plan's totals (either planner).
void Engine::SizeIterationBuffers(size_t R, size_t ncand, size_t nsel, size_t nbig, long long max_mat,
                                  long long max_slots, bool windows) {
  d_sel_cnt_.ensure(R + 1);
  d_res_.ensure(ncand + 1);
  d_sel_keep_.ensure(nsel + 1);
  d_sel_rem_.ensure(nsel + 1);
  d_sel_gain_.ensure(nsel + 1);
  if (windows) return;  // neither candidate lists nor sort slots, and tables by the window (WindowTables)
  d_mat_.ensure(static_cast<size_t>(max_mat) + 256);
  d_bigdesc_.ensure(sizeof(BigDesc) * (nbig + 1));
  max_slots = std::max(max_slots, 1ll);
  for (int k = 0; k < 2; ++k) {
    d_skey_[k].ensure(static_cast<size_t>(max_slots));
    d_sval_[k].ensure(static_cast<size_t>(max_slots));
  }
  // radix-sort scratch of the deferred groups, sized once per iteration
  if (max_slots > 1) {
    size_t bytes = 0;
    CheckCuda(cub::DeviceRadixSort::SortPairs(nullptr, bytes, d_skey_[0].p, d_skey_[1].p, d_sval_[0].p,
                                              d_sval_[1].p, max_slots, 0, 64, stream_), "cub radix sort size");
    d_cub_tmp_.ensure(bytes);
  }
  d_cand_cnt_.ensure(R + 1);
  d_cand_.ensure(ncand + 1);
  d_cand_rep_.ensure(ncand + 1);
  CheckCuda(cudaMemsetAsync(d_cand_rep_.p, 0xff, sizeof(int2) * (ncand + 1), stream_), "memset cand reps");
  d_info_.ensure(sizeof(PairInfo) * (ncand + 1));
  if (cfg_.ranker) {
    d_cand_feat_.ensure(ncand + 1);
    d_rk_keep_.ensure(ncand + 1);
    d_rk_zbuf_.ensure(ncand + 1);
    for (int k = 0; k < 2; ++k) {
      d_rk_zpos_[k].ensure(static_cast<size_t>(RankerExploreCap(static_cast<long long>(ncand))));
      d_rk_zgain_[k].ensure(static_cast<size_t>(RankerExploreCap(static_cast<long long>(ncand))));
    }
  }
  rk_iter_slots_ = static_cast<long long>(ncand);
}

// The plan of an iteration of one block, or of several of at least
// kDevicePlanGroups groups, made on the device from the Divide output (the same
// lists and offsets as PrepareIterationBuffers); one small read-back brings the
// totals, the sums at the blocks' borders and the entry-pool top to the host.
// (Planned on the host, an iteration of 1.7 million groups read 13.5 MB back and
// spent 5 ms in loops with the GPU idle.)
void Engine::PlanOnDevice() {
  const long long G = n_groups_;
  const size_t cap = static_cast<size_t>(G) + 1;
  for (DevBuf<int>* b : {&d_real_, &d_small_, &d_med_, &d_big_, &d_sel_small_, &d_sel_mid_, &d_sel_big_}) b->ensure(cap);
  for (DevBuf<long long>* b : {&d_cand_off_, &d_sel_off_, &d_mat_off_, &d_big_moff_, &d_soff_}) b->ensure(cap);
  const int tiles = static_cast<int>((G + kPlanTile - 1) / kPlanTile);
  d_plan_tiles_.ensure(sizeof(PlanSums) * (2 * static_cast<size_t>(tiles) + 1));
  d_plan_scalars_.ensure(kPlanScalars);
  CheckCuda(cudaMemsetAsync(d_plan_scalars_.p, 0, sizeof(long long) * kPlanScalars, stream_), "memset plan");
  PlanParams P;
  P.glen = d_glen_.p;
  P.gent = d_gent_.p;
  P.G = G;
  P.top_k = cfg_.top_k > 0 ? cfg_.top_k : 1;
  P.mode = windowed_ ? kPlanWindows : PlanFused() ? kPlanFused : kPlanLists;
  P.tile_sums = reinterpret_cast<PlanSums*>(d_plan_tiles_.p);
  P.tile_off = P.tile_sums + tiles;
  P.tiles = tiles;
  P.scalars = d_plan_scalars_.p;
  P.real = d_real_.p;
  P.cand_off = d_cand_off_.p;
  P.sel_off = d_sel_off_.p;
  P.mat_off = d_mat_off_.p;
  P.small = d_small_.p;
  P.med = d_med_.p;
  P.big = d_big_.p;
  P.big_moff = d_big_moff_.p;
  P.soff = d_soff_.p;
  P.sel_small = d_sel_small_.p;
  P.sel_mid = d_sel_mid_.p;
  P.sel_big = d_sel_big_.p;
  const long long batch = cfg_.group_batch_size;
  const long long blocks = windowed_ ? 1 : (G + batch - 1) / batch;
  P.block_sums = nullptr;
  P.batch = batch;
  P.one_class = blocks > 1 ? 1 : 0;
  if (blocks > 1) {
    d_plan_blocks_.ensure(sizeof(PlanSums) * static_cast<size_t>(blocks));
    P.block_sums = reinterpret_cast<PlanSums*>(d_plan_blocks_.p);
  }
  P.ri_of = nullptr;
  if (windowed_) {
    d_ri_of_.ensure(cap);
    P.ri_of = d_ri_of_.p;
  }
  if (tiles > 0) {
    ++launches_;
    LaunchFollowing(PlanTileKernel, tiles, kPlanThreads, 0, stream_, P);
  }
  ++launches_;
  LaunchFollowing(PlanScanKernel, 1, kPlanThreads, 0, stream_, P);
  if (tiles > 0) {
    ++launches_;
    LaunchFollowing(PlanScatterKernel, tiles, kPlanThreads, 0, stream_, P);
  }
  static_assert(kPlanScalars + 1 <= 32, "room in the pinned words");
  long long* hs = h_pin_.p + 16;  // read back: totals and pool top
  CheckCuda(cudaMemcpyAsync(hs, d_plan_scalars_.p, sizeof(long long) * kPlanScalars, cudaMemcpyDeviceToHost,
                            stream_), "d2h plan");
  CheckCuda(cudaMemcpyAsync(hs + kPlanScalars, d_pool_top_.p, sizeof(long long), cudaMemcpyDeviceToHost, stream_),
            "d2h pool top");
  std::vector<PlanSums> sums(static_cast<size_t>(blocks) + 1);
  if (blocks > 1) {
    CheckCuda(cudaMemcpyAsync(sums.data(), d_plan_blocks_.p, sizeof(PlanSums) * static_cast<size_t>(blocks),
                              cudaMemcpyDeviceToHost, stream_), "d2h block plan");
  }
  QueueError();
  CheckCuda(cudaStreamSynchronize(stream_), "plan sync");
  ThrowError();
  long long v[kPlanScalars + 1];
  std::memcpy(v, hs, sizeof(v));
  EnsurePoolRoom(static_cast<unsigned long long>(v[kPlanScalars]));
  const size_t R = static_cast<size_t>(v[kPlanR]);
  if (blocks <= 1) sums[0] = PlanSums{};
  PlanSums& end = sums[static_cast<size_t>(std::max(blocks, 1ll))];
  end = PlanSums{};
  end.real = static_cast<int>(R);
  end.cand = v[kPlanCand];
  end.sel = v[kPlanSel];
  end.small[0] = static_cast<int>(v[kPlanSmall]);
  end.med = static_cast<int>(v[kPlanMed]);
  end.big = static_cast<int>(v[kPlanBig]);
  end.moff = v[kPlanMembers];
  end.soff = v[kPlanSlots];
  end.mat = v[kPlanMat];
  end.ssmall = static_cast<int>(v[kPlanSelSmall]);
  end.smid = static_cast<int>(v[kPlanSelMid]);
  end.sbig = static_cast<int>(v[kPlanSelBig]);
  plans_.clear();
  long long max_mat = 0, max_slots = 0;
  for (size_t i = 0; i + 1 < sums.size(); ++i) {
    const PlanSums& p = sums[i];
    const PlanSums& q = sums[i + 1];
    BlockPlan bp;
    bp.rg0 = p.real;
    bp.rg1 = q.real;
    bp.slots = q.cand - p.cand;
    bp.sel_slots = q.sel - p.sel;
    bp.s0 = p.small[0];
    bp.s1 = q.small[0];
    bp.m0 = p.med;
    bp.m1 = q.med;
    bp.b0 = p.big;
    bp.b1 = q.big;
    bp.by_lists = blocks > 1 || PlanFused();
    bp.members = q.moff - p.moff;
    bp.slot0 = p.soff;
    bp.nslots = q.soff - p.soff;
    bp.mat0 = p.mat;
    bp.mat_bytes = q.mat - p.mat;
    bp.ss0 = p.ssmall;
    bp.ss1 = q.ssmall;
    bp.sm0 = p.smid;
    bp.sm1 = q.smid;
    bp.sb0 = p.sbig;
    bp.sb1 = q.sbig;
    max_mat = std::max(max_mat, bp.mat_bytes);
    max_slots = std::max(max_slots, bp.nslots);
    plans_.push_back(bp);
  }
  SizeIterationBuffers(R, static_cast<size_t>(v[kPlanCand]), static_cast<size_t>(v[kPlanSel]),
                       static_cast<size_t>(v[kPlanBig]), max_mat, max_slots, windowed_);
}

QuotientView Engine::View() {
  QuotientView Q;
  Q.ent = d_pool_[cur_pool_].p;
  Q.off = d_qoff_.p;
  Q.len = d_qlen_.p;
  Q.cap = d_qcap_.p;
  Q.size = d_qsize_.p;
  Q.internal = d_qint_.p;
  return Q;
}

namespace {
// The parts of the commit that a window sets.
void CommitDefaults(CommitParams* C) {
  C->windowed = 0;
  C->W = WindowParams{};
}
}  // namespace

void Engine::LaunchCommit(int rg0, int nrg, int64_t max_pairs, bool verify, const void* window) {
  CommitParams C;
  CommitDefaults(&C);
  if (window) {
    C.windowed = 1;
    C.W = *static_cast<const WindowParams*>(window);
  }
  C.Q = View();
  C.rg0 = rg0;
  C.nrg = nrg;
  C.sel_off = d_sel_off_.p;
  C.sel_keep = d_sel_keep_.p;
  C.sel_rem = d_sel_rem_.p;
  C.sel_gain = d_sel_gain_.p;
  C.sel_cnt = d_sel_cnt_.p;
  C.head = d_head_.p;
  C.next = d_next_.p;
  C.tail = d_tail_.p;
  C.fwd = d_fwd_.p;
  C.stamp = d_stamp_.p;
  C.partner = d_partner_.p;
  C.seq = d_seq_.p;
  C.claim = d_claim_.p;
  C.block_stamp = block_stamp_;
  C.pool_top = d_pool_top_.p;
  C.pool_cap = pool_cap_;
  C.scratch = d_scratch_.p;
  C.scratch_cap = d_scratch_.n;
  C.ctl = d_ctl_.p;
  C.stats = d_stats_.p;
  C.err = d_err_.p;
  C.rows_short = d_rows_short_.p;
  C.rows_long = d_rows_long_.p;
  // a row of more than `limit` entries holds that many of the arcs
  const size_t limit = window ? kWindowRow : kRowSmem;
  d_rows_huge_.ensure(sizeof(HugeRow) * (static_cast<size_t>(arcs_) / limit + 1));
  d_huge_units_.ensure(static_cast<size_t>(arcs_) / kHugeUnit + static_cast<size_t>(arcs_) / limit + 1);
  C.rows_huge = reinterpret_cast<HugeRow*>(d_rows_huge_.p);
  C.huge_units = d_huge_units_.p;
  C.ticket = d_rw_ticket_.p;
  C.sel_list = d_sel_list_.p;
  // warp-per-pair commit for short pairs, except in small blocks, where one
  // launch is cheaper than a second one
  C.warp_pairs = nrg > kFewGroups && !window ? 1 : 0;
  if (verify) {
    const int vb = static_cast<int>(std::min<int64_t>((max_pairs + 7) / 8 + 1, 152 * 8));
    ++launches_;
    VerifyKernel<<<vb, 256, 0, stream_>>>(C);
  }
  const int grid = static_cast<int>(std::min<int64_t>(std::max<int64_t>(max_pairs, 1), kRowsGrid));
  BeginTimed(kTimeUpdate);
  ++launches_;
  // the warp kernel goes first: a pair it commits still reads as short to
  // CommitKernel (its keep row can only be short), which skips it; a long
  // pair is untouched until CommitKernel
  if (C.warp_pairs) {
    LaunchFollowing(CommitShortKernel, static_cast<int>(std::min<int64_t>((max_pairs + 7) / 8 + 1, 152 * 8)), 256, 0,
                    stream_, C);
    ++launches_;
  }
  launches_ += 3;
  const bool ahead = window || SmallBlocks();
  LaunchAhead(ahead, CommitKernel, grid, kRowsThreads, sizeof(RowsSmem), stream_, C);
  LaunchAhead(ahead, RewriteRowsKernel, kRowsGrid, kRowsThreads, sizeof(RowsSmem), stream_, C);
  LaunchAhead(ahead, RewriteHugeKernel, kHugeGrid, kHugeThreads, sizeof(HugeSmem), stream_, C);
  EndTimed(kTimeUpdate);
}

// EA-proxy candidates for the small-group list entries [s0, s1) (one warp
// per group) and the big-group entries [b0, b1) (one CTA per group).
// Row sums and pair sums are written by the block's own prepare kernels from
// its block-start state and read by its scoring pass only, so every block uses
// them, on graphs whose shared targets fit their field of the pair words.
bool Engine::RowSumsOn() const { return arcs_ < row_sum_arcs_; }

void Engine::LaunchPrepare(const BlockPlan& bp) {
  const int s0 = bp.s0, s1 = bp.s1, b0 = bp.b0, b1 = bp.b1;
  PrepareParams PP;
  PP.Q = View();
  PP.order = d_order_.p;
  PP.gstart = d_gstart_.p;
  PP.glen = d_glen_.p;
  PP.group_of = d_group_of_.p;
  PP.idx_in_group = d_idx_in_group_.p;
  PP.real = d_real_.p;
  PP.cand_off = d_cand_off_.p;
  PP.cand = d_cand_.p;
  PP.cand_cnt = d_cand_cnt_.p;
  PP.mat_off = d_mat_off_.p;
  // the block's pair tables start at the buffer's start
  PP.mat = reinterpret_cast<unsigned char*>(reinterpret_cast<uintptr_t>(d_mat_.p) - static_cast<uintptr_t>(bp.mat0));
  PP.mat_zeroed = 0;
  PP.rc = nullptr;
  PP.info = nullptr;
  if (RowSumsOn()) {
    d_rc_.ensure(sizeof(RowSums) * static_cast<size_t>(n_));
    PP.rc = reinterpret_cast<RowSums*>(d_rc_.p);
    PP.info = reinterpret_cast<PairInfo*>(d_info_.p);
  }
  PP.scratch = d_scratch_.p;
  PP.scratch_cap = d_scratch_.n;
  PP.ctl = d_ctl_.p;
  PP.top_k = cfg_.top_k;
  PP.stats = d_stats_.p;
  PP.err = d_err_.p;
  PP.cand_feat = cfg_.ranker ? d_cand_feat_.p : nullptr;
  PP.cand_rep = d_cand_rep_.p;
  BeginTimed(kTimePrepare);
  if (s1 > s0) {
    PP.list = d_small_.p;
    PP.list0 = s0;
    PP.nlist = s1 - s0;
    ++launches_;
    LaunchFollowing(PrepareSmallKernel, (s1 - s0 + kSmallWarps - 1) / kSmallWarps, kSmallWarps * 32,
                    sizeof(SmallSmem), stream_, PP);
  }
  if (b1 > b0) {
    PP.list = d_big_.p;
    PP.list0 = b0;
    PP.nlist = b1 - b0;
    PP.moff = d_big_moff_.p;
    const long long members = bp.members;
    PP.desc = reinterpret_cast<BigDesc*>(d_bigdesc_.p);
    PP.soff = d_soff_.p;
    PP.slot0 = bp.slot0;
    PP.nslots = bp.nslots;
    if (bp.rg1 - bp.rg0 > kFewGroups && bp.mat_bytes > 0) {
      // one memset clears every pair table of a large block (a CTA clearing
      // its own group's tables is the tail of the kernel for large groups)
      CheckCuda(cudaMemsetAsync(d_mat_.p, 0, static_cast<size_t>(bp.mat_bytes), stream_), "memset pair tables");
      PP.mat_zeroed = 1;
    }
    PP.bits = SlotLayout(n_, b1 - b0);
    PP.skey = d_skey_[0].p;
    PP.sval = d_sval_[0].p;
    PP.skey_sorted = d_skey_[1].p;
    PP.sval_sorted = d_sval_[1].p;
    ++launches_;
    LaunchFollowing(PrepareKernel, b1 - b0, kPrepThreads, sizeof(PrepSmem), stream_, PP);
    if (PP.nslots > 0) {
      const long long windows = (PP.nslots + kFillWindow - 1) / kFillWindow;
      ++launches_;
      LaunchAhead(SmallBlocks(), PrepareFillKernel, static_cast<int>(std::min(windows, 152ll * 32)), kFillThreads, 0,
                  stream_, PP);
      const int bits = PP.bits.sorted();
      size_t bytes = 0;
      CheckCuda(cub::DeviceRadixSort::SortPairs(nullptr, bytes, d_skey_[0].p, d_skey_[1].p, d_sval_[0].p,
                                                d_sval_[1].p, PP.nslots, 0, bits, stream_), "cub radix sort size");
      d_cub_tmp_.ensure(bytes);
      CheckCuda(cub::DeviceRadixSort::SortPairs(d_cub_tmp_.p, bytes, d_skey_[0].p, d_skey_[1].p, d_sval_[0].p,
                                                d_sval_[1].p, PP.nslots, 0, bits, stream_), "cub radix sort");
      const long long want = ((PP.nslots + 31) / 32 * kAccumSplit + kAccumThreads / 32 - 1) / (kAccumThreads / 32);
      ++launches_;
      LaunchFollowing(PrepareAccumKernel, static_cast<int>(std::min<long long>(want, accum_grid_)), kAccumThreads, 0,
                      stream_, PP);
    }
    ++launches_;
    LaunchFollowing(PrepareMembersKernel, static_cast<int>((members + 7) / 8), 256, 0, stream_, PP);
    ++launches_;
    LaunchFollowing(PrepareOutputKernel, b1 - b0, kPrepThreads, 0, stream_, PP);
  }
  EndTimed(kTimePrepare);
}

void Engine::LaunchMedium(const BlockPlan& bp, double threshold) {
  if (bp.m1 <= bp.m0) return;
  MediumParams M{};
  M.Q = View();
  M.order = d_order_.p;
  M.gstart = d_gstart_.p;
  M.glen = d_glen_.p;
  M.group_of = d_group_of_.p;
  M.idx_in_group = d_idx_in_group_.p;
  M.real = d_real_.p;
  M.list = d_med_.p;
  M.list0 = bp.m0;
  M.top_k = cfg_.top_k;
  M.threshold = threshold;
  M.thr = SplitThreshold(threshold);
  M.use_threshold = cfg_.ea_use_threshold ? 1 : 0;
  M.strict = bp.rg1 - bp.rg0 <= kFewGroups ? 1 : 0;
  M.sel_off = d_sel_off_.p;
  M.sel_keep = d_sel_keep_.p;
  M.sel_rem = d_sel_rem_.p;
  M.sel_gain = d_sel_gain_.p;
  M.sel_cnt = d_sel_cnt_.p;
  M.stamp = d_stamp_.p;
  M.partner = d_partner_.p;
  M.seq = d_seq_.p;
  M.sel_list = d_sel_list_.p;
  M.ctl = d_ctl_.p;
  M.block_stamp = block_stamp_;
  M.stats = d_stats_.p;
  M.err = d_err_.p;
  routes_[kRouteMediumGroups] += bp.m1 - bp.m0;
  BeginTimed(kTimePrepare);
  ++launches_;
  LaunchFollowing(MediumKernel, bp.m1 - bp.m0, kMedThreads, sizeof(MediumSmem), stream_, M);
  EndTimed(kTimePrepare);
}

void Engine::RunBlock(const BlockPlan& bp, double threshold, int iter, int total_iterations) {
  ++block_stamp_;
  ++hstats_.blocks;
  const int rg0 = bp.rg0;
  const int nrg = bp.rg1 - bp.rg0;
  const long long slots = bp.slots;
  const long long sel_slots = bp.sel_slots;
  // the block control words are zero: cleared by Merge before the first
  // block and by the previous block's last kernel
  LaunchMedium(bp, threshold);
  LaunchPrepare(bp);
  ScoreParams SP;
  SP.Q = View();
  SP.order = d_order_.p;
  SP.gstart = d_gstart_.p;
  SP.real = d_real_.p;
  SP.rg0 = rg0;
  SP.nrg = nrg;
  SP.cand_off = d_cand_off_.p;
  SP.cand = d_cand_.p;
  SP.cand_cnt = d_cand_cnt_.p;
  SP.cand_rep = d_cand_rep_.p;
  SP.ctl = d_ctl_.p;
  SP.res = d_res_.p;
  SP.stats = d_stats_.p;
  SP.err = d_err_.p;
  SP.threshold = threshold;
  SP.thr = SplitThreshold(threshold);
  SP.use_threshold = cfg_.ea_use_threshold ? 1 : 0;
  SP.audit = cfg_.ranker_audit ? 1 : 0;
  SP.phase = 0;
  SP.keep = d_rk_keep_.p;
  SP.zbuf = d_rk_zbuf_.p;
  SP.zpos = d_rk_zpos_[0].p;
  SP.zgain = d_rk_zgain_[0].p;
  SP.npos = d_rk_npos_.p;
  SP.zcap = 0;
  SP.cutoff = d_rk_cut_.p;
  SP.rc = nullptr;
  SP.info = nullptr;
  if (RowSumsOn()) {
    // written by this block's prepare kernels
    SP.rc = reinterpret_cast<const RowSums*>(d_rc_.p);
    SP.info = reinterpret_cast<const PairInfo*>(d_info_.p);
  }
  SP.strict = nrg <= kFewGroups ? 1 : 0;
  const int fetch = SP.rc ? kScoreFetch : kScoreFetchMerge;
  const int sgrid = static_cast<int>(
      std::min<long long>((slots + fetch * 8 - 1) / (fetch * 8), score_grid_));
  // learned ranker: trained after the logging iterations; afterwards the
  // exploration subset is scored first, then the rest above the cutoff
  const bool ranking = cfg_.ranker && rk_trained_ && iter > cfg_.ranker_train_iters;
  if (ranking) {
    RankerRank(rg0, nrg, slots, threshold, iter);
    SP.phase = 1;
    SP.zcap = static_cast<unsigned>(RankerExploreCap(slots));
    BeginTimed(kTimeScore);
    ++launches_;
    LaunchFollowing(ScoreKernel, sgrid, kScoreThreads, 0, stream_, SP);
    EndTimed(kTimeScore);
    RankerCutoff(slots);
    SP.phase = 2;
  }
  BeginTimed(kTimeScore);
  ++launches_;
  LaunchFollowing(ScoreKernel, sgrid, kScoreThreads, 0, stream_, SP);
  EndTimed(kTimeScore);
  if (cfg_.ranker && !rk_trained_ && iter <= cfg_.ranker_train_iters) {
    RankerLog(rg0, nrg, slots, iter, threshold, total_iterations);
  }
  SelectParams LP;
  LP.order = d_order_.p;
  LP.gstart = d_gstart_.p;
  LP.glen = d_glen_.p;
  LP.real = d_real_.p;
  LP.rg0 = rg0;
  LP.cand_off = d_cand_off_.p;
  LP.cand = d_cand_.p;
  LP.cand_cnt = d_cand_cnt_.p;
  LP.res = d_res_.p;
  LP.sel_off = d_sel_off_.p;
  LP.sel_keep = d_sel_keep_.p;
  LP.sel_rem = d_sel_rem_.p;
  LP.sel_gain = d_sel_gain_.p;
  LP.sel_cnt = d_sel_cnt_.p;
  LP.qlen = d_qlen_.p;
  LP.stamp = d_stamp_.p;
  LP.partner = d_partner_.p;
  LP.seq = d_seq_.p;
  LP.block_stamp = block_stamp_;
  LP.threshold = threshold;
  LP.thr = SplitThreshold(threshold);
  LP.use_threshold = cfg_.ea_use_threshold ? 1 : 0;
  LP.scratch = d_scratch_.p;
  LP.scratch_cap = d_scratch_.n;
  LP.ctl = d_ctl_.p;
  LP.stats = d_stats_.p;
  LP.err = d_err_.p;
  LP.sel_list = d_sel_list_.p;
  const int ss0 = bp.ss0, ss1 = bp.ss1;
  const int sb0 = bp.sb0, sb1 = bp.sb1;
  if (nrg <= kFewGroups && !bp.by_lists) {
    // a small block: one launch, a CTA per group (same selection)
    LP.list = nullptr;
    LP.list0 = rg0;
    LP.nlist = nrg;
    ++launches_;
    LaunchFollowing(SelectMatchKernel, nrg, kMatchThreads, 8 * kMatchSmemKeys, stream_, LP);
    LaunchCommit(rg0, nrg, sel_slots, cfg_.verify_cuda_gain, nullptr);
    return;
  }
  if (ss1 > ss0) {
    LP.list = d_sel_small_.p;
    LP.list0 = ss0;
    LP.nlist = ss1 - ss0;
    ++launches_;
    LaunchFollowing(SelectSmallKernel, (ss1 - ss0 + kSelectSmallWarps - 1) / kSelectSmallWarps,
                    kSelectSmallWarps * 32, 0, stream_, LP);
  }
  const int sm0 = bp.sm0, sm1 = bp.sm1;
  if (sm1 > sm0) {
    LP.list = d_sel_mid_.p;
    LP.list0 = sm0;
    LP.nlist = sm1 - sm0;
    ++launches_;
    SelectKernel<kSelectMidThreads, kSelectMidKeys><<<sm1 - sm0, kSelectMidThreads, 8 * kSelectMidKeys, stream_>>>(LP);
  }
  if (sb1 > sb0) {
    LP.list = d_sel_big_.p;
    LP.list0 = sb0;
    LP.nlist = sb1 - sb0;
    ++launches_;
    LaunchFollowing(SelectMatchKernel, sb1 - sb0, kMatchThreads, 8 * kMatchSmemKeys, stream_, LP);
  }
  LaunchCommit(rg0, nrg, sel_slots, cfg_.verify_cuda_gain, nullptr);
}

bool Engine::WindowsOn() const {
  // the ranker calibrates itself on whole blocks
  return cfg_.group_batch_size <= kWindowMaxBatch && !cfg_.ranker && RowSumsOn();
}

// Makes room for the tables of a round's big groups (group positions and block
// ends are set up); returns the groups that a window may take in: all it likes
// where the whole iteration's tables are few, else as many as stay within the
// limit, one block at the least. Where the device has no such room left, fewer.
int Engine::WindowTables(int R) {
  auto fits = [&](long long bytes) {
    try {
      d_mat_.ensure(static_cast<size_t>(bytes) + 256);
      return true;
    } catch (const std::runtime_error&) {
      return false;
    }
  };
  const long long total = plans_[0].mat_bytes;
  if (total <= window_tables_ && fits(total)) return kWindowMaxGroups;
  static_assert(kWindowLengths <= kPlanScalars, "room in the plan's words");
  unsigned long long* most = reinterpret_cast<unsigned long long*>(d_plan_scalars_.p);
  CheckCuda(cudaMemsetAsync(most, 0, sizeof(long long) * kWindowLengths, stream_), "memset window spans");
  ++launches_;
  LaunchFollowing(WindowSpanKernel, (R + 255) / 256, 256, 0, stream_, d_mat_off_.p, d_blk_beg_.p, d_blk_end_.p, R, most);
  CheckCuda(cudaMemcpyAsync(h_pin_.p + 16, most, sizeof(long long) * kWindowLengths, cudaMemcpyDeviceToHost, stream_),
            "d2h window spans");
  CheckCuda(cudaStreamSynchronize(stream_), "sync");
  for (int k = 0; k + 1 < kWindowLengths; ++k) {
    if (h_pin_.p[16 + k] <= window_tables_ && fits(h_pin_.p[16 + k])) return kWindowMaxGroups >> k;
  }
  d_mat_.ensure(static_cast<size_t>(h_pin_.p[16 + kWindowLengths - 1]) + 256);
  return 1;
}

// An iteration's blocks through windows (window.cuh).
void Engine::RunWindows(double threshold) {
  const int R = plans_[0].rg1;
  if (R == 0) return;
  const size_t ur = static_cast<size_t>(R);
  d_node_ri_.ensure(static_cast<size_t>(n_));
  d_blk_end_.ensure(ur + 1);
  d_blk_beg_.ensure(ur + 1);
  d_dirty_.ensure(ur + 1);
  d_gs_.ensure(sizeof(GroupStats) * (ur + 1));
  d_win_list_.ensure(2 * static_cast<size_t>(kWindowList));
  d_win_big_.ensure(sizeof(BigGroup) * kWindowList);
  d_win_off_.ensure(2 * static_cast<size_t>(kWindowList) + 2);
  d_conflict_.ensure(ur + 1);
  d_units_.ensure(sizeof(LongUnit) * kLongUnits);
  d_rc_.ensure(sizeof(RowSums) * static_cast<size_t>(n_));
  WindowParams W{};
  W.Q = View();
  W.order = d_order_.p;
  W.gstart = d_gstart_.p;
  W.glen = d_glen_.p;
  W.gent = d_gent_.p;
  W.group_of = d_group_of_.p;
  W.real = d_real_.p;
  W.node_ri = d_node_ri_.p;
  W.blk_end = d_blk_end_.p;
  W.blk_beg = d_blk_beg_.p;
  W.idx_in_group = d_idx_in_group_.p;
  W.ctl = reinterpret_cast<WindowCtl*>(d_wctl_.p);
  W.gs = reinterpret_cast<GroupStats*>(d_gs_.p);
  W.conflict = d_conflict_.p;
  W.units = reinterpret_cast<LongUnit*>(d_units_.p);
  W.dirty = d_dirty_.p;
  W.list_dirty = d_win_list_.p;
  W.list_small = d_win_list_.p + kWindowList;
  W.list_big = reinterpret_cast<BigGroup*>(d_win_big_.p);
  W.moff = d_win_off_.p;
  W.poff = d_win_off_.p + kWindowList + 1;
  W.cand_off = d_cand_off_.p;
  W.keys = reinterpret_cast<unsigned long long*>(d_res_.p);
  W.rc = reinterpret_cast<RowSums*>(d_rc_.p);
  W.sel_off = d_sel_off_.p;
  W.sel_keep = d_sel_keep_.p;
  W.sel_rem = d_sel_rem_.p;
  W.sel_gain = d_sel_gain_.p;
  W.sel_cnt = d_sel_cnt_.p;
  W.stamp = d_stamp_.p;
  W.partner = d_partner_.p;
  W.seq = d_seq_.p;
  W.sel_list = d_sel_list_.p;
  W.bctl = d_ctl_.p;
  W.top_k = cfg_.top_k;
  W.threshold = threshold;
  W.thr = SplitThreshold(threshold);
  W.use_threshold = cfg_.ea_use_threshold ? 1 : 0;
  W.all_strict = cfg_.group_batch_size <= kFewGroups ? 1 : 0;
  W.stats = d_stats_.p;
  W.err = d_err_.p;
  // the frontier and the rounds done, written by the device after each round
  int* seen = reinterpret_cast<int*>(h_pin_.p + 48);
  __atomic_store_n(&seen[0], 0, __ATOMIC_RELEASE);
  __atomic_store_n(&seen[1], 0, __ATOMIC_RELEASE);
  W.host_f = seen;
  CheckCuda(cudaMemsetAsync(&W.ctl->blocks, 0, sizeof(long long), stream_), "memset blocks");
  const int count = static_cast<int>(n_active_);
  ++launches_;
  LaunchFollowing(WindowSetupKernel, (std::max(count, R) + 255) / 256, 256, 0, stream_, W.order, W.group_of,
                  d_ri_of_.p, count, W.real, R, cfg_.group_batch_size, d_node_ri_.p, d_blk_beg_.p, d_blk_end_.p,
                  W.dirty, W.ctl);
  W.max_groups = WindowTables(R);
  W.mat_off = d_mat_off_.p;
  W.mat = d_mat_.p;
  ++launches_;
  LaunchFollowing(WindowBeginKernel, 1, kHugeThreads, 0, stream_, W, R);
  // the host keeps a few rounds queued behind the one running; a round past
  // the end finds nothing to do. It waits as the process has asked the driver to
  // wait: asleep on the round's event, giving its core away, or (the driver's
  // default too) watching the mapped words, which reach it some microseconds
  // before an event would.
  unsigned flags = 0;
  CheckCuda(cudaGetDeviceFlags(&flags), "device flags");
  const bool asleep = (flags & cudaDeviceScheduleMask) == cudaDeviceScheduleBlockingSync;
  const bool yielding = (flags & cudaDeviceScheduleMask) == cudaDeviceScheduleYield;
  while (asleep && round_ev_.size() < kWindowAhead) {
    cudaEvent_t e;
    CheckCuda(cudaEventCreateWithFlags(&e, cudaEventBlockingSync | cudaEventDisableTiming), "cudaEventCreate");
    round_ev_.push_back(e);
  }
  long long queued = 0;
  for (long long idle = 0;;) {
    const int done = __atomic_load_n(&seen[1], __ATOMIC_ACQUIRE) - 1;  // the first lists count as one
    if (__atomic_load_n(&seen[0], __ATOMIC_ACQUIRE) >= R) break;
    if (queued - done >= kWindowAhead) {
      if (asleep) {  // until the oldest round not seen done is
        CheckCuda(cudaEventSynchronize(round_ev_[static_cast<size_t>((done + 1) % kWindowAhead)]), "window rounds");
        continue;
      }
      if (yielding) std::this_thread::yield();
      if (++idle % 4096 == 0) {
        const cudaError_t st = cudaStreamQuery(stream_);
        if (st != cudaErrorNotReady) CheckCuda(st, "window rounds");
      }
      continue;
    }
    // every round commits at least one block
    if (queued > R + kWindowAhead) throw std::runtime_error("merge windows made no progress");
    ++queued;
    ++routes_[kRouteWindowRounds];
    ++block_stamp_;
    W.block_stamp = block_stamp_;
    BeginTimed(kTimePrepare);
    LaunchFollowing(WindowEvalKernel, kEvalGrid, kEvalWarps * 32, sizeof(EvalSmem), stream_, W);
    LaunchFollowing(WindowLongKernel, kLongGrid, kLongThreads, 0, stream_, W);
    LaunchFollowing(WindowPairsKernel, kPairGrid, kPairWarps * 32, sizeof(PairTable) * kPairWarps, stream_, W);
    EndTimed(kTimePrepare);
    BeginTimed(kTimeScore);
    LaunchFollowing(WindowScoreKernel, kBigGrid, 256, 0, stream_, W);
    LaunchFollowing(WindowSelectKernel, kBigGrid, kMatchThreads, 8 * kMatchSmemKeys, stream_, W);
    EndTimed(kTimeScore);
    LaunchFollowing(WindowMarkKernel, kMarkGrid, kMarkThreads, 0, stream_, W);
    launches_ += 6;
    LaunchCommit(0, R, kBigGrid, cfg_.verify_cuda_gain, &W);
    if (asleep) {
      CheckCuda(cudaEventRecord(round_ev_[static_cast<size_t>(queued % kWindowAhead)], stream_), "event record");
    }
  }
  CheckCuda(cudaMemcpyAsync(h_pin_.p + 9, &W.ctl->blocks, sizeof(long long), cudaMemcpyDeviceToHost, stream_),
            "d2h blocks");
  CheckCuda(cudaStreamSynchronize(stream_), "windows sync");
  hstats_.blocks += static_cast<uint64_t>(h_pin_.p[9]);
}

void Engine::Merge(int iter, int total_iterations) {
  AllocScope alloc(stream_);
  if (n_groups_ < 0) throw std::runtime_error("Merge requires a preceding Divide");
  // ComputeMergeThreshold, reciprocal policy (src/sweg.cpp:400-406)
  const double threshold = 1.0 / static_cast<double>(iter + 1);
  if (plan_on_device_ || windowed_) {
    if (!windowed_) ++routes_[kRouteDevicePlans];
    PlanOnDevice();
  } else {
    ++routes_[kRouteHostPlans];
    EnsurePoolRoom();
    PrepareIterationBuffers();
  }
  CheckCuda(cudaMemsetAsync(d_ctl_.p, 0, sizeof(BlockCtl), stream_), "memset ctl");
  if (windowed_) {
    RunWindows(threshold);
  } else {
    for (const BlockPlan& bp : plans_) {
      if (bp.rg1 > bp.rg0) RunBlock(bp, threshold, iter, total_iterations);
    }
  }
  ++launches_;
  LaunchFollowing(RelabelKernel, (n_ + 255) / 256, 256, 0, stream_, d_label_.p, d_fwd_.p, n_);
  n_groups_ = -1;  // the groups are consumed
  // accepted merges so far, read back with this synchronisation: the next
  // Divide knows the active count without a round trip of its own
  CheckCuda(cudaMemcpyAsync(h_pin_.p + 8, d_stats_.p + kStAccepted, sizeof(unsigned long long),
                            cudaMemcpyDeviceToHost, stream_), "d2h accepted");
  QueueError();
  CheckCuda(cudaStreamSynchronize(stream_), "merge sync");
  ThrowError();
  {
    unsigned long long accepted = 0;
    std::memcpy(&accepted, h_pin_.p + 8, sizeof(accepted));
    known_active_ = static_cast<int64_t>(n_) - static_cast<int64_t>(accepted);
  }
  if (cfg_.ranker && !rk_trained_ && iter == cfg_.ranker_train_iters) RankerTrain();
  if (cfg_.ranker && rk_trained_ && iter > cfg_.ranker_train_iters) RankerFinishIteration();
}

void Engine::ScorePairs(const int32_t* rep_a, const int32_t* rep_b, int64_t count, int64_t* gain,
                        int64_t* before) {
  AllocScope alloc(stream_);
  if (count <= 0) return;
  uint32_t largest = 0;  // a negative id is a large one
  for (int64_t i = 0; i < count; ++i) {
    largest = std::max(largest, std::max(static_cast<uint32_t>(rep_a[i]), static_cast<uint32_t>(rep_b[i])));
  }
  if (largest >= static_cast<uint32_t>(n_)) throw std::out_of_range("quotient supernode is out of range");
  const size_t uc = static_cast<size_t>(count);
  const unsigned long long max_units = 1ull << 20;  // longer pairs beyond these are one warp's work
  DevBuf<int> da, db;
  DevBuf<long long> dg;
  DevBuf<unsigned char> du;
  da.ensure(uc);
  db.ensure(uc);
  dg.ensure(2 * uc + 1);
  du.ensure(sizeof(PairUnit) * max_units);
  CheckCuda(cudaMemcpyAsync(da.p, rep_a, sizeof(int) * uc, cudaMemcpyHostToDevice, stream_), "h2d pairs");
  CheckCuda(cudaMemcpyAsync(db.p, rep_b, sizeof(int) * uc, cudaMemcpyHostToDevice, stream_), "h2d pairs");
  unsigned long long* nunits = reinterpret_cast<unsigned long long*>(dg.p + 2 * uc);
  CheckCuda(cudaMemsetAsync(nunits, 0, sizeof(unsigned long long), stream_), "memset units");
  const int blocks = static_cast<int>(std::min<int64_t>((count + 7) / 8, 152 * 16));
  PairUnit* units = reinterpret_cast<PairUnit*>(du.p);
  launches_ += 2;
  ScorePairsKernel<<<blocks, kScoreThreads, 0, stream_>>>(View(), da.p, db.p, count, dg.p, dg.p + uc, units, nunits,
                                                          max_units, d_err_.p);
  ScoreLongPairsKernel<<<152 * 6, kScoreThreads, 0, stream_>>>(View(), da.p, db.p, dg.p, dg.p + uc, units, nunits,
                                                               max_units, d_err_.p);
  CheckError();  // a call that fails leaves the caller's arrays alone
  CheckCuda(cudaMemcpyAsync(gain, dg.p, sizeof(int64_t) * uc, cudaMemcpyDeviceToHost, stream_), "d2h gains");
  CheckCuda(cudaMemcpyAsync(before, dg.p + uc, sizeof(int64_t) * uc, cudaMemcpyDeviceToHost, stream_), "d2h costs");
  CheckCuda(cudaStreamSynchronize(stream_), "score sync");
}

int64_t Engine::PrepareGroup(const int32_t* q, int g, int32_t* a_idx, int32_t* b_idx, int64_t cap) {
  AllocScope alloc(stream_);
  if (g < 0 || g > kMaxGroup) throw std::invalid_argument("group size out of range");
  std::vector<int> hq(q, q + g);
  for (int i = 0; i < g; ++i) {
    if (hq[static_cast<size_t>(i)] < 0 || hq[static_cast<size_t>(i)] >= n_) {
      throw std::out_of_range("quotient supernode is out of range");
    }
  }
  if (g < 2) return 0;
  // One explicit group; the Divide output is overwritten.
  n_groups_ = 1;
  h_glen_.assign(1, g);
  // the group's row entries (routing and deferred-group sort slots)
  {
    std::vector<int> lens(static_cast<size_t>(n_));
    CheckCuda(cudaMemcpyAsync(lens.data(), d_qlen_.p, sizeof(int) * static_cast<size_t>(n_), cudaMemcpyDeviceToHost,
                              stream_), "d2h row lengths");
    CheckCuda(cudaStreamSynchronize(stream_), "sync");
    int64_t e = 0;
    for (int i = 0; i < g; ++i) e += lens[static_cast<size_t>(hq[static_cast<size_t>(i)])];
    if (e > INT32_MAX) throw std::invalid_argument("group row entries exceed the supported maximum");
    h_gent_.assign(1, static_cast<unsigned>(e));
  }
  const int zero = 0;
  CheckCuda(cudaMemcpyAsync(d_order_.p, hq.data(), sizeof(int) * static_cast<size_t>(g), cudaMemcpyHostToDevice,
                            stream_), "h2d group");
  CheckCuda(cudaMemcpyAsync(d_gstart_.p, &zero, sizeof(int), cudaMemcpyHostToDevice, stream_), "h2d gstart");
  CheckCuda(cudaMemcpyAsync(d_glen_.p, &g, sizeof(int), cudaMemcpyHostToDevice, stream_), "h2d glen");
  std::vector<int> idx(static_cast<size_t>(g));
  for (int i = 0; i < g; ++i) idx[static_cast<size_t>(i)] = i;
  // group_of / idx_in_group for the members; every other rep must not match
  // group 0, so the array is first filled with -1.
  CheckCuda(cudaMemsetAsync(d_group_of_.p, 0xff, sizeof(int) * static_cast<size_t>(n_), stream_), "memset");
  DevBuf<int> dq, di;
  dq.ensure(static_cast<size_t>(g));
  di.ensure(static_cast<size_t>(g));
  CheckCuda(cudaMemcpyAsync(dq.p, hq.data(), sizeof(int) * static_cast<size_t>(g), cudaMemcpyHostToDevice, stream_),
            "h2d");
  CheckCuda(cudaMemcpyAsync(di.p, idx.data(), sizeof(int) * static_cast<size_t>(g), cudaMemcpyHostToDevice, stream_),
            "h2d");
  ++launches_;
  ScatterGroupKernel<<<(g + 255) / 256, 256, 0, stream_>>>(dq.p, di.p, g, d_group_of_.p, d_idx_in_group_.p);
  std::vector<int> sorted(hq);
  std::sort(sorted.begin(), sorted.end());
  members_repeat_ = std::adjacent_find(sorted.begin(), sorted.end()) != sorted.end();
  PrepareIterationBuffers();
  members_repeat_ = false;
  CheckCuda(cudaMemsetAsync(d_ctl_.p, 0, sizeof(BlockCtl), stream_), "memset ctl");
  LaunchPrepare(plans_.at(0));
  int cnt = 0;
  CheckCuda(cudaMemcpyAsync(&cnt, d_cand_cnt_.p, sizeof(int), cudaMemcpyDeviceToHost, stream_), "d2h");
  CheckCuda(cudaStreamSynchronize(stream_), "prepare sync");
  CheckError();
  std::vector<int2> h(static_cast<size_t>(cnt));
  if (cnt > 0) {
    CheckCuda(cudaMemcpy(h.data(), d_cand_.p, sizeof(int2) * static_cast<size_t>(cnt), cudaMemcpyDeviceToHost),
              "d2h cand");
  }
  for (int i = 0; i < cnt && i < cap; ++i) {
    a_idx[i] = h[static_cast<size_t>(i)].x;
    b_idx[i] = h[static_cast<size_t>(i)].y;
  }
  n_groups_ = -1;
  return cnt;
}

void Engine::MergePairs(const int32_t* keep, const int32_t* remove, int64_t count) {
  AllocScope alloc(stream_);
  if (count <= 0) return;
  known_active_ = -1;
  std::vector<char> seen(static_cast<size_t>(n_), 0);
  for (int64_t i = 0; i < count; ++i) {
    const int k = keep[i], r = remove[i];
    if (k < 0 || r < 0 || k >= n_ || r >= n_ || k == r) throw std::invalid_argument("invalid merge endpoints");
    if (seen[static_cast<size_t>(k)] || seen[static_cast<size_t>(r)]) {
      throw std::invalid_argument("merge batch requires endpoint-disjoint pairs");
    }
    seen[static_cast<size_t>(k)] = 1;
    seen[static_cast<size_t>(r)] = 1;
  }
  std::vector<int> hs(static_cast<size_t>(n_));
  CheckCuda(cudaMemcpy(hs.data(), d_qsize_.p, sizeof(int) * static_cast<size_t>(n_), cudaMemcpyDeviceToHost), "d2h");
  for (int64_t i = 0; i < count; ++i) {
    if (hs[static_cast<size_t>(keep[i])] <= 0 || hs[static_cast<size_t>(remove[i])] <= 0) {
      throw std::invalid_argument("quotient supernode is inactive");
    }
  }
  EnsurePoolRoom();
  // the batch is one pseudo-group's selection list
  const int cnt = static_cast<int>(count);
  h_sel_off_.assign(2, 0);
  h_sel_off_[1] = count;
  d_sel_off_.ensure(2);
  d_sel_cnt_.ensure(1);
  d_sel_keep_.ensure(static_cast<size_t>(count));
  d_sel_rem_.ensure(static_cast<size_t>(count));
  d_sel_gain_.ensure(static_cast<size_t>(count));
  CheckCuda(cudaMemcpyAsync(d_sel_off_.p, h_sel_off_.data(), 2 * sizeof(long long), cudaMemcpyHostToDevice, stream_),
            "h2d");
  CheckCuda(cudaMemcpyAsync(d_sel_cnt_.p, &cnt, sizeof(int), cudaMemcpyHostToDevice, stream_), "h2d");
  CheckCuda(cudaMemcpyAsync(d_sel_keep_.p, keep, sizeof(int) * static_cast<size_t>(count), cudaMemcpyHostToDevice,
                            stream_), "h2d");
  CheckCuda(cudaMemcpyAsync(d_sel_rem_.p, remove, sizeof(int) * static_cast<size_t>(count), cudaMemcpyHostToDevice,
                            stream_), "h2d");
  CheckCuda(cudaMemsetAsync(d_sel_gain_.p, 0, sizeof(long long) * static_cast<size_t>(count), stream_), "memset");
  ++block_stamp_;
  CheckCuda(cudaMemsetAsync(d_ctl_.p, 0, sizeof(BlockCtl), stream_), "memset ctl");
  ++launches_;
  MarkKernel<<<(cnt + 255) / 256, 256, 0, stream_>>>(d_sel_keep_.p, d_sel_rem_.p, cnt, d_stamp_.p, d_partner_.p,
                                                    d_seq_.p, block_stamp_, d_sel_list_.p, d_ctl_.p);
  LaunchCommit(0, 1, count, false, nullptr);
  ++launches_;
  LaunchFollowing(RelabelKernel, (n_ + 255) / 256, 256, 0, stream_, d_label_.p, d_fwd_.p, n_);
  n_groups_ = -1;
  CheckCuda(cudaStreamSynchronize(stream_), "merge pairs sync");
  CheckError();
}

}  // namespace beam
