// Merge over windows of blocks: the plain form (blocks of a few groups), with
// the groups of many blocks evaluated at once. Included by merge.cu only.
//
// The reference handles its blocks one after another, since a block's merges
// change rows that later blocks read. A merge of (k, r) changes what another
// group sees only through members that are neighbours of k or r (their rows
// and the sizes behind them), and on a large graph few of the next blocks'
// groups hold such a member. So a window of groups is evaluated (candidates,
// exact gains, selection) against one state, and
//   - each selected pair's neighbours give the first later group that it
//     touches; the smallest of these over the window is the first block whose
//     evaluation may be out of date;
//   - every block before it is committed as one batch: none of them touches
//     another, so the batch is the sequence of their commits;
//   - the evaluated groups that the batch touched are evaluated again, together
//     with the groups that the window takes in next.
// The decisions, counters and rows are those of the blocks in order; only
// evaluations that stood when their block's turn came are counted.
//
// One round is nine launches that take their work from device memory, for as
// many blocks as turned out independent (a block at a time took a dozen
// launches, 75 to 120 us, latency only). Rounds follow each other without the
// host, which watches the frontier through mapped memory and keeps a few
// rounds queued. Measured with 64-group blocks, 20 iterations, a block at a time
// -> windows: R-MAT 16 (edge factor 8) 609 -> 116 ms, R-MAT 12 36.7 -> 13.8 ms,
// Chung-Lu of 20,000 nodes with twins 108 -> 49 ms.
#pragma once

// Blocks of at most this many groups go through windows; larger ones fill the
// GPU by themselves and touch too much of each other. 20 iterations a block at a
// time -> windows, blocks of 512, 1024 and 2048 groups: grid + Chung-Lu union of
// 0.5 M nodes 836 -> 295, 590 -> 257, 410 -> 215 ms; Chung-Lu of 100,000 nodes
// 169 -> 107, 118 -> 83, 79 -> 65; R-MAT 15 (edge factor 16) 71 -> 54, 50 -> 46,
// 37 -> 41; a uniform graph of 20,000 nodes 15.9 -> 12.2, 11.6 -> 10.9, 9.1 -> 10.0.
constexpr int kWindowMaxBatch = 1024;
constexpr int kWindowMaxGroups = 8192;  // groups a window takes in at most (then to the block's end)
constexpr int kWindowMinGroups = 256;
constexpr int kWindowMinAgain = 64;
// Tables of a round's big groups take at most this much memory, unless one block
// needs more by itself: an iteration whose tables are beyond it in all goes
// through windows of fewer groups (WindowSpanKernel). 4.5 KB a node in groups of
// 500 members, 9 KB at 1,024, else limit the graphs that fit. Runs with the limit
// at one block / 64 MB / 256 MB / 1 GB / 4 GB / none: 2 M nodes in groups of 500,
// two iterations, 1070 / 228 / 146 / 121 / 133 / 138 ms; R-MAT 20 (edge factor
// 16), two iterations, 1153 / 267 / 112 / 111 / 110 / 111; R-MAT 22 with groups of
// up to 1,024, one iteration, 2434 / 861 / 476 / 390 / 387 / 384.
constexpr long long kWindowTables = 4ll << 30;
constexpr int kWindowLengths = 14;  // kWindowMaxGroups, halved down to 1 (then to the block's end)
static_assert(kWindowMaxGroups >> (kWindowLengths - 1) == 1, "the last length is one block");
constexpr int kWindowList = 2 * (kWindowMaxGroups + kWindowMaxBatch) + 1024;
constexpr int kEvalWarps = 4;
constexpr int kEvalCtas = 8;     // per SM
constexpr int kEvalGrid = 152 * kEvalCtas;
constexpr int kBigGrid = 152 * 2;
constexpr int kMarkGrid = 16;
constexpr int kMarkThreads = 256;
constexpr int kWindowAhead = 2;  // rounds queued by the host and not seen done
// Rows longer than this are handed on in units, so that no warp holds up a
// round with a hub's row.
constexpr int kLongRow = 256;
constexpr int kLongRowUnit = 256;   // entries per unit
constexpr int kLongUnits = 1 << 19;  // units at most; what does not fit is done in place
constexpr int kLongThreads = 256;
constexpr int kLongGrid = 152 * 6;
// A warp handles a group of this size alone. Its steps are a chain, 5 us at
// this size and up to 75 us at 17 members with 256 entries; spread over the
// GPU, larger groups cost three more launches' latency and little else.
constexpr int kEvalSmall = 8;
constexpr int kEvalEntries = 64;
constexpr int kEvalSmallPairs = kEvalSmall * (kEvalSmall - 1) / 2;
// Pair pass: rows of at most kTableRow entries go into a warp's hash table of
// kTableSlots; a group's members are split in parts of about kPartEntries.
constexpr int kTableRow = 512;
constexpr int kTableSlots = 2 * kTableRow;
constexpr int kPartEntries = 1024;
constexpr int kMaxParts = 128;
constexpr int kPairWarps = 4;
constexpr int kPairDeep = 4;  // entries per lane in flight
// Per SM: what shared memory holds (42 KB of tables each). With a grid of six,
// a sixth of the work is a second wave: R-MAT 16 118.7 ms, 116.0 with five.
constexpr int kPairCtas = 5;
constexpr int kPairGrid = 152 * kPairCtas;

__host__ __device__ __forceinline__ int WindowParts(unsigned entries) {
  const unsigned p = (entries + kPartEntries - 1) / kPartEntries;
  return p < 1 ? 1 : p > static_cast<unsigned>(kMaxParts) ? kMaxParts : static_cast<int>(p);
}

// A big group's memory: the pair tables and old costs, every member's place
// among the staged entries (first, length, size), the staged entries.
__host__ __device__ __forceinline__ long long PlaceOffset(long long g) { return (OldCostOffset(g * g) + 8 * g + 15) & ~15ll; }
__host__ __device__ __forceinline__ long long StageOffset(long long g) { return PlaceOffset(g) + 16 * g; }
__host__ __device__ __forceinline__ long long WindowBytes(long long g, unsigned entries) {
  return (StageOffset(g) + 16ll * entries + 255) & ~255ll;
}

// A listed big group, for one load in the kernels.
struct __align__(16) BigGroup {
  int ri, gid, g, cap;  // cap: entries that the stage holds
  int gstart, parts;
  long long mat;
};

struct __align__(16) StagedEntry {
  int t;       // target
  int size;    // its size
  unsigned c;  // edges
  int j;       // member
};

struct WindowCtl {
  int f, e, R;     // first group not committed; end of the evaluated groups; groups of the iteration
  int p;           // end of the batch being committed
  int stale;       // first evaluated group that is out of date and not listed (INT_MAX: none)
  int pace;        // groups that a round commits, on average
  int nsmall, nbig, ndirty;
  long long members, parts;  // of the listed big groups: members, and members times parts
  unsigned long long work;  // queue of the evaluation kernel
  unsigned units;            // long units handed on
  unsigned pad;
  long long blocks;          // blocks with at least one group (per iteration)
  int rounds;                // lists made in this iteration
};
static_assert(sizeof(WindowCtl) <= 256, "room made in Engine::Reset");

// An evaluation's share of the counters, added when its block is committed.
struct GroupStats {
  unsigned long long examined, cand, uni, ovl, raw_a, raw_b, nnz, rejected, positive, selected, gain, work, entries;
  int err, err_a, err_b, pad;
  int staged_short, staged_long;  // entries staged, of the rows with and without a table
};
constexpr int kGroupStatWords = 13;
static_assert(sizeof(GroupStats) == 128, "");

// Part of a long row.
struct LongUnit {
  unsigned long long* old;  // the member's approximate old cost
  StagedEntry* stage;       // the row's place
  int rep, i;
  int at;  // first entry
  int ri;  // group, -1: nothing to do
};

struct WindowParams {
  QuotientView Q;
  const int* order;
  const int* gstart;
  const int* glen;
  const unsigned* gent;
  const int* group_of;
  const int* real;
  const int* node_ri;   // per active supernode: its group's position, -1 alone
  const int* blk_end;   // per group position: first position of the next block
  const int* blk_beg;   //                     first position of its own block
  const int* idx_in_group;
  WindowCtl* ctl;
  GroupStats* gs;
  int* conflict;        // per group position: first later group its pairs touch (INT_MAX: none)
  LongUnit* units;
  int* dirty;           // per group position: 1 touched since its evaluation (and on list_dirty)
  int* list_dirty;
  int* list_small;
  BigGroup* list_big;
  long long* moff;      // member / part prefixes over list_big
  long long* poff;
  const long long* mat_off;  // per group position: bytes of the tables before its own
  unsigned char* mat;        // tables of the window's groups, from the first not committed
  int max_groups;            // groups that a window takes in at most, by the room for their tables
  const long long* cand_off;
  unsigned long long* keys;  // two per candidate slot
  RowSums* rc;
  const long long* sel_off;
  int* sel_keep;
  int* sel_rem;
  long long* sel_gain;
  int* sel_cnt;
  int* stamp;
  int* partner;
  int* seq;
  int* sel_list;
  BlockCtl* bctl;
  int block_stamp;
  int top_k;
  double threshold;
  ThresholdBits thr;
  int use_threshold;
  int all_strict;  // no block has more than kFewGroups groups
  unsigned long long* stats;
  DevError* err;
  volatile int* host_f;  // mapped: the frontier, and the lists made so far
};

__device__ __forceinline__ bool WindowSmall(int g, unsigned entries) {
  return g <= kEvalSmall && entries <= static_cast<unsigned>(kEvalEntries);
}

// ------------------------------------------------------------ lists

// Per active supernode its group position, per group position the ends of its
// block and a clean mark, and the number of blocks.
__global__ void WindowSetupKernel(const int* order, const int* group_of, const int* ri_of, int count, const int* real,
                                  int R, int batch, int* node_ri, int* blk_beg, int* blk_end, int* dirty,
                                  WindowCtl* ctl) {
  FollowsOn();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) {
    const int rep = order[i];
    node_ri[rep] = ri_of[group_of[rep]];
  }
  if (i < R) {
    const int b = real[i] / batch;
    int lo = i, hi = R;  // first position of a later block
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (real[mid] / batch <= b) lo = mid + 1; else hi = mid;
    }
    blk_end[i] = lo;
    lo = 0, hi = i;  // first position of this block
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (real[mid] / batch < b) lo = mid + 1; else hi = mid;
    }
    blk_beg[i] = lo;
    dirty[i] = 0;
    if (i == 0 || real[i - 1] / batch != b) atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->blocks), 1ull);
  }
}

// Bytes of the tables of a window of at most kWindowMaxGroups >> k groups, the
// most over all blocks that it may start with. A round's groups lie between the
// first block not committed and the end of the blocks taken in (no further than
// the window's length from that block, or from an earlier one).
__global__ void WindowSpanKernel(const long long* mat_off, const int* blk_beg, const int* blk_end, int R,
                                 unsigned long long* most) {
  FollowsOn();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool starts = i < R && blk_beg[i] == i;
  for (int k = 0; k < kWindowLengths; ++k) {
    long long bytes = 0;
    if (starts) bytes = mat_off[blk_end[min(i + (kWindowMaxGroups >> k), R) - 1]] - mat_off[i];
    bytes = WarpMax(bytes);
    if ((threadIdx.x & 31) == 0 && bytes > 0) atomicMax(&most[k], static_cast<unsigned long long>(bytes));
  }
}

// The next evaluation's lists, by one CTA of kHugeThreads: the touched groups
// and those that the window takes in. `done`: groups [f, p) are committed.
struct ListSum {
  long long members, parts;
  int small, big;
};
struct ListSumOp {
  __device__ __forceinline__ ListSum operator()(const ListSum& a, const ListSum& b) const {
    return ListSum{a.members + b.members, a.parts + b.parts, a.small + b.small, a.big + b.big};
  }
};

__device__ __noinline__ void BuildLists(const WindowParams& P) {
  using Scan = cub::BlockScan<ListSum, kHugeThreads, cub::BLOCK_SCAN_WARP_SCANS>;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ ListSum carry;
  __shared__ int s_e0, s_e1, s_dirty, s_again, s_kept, s_stale;
  __shared__ long long s_mat0;  // the window's first table
  WindowCtl* c = P.ctl;
  if (threadIdx.x == 0) {
    // (what does not wait for the pace is loaded first: one memory latency)
    const int f = c->p, e0 = c->e, R = c->R;
    const int next = f < R ? P.blk_end[f] : 0;
    const long long mat0 = P.mat_off[f];
    // new groups are taken in for the next two rounds at the usual pace (the
    // whole window again where all of it was committed); a touched group is
    // evaluated again when its turn is that near, not every time it is touched
    const int committed = f - c->f;
    int pace = c->pace;
    if (f > 0) pace = f == e0 ? max(committed, pace) : (3 * pace + committed) / 4;
    pace = min(pace, kWindowMaxGroups / 2);
    const int take = min(max(2 * pace, kWindowMinGroups), P.max_groups);
    int e = f + take;
    e = e >= R ? R : e == 0 ? 0 : P.blk_end[e - 1];
    s_e0 = e0;
    s_e1 = e > e0 ? e : e0;
    s_dirty = c->ndirty;
    // (the next block in any case, so that every round commits one)
    s_again = max(f + max(2 * pace, kWindowMinAgain), next);
    s_mat0 = mat0;
    s_kept = 0;
    s_stale = 0x7fffffff;
    carry = ListSum{0, 0, 0, 0};
    c->pace = pace;
    c->f = f;
  }
  __syncthreads();
  const int n = s_dirty + (s_e1 - s_e0);
  for (int base = 0; base < n; base += kHugeThreads) {
    const int i = base + threadIdx.x;
    int ri = -1, g = 0, gid = 0;
    unsigned entries = 0;
    ListSum v{0, 0, 0, 0};
    bool later = false;
    if (i < n) {
      ri = i < s_dirty ? P.list_dirty[i] : s_e0 + (i - s_dirty);
      later = i < s_dirty && ri >= s_again;
    }
    __syncthreads();  // the list's entries are read before the kept ones move down
    if (later) {
      P.list_dirty[atomicAdd(&s_kept, 1)] = ri;
      atomicMin(&s_stale, ri);
    } else if (i < n) {
      P.dirty[ri] = 0;
      gid = P.real[ri];
      g = P.glen[gid];
      entries = P.gent[gid];
      if (WindowSmall(g, entries)) {
        v.small = 1;
      } else {
        v.big = 1;
        v.members = g;
        v.parts = static_cast<long long>(g) * WindowParts(entries);
      }
      GroupStats z = {};
      P.gs[ri] = z;
      P.conflict[ri] = 0x7fffffff;
    }
    ListSum ex, total;
    Scan(tmp).ExclusiveScan(v, ex, ListSum{0, 0, 0, 0}, ListSumOp(), total);
    const ListSum c0 = carry;
    if (v.small) P.list_small[c0.small + ex.small] = ri;
    if (v.big) {
      P.list_big[c0.big + ex.big] =
          BigGroup{ri, gid, g, static_cast<int>(entries), P.gstart[gid], WindowParts(entries), P.mat_off[ri] - s_mat0};
      P.moff[c0.big + ex.big] = c0.members + ex.members;
      P.poff[c0.big + ex.big] = c0.parts + ex.parts;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry = ListSumOp()(c0, total);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    P.moff[carry.big] = carry.members;
    P.poff[carry.big] = carry.parts;
    c->nsmall = carry.small;
    c->nbig = carry.big;
    c->members = carry.members;
    c->parts = carry.parts;
    c->ndirty = s_kept;
    c->stale = s_stale;
    c->work = 0;
    c->units = 0;
    c->e = s_e1;
    P.host_f[0] = c->f;
    __threadfence_system();
    P.host_f[1] = ++c->rounds;
  }
}

__global__ void __launch_bounds__(kHugeThreads) WindowBeginKernel(WindowParams P, int R) {
  FollowsOn();
  if (threadIdx.x == 0) {
    P.ctl->f = P.ctl->e = P.ctl->p = 0;
    P.ctl->R = R;
    P.ctl->rounds = 0;
    P.ctl->ndirty = 0;
  }
  __syncthreads();
  BuildLists(P);
}

// ------------------------------------------------------------ evaluation

// Whether a pair of this group is checked against its rows' own capacities too,
// as for a block committed by itself (ScoreParams::strict).
__device__ __forceinline__ int WindowStrict(const WindowParams& P, int ri) {
  return P.all_strict || P.blk_end[ri] - P.blk_beg[ri] <= kFewGroups ? 1 : 0;
}

// First later group (another block) that merging a and b touches: by a warp,
// over one row given by its entries.
__device__ __forceinline__ int FirstTouched(const WindowParams& P, const Entry* row, int len, int end, int first,
                                            int stride) {
  int best = 0x7fffffff;
  for (int k = first; k < len; k += stride) {
    const int ri = P.node_ri[EntNb(row[k])];
    if (ri >= end && ri < best) best = ri;
  }
  return best;
}

struct EvalWarpSmem {
  SmallRowsSmem rows;
  SmallPairsSmem<kEvalSmallPairs> pairs;  // the first array holds the selection keys in the end
  RowSums rs[kEvalSmall];
};
struct EvalSmem {
  EvalWarpSmem w[kEvalWarps];
};
static_assert(kEvalCtas * (sizeof(EvalSmem) + kSmemReserved) <= kSmemPerSm, "the grid is one wave");

// A small group by one warp: candidates, gains and selection.
__device__ void EvalSmallGroup(const WindowParams& P, EvalWarpSmem& W, int ri) {
  constexpr unsigned kFull = 0xffffffffu;
  SmallRowsSmem& S = W.rows;
  const int lane = threadIdx.x & 31;
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  __syncwarp();
  bool wide;
  const int E = StageSmallRows(P.Q, P.order + P.gstart[gid], g, S, &wide);
  GroupStats* gs = P.gs + ri;
  if (E > kSmallStage) {
    if (lane == 0) {
      gs->err = kErrSlots;
      gs->err_a = gid;
      gs->err_b = E;
      P.sel_cnt[ri] = 0;
    }
    return;
  }
  bool slow;
  unsigned examined = SmallSums(P.Q, S, W.pairs, g, E, wide, &slow);
  if (lane < g) SmallFinishRow(P.Q, S, lane, wide, &W.rs[lane]);
  __syncwarp();
  const int npairs = g * (g - 1) / 2;
  SmallTopK(S, g, P.top_k, [&](int a, int b) {
    return slow ? SmallMerge(S, a, b).proxy : static_cast<long long>(W.pairs.pc[TriIndex(a, b, g)] >> 32);
  });
  // gains of the kept pairs, one lane each; the keys of those that pass
  const int strict = WindowStrict(P, ri);
  long long uni = 0, ovl = 0, raw_a = 0, raw_b = 0, nnz = 0;
  int cand = 0, passed = 0, err = 0, err_a = 0, err_b = 0;
  for (int pidx = lane; pidx < npairs; pidx += 32) {
    int a, b;
    TriPair(pidx, g, &a, &b);
    unsigned long long key = ~0ull;
    if ((S.fmask[a] >> b) & 1u) {
      const PairInfo pi = SmallPairInfo(S, a, b, SmallPairAt(S, W.pairs, pidx, a, b, slow));
      const RowSums &A = W.rs[a], &B = W.rs[b];
      GainParts gp;
      if (!GainFromSums(A, B, pi, strict, &gp)) {
        const long long s = static_cast<long long>(A.size) + B.size;
        long long part;
        if (!RowAfter(A, s, &part)) gp.gain += part - StagedRowAfter(S, a, s);
        if (!RowAfter(B, s, &part)) gp.gain += part - StagedRowAfter(S, b, s);
      }
      ++cand;
      uni += gp.uni;
      ovl += gp.ovl;
      raw_a += A.len;
      raw_b += B.len;
      nnz += A.len + (A.internal > 0 ? 1 : 0) + B.len + (B.internal > 0 ? 1 : 0);
      if (PassesFilter(gp.gain, gp.before, P.threshold, P.thr, P.use_threshold)) {
        ++passed;
        if (gp.gain > kKeyGainMax) gp.err = kErrKeyRange;
        key = PackKey(gp.gain, a, b);
      }
      if (gp.err && !err) {
        err = gp.err;
        err_a = S.q[a];
        err_b = S.q[b];
      }
    }
    W.pairs.pc[pidx] = key;
  }
  __syncwarp();
  cand = WarpSumInt(cand);
  passed = WarpSumInt(passed);
  // g0: the smallest key whose ends are both free, again and again
  const long long so = P.sel_off[ri];
  const int end = P.blk_end[ri];
  unsigned used = 0;
  int ns = 0, conflict = 0x7fffffff;
  long long total = 0;
  unsigned long long work = 0;
  while (passed > 0) {
    unsigned long long best = ~0ull;
    for (int k = lane; k < npairs; k += 32) {
      const unsigned long long key = W.pairs.pc[k];
      if (key >= best) continue;
      const int b = static_cast<int>(key & kKeyIdxMask);
      const int a = static_cast<int>((key >> kKeyIdxBits) & kKeyIdxMask);
      if (!((used >> a | used >> b) & 1u)) best = key;
    }
    const unsigned hi = __reduce_min_sync(kFull, static_cast<unsigned>(best >> 32));
    const unsigned lo =
        __reduce_min_sync(kFull, static_cast<unsigned>(best >> 32) == hi ? static_cast<unsigned>(best) : 0xffffffffu);
    best = static_cast<unsigned long long>(hi) << 32 | lo;
    if (best == ~0ull) break;
    const int b = static_cast<int>(best & kKeyIdxMask);
    const int a = static_cast<int>((best >> kKeyIdxBits) & kKeyIdxMask);
    used |= 1u << a | 1u << b;
    const long long gain = kKeyGainMax - static_cast<long long>(best >> (2 * kKeyIdxBits));
    if (lane == 0) {
      P.sel_keep[so + ns] = S.q[a];
      P.sel_rem[so + ns] = S.q[b];
      P.sel_gain[so + ns] = gain;
    }
    ++ns;
    total += gain;
    work += static_cast<unsigned long long>(W.rs[a].len + W.rs[b].len);
    const int ca = FirstTouched(P, S.ent + S.start[a], W.rs[a].len, end, lane, 32);
    const int cb = FirstTouched(P, S.ent + S.start[b], W.rs[b].len, end, lane, 32);
    conflict = min(conflict, min(ca, cb));
  }
  conflict = static_cast<int>(__reduce_min_sync(kFull, conflict));
  examined = __reduce_add_sync(kFull, examined);
  uni = WarpSum(uni);
  ovl = WarpSum(ovl);
  raw_a = WarpSum(raw_a);
  raw_b = WarpSum(raw_b);
  nnz = WarpSum(nnz);
  const unsigned failed = __ballot_sync(kFull, err != 0);
  if (failed) {
    const int src = __ffs(failed) - 1;
    err = __shfl_sync(kFull, err, src);
    err_a = __shfl_sync(kFull, err_a, src);
    err_b = __shfl_sync(kFull, err_b, src);
  }
  if (lane == 0) {
    GroupStats z;
    z.examined = examined;
    z.cand = cand;
    z.uni = uni;
    z.ovl = ovl;
    z.raw_a = raw_a;
    z.raw_b = raw_b;
    z.nnz = nnz;
    z.rejected = cand - passed;
    z.positive = passed;
    z.selected = ns;
    z.gain = total;
    z.work = work;
    z.entries = E;
    z.err = err;
    z.err_a = err_a;
    z.err_b = err_b;
    z.pad = 0;
    *gs = z;
    P.conflict[ri] = conflict;
    P.sel_cnt[ri] = ns;
  }
}

// Hands `count` entries on in units of `per`; false: no room, to be done in place.
__device__ __forceinline__ bool PushUnits(const WindowParams& P, LongUnit u, int count, int per) {
  const int lane = threadIdx.x & 31;
  const unsigned n = static_cast<unsigned>((count + per - 1) / per);
  unsigned at = 0;
  if (lane == 0) at = atomicAdd(&P.ctl->units, n);
  at = __shfl_sync(0xffffffffu, at, 0);
  const bool fits = at + n <= kLongUnits && at + n >= n;
  for (unsigned k = lane; k < n && at + k < kLongUnits && at + k >= at; k += 32) {
    LongUnit v = u;
    v.at = static_cast<int>(k) * per;
    if (!fits) v.ri = -1;
    P.units[at + k] = v;
  }
  return fits;
}

struct RowPart {
  long long old = 0, light = 0;
  HeavyAcc heavy;
};

// Entries [k0, k1) of member i's row staged and summed, by a warp (sums of the
// whole warp on return).
__device__ __forceinline__ void SumEntries(const QuotientView& Q, const Entry* row, int k0, int k1, int rep,
                                           long long si, int i, StagedEntry* stage, RowPart* out) {
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int k = k0 + lane; k < k1; k += 32) {
    const Entry e = row[k];
    const long long c = EntCnt(e);
    const long long st = Q.size[EntNb(e)];
    stage[k] = StagedEntry{EntNb(e), static_cast<int>(st), static_cast<unsigned>(c), i};
    out->old += EncodeCostForPair(rep, si, EntNb(e), st, c);
    if (HeavyEntry(si, st, c)) out->heavy.Add(st, c); else out->light += c;
  }
  out->old = WarpSum(out->old);
  out->light = WarpSum(out->light);
  out->heavy.WarpReduce();
}

// Member i of a big group by one warp: its row sums and approximate old cost,
// its rows of the pair tables cleared, its entries staged beside the other
// members' (rows that fit a table from the front, longer ones from the back).
__device__ void EvalMember(const WindowParams& P, const BigGroup& G, int i) {
  const int lane = threadIdx.x & 31;
  const QuotientView& Q = P.Q;
  const int ri = G.ri, g = G.g, cap = G.cap;
  const int rep = P.order[G.gstart + i];
  unsigned char* mat = P.mat + G.mat;
  unsigned long long* words = reinterpret_cast<unsigned long long*>(mat) + static_cast<long long>(i) * g;
  unsigned char* flags = mat + FlagOffset(static_cast<long long>(g) * g) + static_cast<long long>(i) * g;
  for (int k = lane; k < g; k += 32) {
    words[k] = 0;
    flags[k] = 0;
  }
  const long long si = Q.size[rep];
  const int len = Q.len[rep];
  const Entry* row = Q.ent + Q.off[rep];
  const long long internal = Q.internal[rep];
  const long long own = internal > 0 ? EncodeCostForPair(rep, si, rep, si, 2 * internal) : 0;
  long long* old_out = reinterpret_cast<long long*>(mat + OldCostOffset(static_cast<long long>(g) * g)) + i;
  GroupStats* gs = P.gs + ri;
  int at = 0;
  if (lane == 0) {
    atomicAdd(&gs->entries, static_cast<unsigned long long>(len));
    if (len <= kTableRow) {
      at = atomicAdd(&gs->staged_short, len);
    } else {
      at = cap - atomicAdd(&gs->staged_long, len) - len;
    }
  }
  at = __shfl_sync(0xffffffffu, at, 0);
  const bool fits = at >= 0 && at + len <= cap;  // rows counted at Divide time only shrink
  if (lane == 0) {
    reinterpret_cast<int4*>(mat + PlaceOffset(g))[i] = make_int4(at, fits ? len : 0, static_cast<int>(si), 0);
    if (!fits) {
      gs->err = kErrSlots;
      gs->err_a = G.gid;
      gs->err_b = len;
    }
  }
  StagedEntry* stage = reinterpret_cast<StagedEntry*>(mat + StageOffset(g)) + at;
  if (!fits) return;
  if (len > kLongRow) {
    const LongUnit u{reinterpret_cast<unsigned long long*>(old_out), stage, rep, i, 0, ri};
    if (PushUnits(P, u, len, kLongRowUnit)) {
      // the units stage and add their entries
      if (lane == 0) {
        StoreRowSums(&P.rc[rep], 0, 0, HeavyAcc(), internal, static_cast<int>(si), len);
        *old_out = own;
      }
      return;
    }
  }
  RowPart r;
  SumEntries(Q, row, 0, len, rep, si, i, stage, &r);
  if (lane == 0) {
    StoreRowSums(&P.rc[rep], r.old, r.light, r.heavy, internal, static_cast<int>(si), len);
    *old_out = r.old + own;
  }
}

// Work items in one queue: the members of the big groups, then the small
// groups. One warp each.
__global__ void __launch_bounds__(kEvalWarps * 32, kEvalCtas) WindowEvalKernel(WindowParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  EvalWarpSmem& W = reinterpret_cast<EvalSmem*>(smem_raw)->w[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const long long nm = P.ctl->members;
  const int ns = P.ctl->nsmall, nb = P.ctl->nbig;
  for (;;) {
    long long it = 0;
    if (lane == 0) it = static_cast<long long>(atomicAdd(&P.ctl->work, 1ull));
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it < nm) {
      const int bl = WarpLastLE(P.moff, 0, nb, it);
      EvalMember(P, P.list_big[bl], static_cast<int>(it - P.moff[bl]));
    } else if (it < nm + ns) {
      EvalSmallGroup(P, W, P.list_small[it - nm]);
    } else {
      break;
    }
  }
}

// The long units, a warp each: entries staged, row sums added up.
__global__ void __launch_bounds__(kLongThreads) WindowLongKernel(WindowParams P) {
  FollowsOn();
  const QuotientView& Q = P.Q;
  const int lane = threadIdx.x & 31;
  const unsigned total = P.ctl->units < kLongUnits ? P.ctl->units : kLongUnits;
  const unsigned nw = (gridDim.x * blockDim.x) >> 5;
  for (unsigned t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total; t += nw) {
    const LongUnit u = P.units[t];
    if (u.ri < 0) continue;
    const int len = Q.len[u.rep];
    RowPart r;
    SumEntries(Q, Q.ent + Q.off[u.rep], u.at, min(u.at + kLongRowUnit, len), u.rep, Q.size[u.rep], u.i, u.stage, &r);
    if (lane == 0) {
      RowSums* s = &P.rc[u.rep];
      atomicAdd(u.old, static_cast<unsigned long long>(r.old));
      atomicAdd(reinterpret_cast<unsigned long long*>(&s->before), static_cast<unsigned long long>(r.old));
      atomicAdd(reinterpret_cast<unsigned long long*>(&s->light), static_cast<unsigned long long>(r.light));
      if (r.heavy.n != 0) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&s->heavy_sx), static_cast<unsigned long long>(r.heavy.sx));
        atomicAdd(reinterpret_cast<unsigned long long*>(&s->heavy_c), static_cast<unsigned long long>(r.heavy.c));
        atomicMin(&s->smin, r.heavy.smin);
        atomicMax(&s->smax, r.heavy.smax);
        atomicMax(&s->sbad, r.heavy.sbad);
        atomicAdd(&s->nheavy, r.heavy.n);
      }
    }
  }
}

struct PairTable {
  int key[kTableSlots];  // target, -1 free
  unsigned cnt[kTableSlots];
  int4 hit[32 + 32 * kPairDeep];  // found: member, target's size, the member's count, the table's count
};
static_assert(kPairCtas * (kPairWarps * sizeof(PairTable) + kSmemReserved) <= kSmemPerSm, "the grid is one wave");

__device__ __forceinline__ int StagedLowerBound(const StagedEntry* row, int len, int t) {
  int lo = 0, hi = len;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (row[mid].t < t) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// The pair words of the big groups, a warp per member and part. A row of at
// most kTableRow entries goes into a hash table in shared memory, and the
// entries of the rows staged after it, and of all longer rows, are looked up in
// it, four per lane in flight: two or three instructions' worth of lookups per
// entry, where merging the rows pair by pair took 200 instructions and a chain
// of loads per pair. What is found is queued and added up 32 at a time (a few
// in a hundred lookups find something: handled in place, nearly every step
// would wait for its one or two lanes). Two long rows are
// matched by searching the shorter one's entries in the other.
__global__ void __launch_bounds__(kPairWarps * 32, kPairCtas) WindowPairsKernel(WindowParams P) {
  FollowsOn();
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kDeep = kPairDeep;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PairTable& T = reinterpret_cast<PairTable*>(smem_raw)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int nb = P.ctl->nbig;
  const long long total = P.ctl->parts;
  const long long nw = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long it = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; it < total; it += nw) {
    const int bl = WarpLastLE(P.poff, 0, nb, it);
    const BigGroup G = P.list_big[bl];
    const int ri = G.ri, gid = G.gid, g = G.g, cap = G.cap, parts = G.parts;
    const int local = static_cast<int>(it - P.poff[bl]);
    const int part = local / g, i = local - part * g;  // a part's members side by side
    unsigned char* mat = P.mat + G.mat;
    unsigned long long* pmat = reinterpret_cast<unsigned long long*>(mat);
    const int4* place = reinterpret_cast<const int4*>(mat + PlaceOffset(g));
    const StagedEntry* stage = reinterpret_cast<const StagedEntry*>(mat + StageOffset(g));
    const int4 me = place[i];
    if (me.y == 0) continue;
    const long long si = me.z;
    unsigned examined = 0;
    auto direct = [&](const StagedEntry& e) {
      if (P.group_of[e.t] == gid) AddDirect(pmat, g, i, P.idx_in_group[e.t], e.c);
    };
    if (me.y <= kTableRow) {
      int mask = 32;
      while (mask < 2 * me.y) mask <<= 1;
      --mask;
      __syncwarp();
      for (int k = lane; k <= mask; k += 32) T.key[k] = -1;
      __syncwarp();
      for (int k = lane; k < me.y; k += 32) {
        const StagedEntry e = stage[me.x + k];
        int h = static_cast<int>(BucketHash(e.t, mask));
        while (atomicCAS(&T.key[h], -1, e.t) != -1) h = (h + 1) & mask;
        T.cnt[h] = e.c;
        if (part == 0) direct(e);
      }
      __syncwarp();
      int queued = 0;
      auto add = [&](const int4& x) {
        ++examined;
        AddShared(pmat, g, i, x.x, si, place[x.x].z, x.y, static_cast<unsigned>(x.w), static_cast<unsigned>(x.z), true);
      };
      // the entries to look up: the shorter rows staged later, the longer rows
      const int first = me.x + me.y, n1 = P.gs[ri].staged_short - first;
      const int n2 = P.gs[ri].staged_long, back = cap - n2;
      const long long n = static_cast<long long>(n1) + n2;
      const int k0 = static_cast<int>(n * part / parts), k1 = static_cast<int>(n * (part + 1) / parts);
      for (int b = k0; b < k1; b += 32 * kDeep) {
        StagedEntry e[kDeep];
#pragma unroll
        for (int d = 0; d < kDeep; ++d) {
          const int k = b + 32 * d + lane;
          e[d].t = -1;
          if (k < k1) e[d] = stage[k < n1 ? first + k : back + (k - n1)];
        }
#pragma unroll
        for (int d = 0; d < kDeep; ++d) {
          int h = static_cast<int>(BucketHash(e[d].t, mask));
          int key = e[d].t >= 0 ? T.key[h] : -1;
          while (key != -1 && key != e[d].t) {
            h = (h + 1) & mask;
            key = T.key[h];
          }
          const bool found = e[d].t >= 0 && key != -1;
          const unsigned m = __ballot_sync(kFull, found);
          if (found) {
            T.hit[queued + __popc(m & ((1u << lane) - 1u))] =
                make_int4(e[d].j, e[d].size, static_cast<int>(e[d].c), static_cast<int>(T.cnt[h]));
          }
          queued += __popc(m);
        }
        __syncwarp();
        for (; queued >= 32; queued -= 32) add(T.hit[queued - 32 + lane]);
        __syncwarp();
      }
      if (lane < queued) add(T.hit[lane]);
    } else {
      for (int k = static_cast<int>(static_cast<long long>(me.y) * part / parts) + lane;
           k < static_cast<int>(static_cast<long long>(me.y) * (part + 1) / parts); k += 32) {
        direct(stage[me.x + k]);
      }
      for (int j = i + 1; j < g; ++j) {
        const int4 other = place[j];
        if (other.y <= kTableRow) continue;
        const bool mine_long = me.y >= other.y;
        const StagedEntry* lr = stage + (mine_long ? me.x : other.x);
        const StagedEntry* sr = stage + (mine_long ? other.x : me.x);
        const int ll = mine_long ? me.y : other.y, ls = mine_long ? other.y : me.y;
        const int k0 = static_cast<int>(static_cast<long long>(ls) * part / parts);
        const int k1 = static_cast<int>(static_cast<long long>(ls) * (part + 1) / parts);
        if (k0 >= k1) continue;
        const long long sj = other.z;
        // the part of the long row that these ids span
        int edge = 0;
        if (lane < 2) edge = StagedLowerBound(lr, ll, sr[lane == 0 ? k0 : k1 - 1].t);
        const int lo0 = __shfl_sync(kFull, edge, 0);
        const int hi0 = min(__shfl_sync(kFull, edge, 1) + 1, ll);
        long long delta = 0, corr = 0;
        unsigned ovl = 0;
        bool any_bad = false;
        for (int b = k0; b < k1; b += 32 * kDeep) {
          StagedEntry e[kDeep];
          int at[kDeep], hi[kDeep];
#pragma unroll
          for (int d = 0; d < kDeep; ++d) {
            const int k = b + 32 * d + lane;
            e[d].t = -1;
            if (k < k1) e[d] = sr[k];
            at[d] = lo0;
            hi[d] = k < k1 ? hi0 : lo0;
          }
          // the lanes' searches side by side
          for (int span = hi0 - lo0; span > 0; span >>= 1) {
#pragma unroll
            for (int d = 0; d < kDeep; ++d) {
              if (at[d] < hi[d]) {
                const int mid = (at[d] + hi[d]) >> 1;
                if (lr[mid].t < e[d].t) at[d] = mid + 1; else hi[d] = mid;
              }
            }
          }
#pragma unroll
          for (int d = 0; d < kDeep; ++d) {
            if (e[d].t < 0 || at[d] >= ll || lr[at[d]].t != e[d].t) continue;
            const long long cl = lr[at[d]].c, cs = e[d].c;
            bool bad;
            const SharedTerm x = TermOf(si, sj, e[d].size, mine_long ? cl : cs, mine_long ? cs : cl, &bad);
            delta += x.delta;
            corr += x.corr;
            any_bad |= bad;
            ++ovl;
          }
        }
        ovl = __reduce_add_sync(kFull, ovl);
        if (ovl == 0) continue;
        delta = WarpSum(delta);
        corr = WarpSum(corr);
        const bool bad = __any_sync(kFull, any_bad);
        if (lane == 0) {
          examined += ovl;
          atomicAdd(&pmat[static_cast<long long>(i) * g + j], static_cast<unsigned long long>(delta) + ovl * kOvlOne);
          if (bad || corr != 0) {
            atomicAdd(&pmat[static_cast<long long>(j) * g + i], static_cast<unsigned long long>(bad ? kCorrBad : corr));
          }
        }
      }
    }
    examined = __reduce_add_sync(kFull, examined);
    if (lane == 0 && examined) atomicAdd(&P.gs[ri].examined, static_cast<unsigned long long>(examined));
  }
}

// Members of the big groups, a warp each: the member's top_k partners, and the
// gains of the pairs that no other member's warp has taken yet (the first to
// set a pair's flag scores it). Keys of the pairs that pass go to the group's
// list.
__global__ void __launch_bounds__(256, 2) WindowScoreKernel(WindowParams P) {
  FollowsOn();
  constexpr unsigned kFull = 0xffffffffu;
  __shared__ int cand_j[8][32];
  __shared__ unsigned short kept[8][kMaxGroup];
  __shared__ int nkept[8];
  const QuotientView& Q = P.Q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nb = P.ctl->nbig;
  const long long total = P.ctl->members;
  const long long nw = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  for (long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; w < total; w += nw) {
    const int bl = WarpLastLE(P.moff, 0, nb, w);
    const BigGroup G = P.list_big[bl];
    const int ri = G.ri, g = G.g;
    const int i = static_cast<int>(w - P.moff[bl]);
    const int* q = P.order + G.gstart;
    unsigned char* mat = P.mat + G.mat;
    const unsigned long long* pmat = reinterpret_cast<const unsigned long long*>(mat);
    unsigned* flags = reinterpret_cast<unsigned*>(mat + FlagOffset(static_cast<long long>(g) * g));
    if (lane == 0) nkept[warp] = 0;
    __syncwarp();
    const long long* old = reinterpret_cast<const long long*>(mat + OldCostOffset(static_cast<long long>(g) * g));
    auto proxy = [&](int x, int j) { return ProxyOf(PairWord(pmat, g, x, j)); };
    RankMember(g, i, q, old, P.top_k, cand_j[warp], proxy, [&](int a, int b) {
      const long long at = static_cast<long long>(a) * g + b;
      const unsigned bit = 1u << (8 * (at & 3));
      if (!(atomicOr(&flags[at >> 2], bit) & bit)) {
        kept[warp][atomicAdd(&nkept[warp], 1)] = static_cast<unsigned short>(a == i ? b : a);
      }
    });
    __syncwarp();
    const int n = nkept[warp];
    if (n == 0) continue;
    GroupStats* gs = P.gs + ri;
    unsigned long long* keys = P.keys + 2 * P.cand_off[ri];
    const int strict = WindowStrict(P, ri);
    long long uni = 0, ovl = 0, raw_a = 0, raw_b = 0, nnz = 0;
    for (int k0 = 0; k0 < n; k0 += 32) {
      const bool have = k0 + lane < n;
      bool sums = true;
      int a = 0, b = 0, qa = 0, qb = 0;
      GainParts gp = {0, 0, 0, 0, 0};
      RowSums A, B;
      if (have) {
        const int j = kept[warp][k0 + lane];
        a = i < j ? i : j;
        b = i < j ? j : i;
        qa = q[a];
        qb = q[b];
        A = P.rc[qa];
        B = P.rc[qb];
        const PairInfo pi = PairInfoOf(Q, qa, qb, pmat[static_cast<long long>(a) * g + b],
                                       static_cast<long long>(pmat[static_cast<long long>(b) * g + a]));
        sums = GainFromSums(A, B, pi, strict, &gp);
      }
      for (unsigned rest = __ballot_sync(kFull, !sums); rest; rest &= rest - 1) {
        const int src = __ffs(rest) - 1;
        const int xa = __shfl_sync(kFull, qa, src), xb = __shfl_sync(kFull, qb, src);
        const RowSums RA = P.rc[xa], RB = P.rc[xb];
        const long long s = static_cast<long long>(RA.size) + RB.size;
        long long part, fix = 0;
        if (!RowAfter(RA, s, &part)) fix += part - WarpRowAfter(Q, xa, s);
        if (!RowAfter(RB, s, &part)) fix += part - WarpRowAfter(Q, xb, s);
        if (lane == src) gp.gain += fix;
      }
      if (have) {
        uni += gp.uni;
        ovl += gp.ovl;
        raw_a += A.len;
        raw_b += B.len;
        nnz += A.len + (A.internal > 0 ? 1 : 0) + B.len + (B.internal > 0 ? 1 : 0);
        if (PassesFilter(gp.gain, gp.before, P.threshold, P.thr, P.use_threshold)) {
          if (gp.gain > kKeyGainMax) gp.err = kErrKeyRange;
          keys[atomicAdd(&gs->positive, 1ull)] = PackKey(gp.gain, a, b);
        }
        if (gp.err && atomicCAS(&gs->err, 0, gp.err) == 0) {
          gs->err_a = qa;
          gs->err_b = qb;
        }
      }
    }
    uni = WarpSum(uni);
    ovl = WarpSum(ovl);
    raw_a = WarpSum(raw_a);
    raw_b = WarpSum(raw_b);
    nnz = WarpSum(nnz);
    if (lane == 0) {
      atomicAdd(&gs->cand, static_cast<unsigned long long>(n));
      atomicAdd(&gs->uni, static_cast<unsigned long long>(uni));
      atomicAdd(&gs->ovl, static_cast<unsigned long long>(ovl));
      atomicAdd(&gs->raw_a, static_cast<unsigned long long>(raw_a));
      atomicAdd(&gs->raw_b, static_cast<unsigned long long>(raw_b));
      atomicAdd(&gs->nnz, static_cast<unsigned long long>(nnz));
    }
  }
}

// A big group by one CTA: matching rounds over its keys, and what the selected
// pairs touch.
__global__ void __launch_bounds__(kMatchThreads) WindowSelectKernel(WindowParams P) {
  FollowsOn();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* skeys = reinterpret_cast<unsigned long long*>(smem_raw);
  __shared__ MatchSmem<kMaxGroup> M;
  __shared__ unsigned long long s_gain, s_work;
  __shared__ int s_conflict;
  const QuotientView& Q = P.Q;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = P.ctl->nbig;
  for (int bl = blockIdx.x; bl < nb; bl += gridDim.x) {
    const BigGroup G = P.list_big[bl];
    const int ri = G.ri;
    GroupStats* gs = P.gs + ri;
    const int m = static_cast<int>(gs->positive);
    if (m == 0) {  // most groups
      if (tid == 0) {
        gs->rejected = gs->cand;
        P.sel_cnt[ri] = 0;
      }
      continue;
    }
    const int g = G.g;
    const int* q = P.order + G.gstart;
    unsigned long long* keys = P.keys + 2 * P.cand_off[ri];
    unsigned long long* spare = keys + (P.cand_off[ri + 1] - P.cand_off[ri]);
    __syncthreads();  // the last group's shared state is read
    if (2 * m <= kMatchSmemKeys) {
      for (int k = tid; k < m; k += kMatchThreads) skeys[k] = keys[k];
      keys = skeys;
      spare = skeys + m;
    }
    if (tid == 0) {
      s_gain = s_work = 0;
      s_conflict = 0x7fffffff;
    }
    __syncthreads();
    const int ns = MatchKeys<kMatchThreads>(M, keys, spare, m, g);
    // the selected pairs in greedy order, and what they touch: a warp per
    // pair, the whole CTA where a row is long
    const long long so = P.sel_off[ri];
    const int end = P.blk_end[ri];
    int conflict = 0x7fffffff;
    for (int i = warp; i < ns; i += kMatchThreads / 32) {
      const unsigned long long key = M.chosen[i];
      const int ka = q[(key >> kKeyIdxBits) & kKeyIdxMask], kb = q[key & kKeyIdxMask];
      const int la = Q.len[ka], lb = Q.len[kb];
      if (lane == 0) {
        const long long gain = kKeyGainMax - static_cast<long long>(key >> (2 * kKeyIdxBits));
        P.sel_keep[so + i] = ka;
        P.sel_rem[so + i] = kb;
        P.sel_gain[so + i] = gain;
        atomicAdd(&s_gain, static_cast<unsigned long long>(gain));
        atomicAdd(&s_work, static_cast<unsigned long long>(la + lb));
      }
      if (la <= kRowSmem) conflict = min(conflict, FirstTouched(P, Q.ent + Q.off[ka], la, end, lane, 32));
      if (lb <= kRowSmem) conflict = min(conflict, FirstTouched(P, Q.ent + Q.off[kb], lb, end, lane, 32));
    }
    for (int i = 0; i < 2 * ns; ++i) {
      const unsigned long long key = M.chosen[i >> 1];
      const int r = q[(i & 1 ? key : key >> kKeyIdxBits) & kKeyIdxMask];
      const int len = Q.len[r];
      if (len > kRowSmem) conflict = min(conflict, FirstTouched(P, Q.ent + Q.off[r], len, end, tid, kMatchThreads));
    }
    conflict = __reduce_min_sync(0xffffffffu, conflict);
    if (lane == 0) atomicMin(&s_conflict, conflict);
    __syncthreads();
    if (tid == 0) {
      gs->rejected = gs->cand - static_cast<unsigned long long>(m);
      gs->selected = ns;
      gs->gain = s_gain;
      gs->work = s_work;
      P.conflict[ri] = s_conflict;
      P.sel_cnt[ri] = ns;
    }
  }
}

// ------------------------------------------------------------ commit

// The batch: every CTA finds its end p, the first block that a selected pair
// of the window touches, and takes its share of the groups before it: their
// counters, and their pairs onto the commit list. Errors of an evaluation
// count here too, when its block's turn has come.
__global__ void __launch_bounds__(kMarkThreads) WindowMarkKernel(WindowParams P) {
  FollowsOn();
  __shared__ int s_min;
  __shared__ unsigned long long acc[kGroupStatWords + 3];  // + groups, member pairs, largest group
  const int tid = threadIdx.x, lane = tid & 31;
  const int f = P.ctl->f, e = P.ctl->e;
  if (f >= e) {
    if (blockIdx.x == 0 && tid == 0) P.ctl->p = f;
    return;
  }
  if (tid == 0) s_min = min(e, P.ctl->stale);
  if (tid < kGroupStatWords + 3) acc[tid] = 0;
  __syncthreads();
  int first = e;
#pragma unroll 4
  for (int ri = f + tid; ri < e; ri += kMarkThreads) first = min(first, P.conflict[ri]);
  first = __reduce_min_sync(0xffffffffu, first);
  if (lane == 0) atomicMin(&s_min, first);
  __syncthreads();
  const int p = s_min < e ? P.blk_beg[s_min] : e;
  if (blockIdx.x == 0 && tid == 0) P.ctl->p = p;
  // commit list, a thread per group
  unsigned long long raw = 0;
  int groups = 0, largest = 0;
  for (int ri = f + blockIdx.x * kMarkThreads + tid; ri < p; ri += gridDim.x * kMarkThreads) {
    const int g = P.glen[P.real[ri]];
    const GroupStats* z = P.gs + ri;
    if (z->err) RaiseError(P.err, z->err, z->err_a, z->err_b, 0);
    const long long so = P.sel_off[ri];
    const int ns = P.sel_cnt[ri];
    if (ns > 0) {
      const unsigned at = atomicAdd(&P.bctl->sel_total, static_cast<unsigned>(ns));
      for (int i = 0; i < ns; ++i) {
        const int keep = P.sel_keep[so + i], rem = P.sel_rem[so + i];
        P.stamp[keep] = 2 * P.block_stamp;
        P.stamp[rem] = 2 * P.block_stamp + 1;
        P.partner[keep] = rem;
        P.partner[rem] = keep;
        P.seq[rem] = static_cast<int>(so + i);
        P.sel_list[at + i] = static_cast<int>(so + i);
      }
    }
    ++groups;
    raw += static_cast<unsigned long long>(g) * (g - 1) / 2;
    largest = g > largest ? g : largest;
  }
  groups = WarpSumInt(groups);
  raw = static_cast<unsigned long long>(WarpSum(static_cast<long long>(raw)));
  largest = __reduce_max_sync(0xffffffffu, largest);
  if (lane == 0 && groups) {
    atomicAdd(&acc[kGroupStatWords], static_cast<unsigned long long>(groups));
    atomicAdd(&acc[kGroupStatWords + 1], raw);
    atomicMax(&acc[kGroupStatWords + 2], static_cast<unsigned long long>(largest));
  }
  // counters, a warp per group, a lane per counter
  unsigned long long sum = 0;
  const int nwarps = gridDim.x * (kMarkThreads / 32);
  if (lane < kGroupStatWords) {
#pragma unroll 4
    for (int ri = f + ((blockIdx.x * kMarkThreads + tid) >> 5); ri < p; ri += nwarps) {
      sum += reinterpret_cast<const unsigned long long*>(P.gs + ri)[lane];
    }
    if (sum) atomicAdd(&acc[lane], sum);
  }
  __syncthreads();
  if (tid < kGroupStatWords + 3) {
    // the counters that each word feeds (GroupStats in order)
    auto add = [&](int k, unsigned long long v) {
      if (v) atomicAdd(&P.stats[k], v);
    };
    const unsigned long long v = acc[tid];
    switch (tid) {
      case 0: add(kStProxyExamined, v); break;
      case 1:
        add(kStCandAfterPrune, v);
        add(kStExactCalls, v);
        add(kStScoreBytes, v * (2 * sizeof(RowSums) + sizeof(PairInfo) + 24));
        break;
      case 2: add(kStUnion, v); break;
      case 3: add(kStOverlap, v); break;
      case 4: add(kStRawA, v); break;
      case 5: add(kStRawB, v); break;
      case 6: add(kStInputNnz, v); break;
      case 7: add(kStRejThreshold, v); break;
      case 8:
        add(kStPositive, v);
        add(kStCandPairs, v);
        add(kStRejOverlap, v - acc[9]);
        break;
      case 9:
        add(kStSelected, v);
        add(kStValidationCalls, v);
        break;
      case 10:
        add(kStLocalGain, v);
        add(kStIsolatedGain, v);
        break;
      case 11: add(kStValidationWork, v); break;
      case 12: add(kStPrepareBytes, 12ull * v); break;
      case kGroupStatWords: add(kStGroupCount, v); break;
      case kGroupStatWords + 1: add(kStRawPairCount, v); break;
      default: atomicMax(&P.stats[kStGroupMaxSize], v); break;
    }
  }
}
