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
// One round is eight launches that take their work from device memory, for as
// many blocks as turned out independent (a block at a time took a dozen
// launches, 75 to 120 us, latency only). Rounds follow each other without the
// host, which watches the frontier through mapped memory and keeps a few
// rounds queued. Measured with 64-group blocks, 20 iterations, a block at a time
// -> windows: R-MAT 16 (edge factor 8) 621 -> 132 ms, R-MAT 12 36.7 -> 18.4 ms,
// Chung-Lu of 20,000 nodes with twins 109 -> 69 ms.
#pragma once

// Blocks of at most this many groups go through windows; larger ones fill the
// GPU by themselves and touch too much of each other.
constexpr int kWindowMaxBatch = 256;
constexpr int kWindowMaxGroups = 8192;  // groups a window takes in at most (then to the block's end)
constexpr int kWindowMinGroups = 256;
constexpr int kWindowList = 2 * (kWindowMaxGroups + kWindowMaxBatch) + 1024;
constexpr int kEvalWarps = 4;
constexpr int kEvalPairs = 16;   // member pairs per work item of a big group, at most
constexpr int kEvalCtas = 8;     // per SM
constexpr int kEvalGrid = 152 * kEvalCtas;
constexpr int kBigGrid = 152 * 2;
constexpr int kMarkGrid = 16;
constexpr int kMarkThreads = 256;
// Rows and pairs of rows longer than this are handed on in units, so that no
// warp holds up a round with a hub's row.
constexpr int kLongRow = 1024;       // entries of a row (sums), of two rows to merge
constexpr int kLongProbe = 96;       // entries to look up in a far longer row
constexpr int kLongRowUnit = 1024;   // entries of a row per unit
constexpr int kLongPairUnit = 128;   // entries of the shorter row per unit
constexpr int kLongUnits = 1 << 19;  // units at most; what does not fit is done in place
constexpr int kLongThreads = 256;
constexpr int kLongGrid = 152 * 6;
// Groups of at most top_k + 1 members need no ranking; a warp handles one with
// up to this many.
constexpr int kEvalSmall = 17;
constexpr int kEvalSmallPairs = kEvalSmall * (kEvalSmall - 1) / 2;
constexpr int kWindowAhead = 2;  // rounds queued by the host and not seen done
// Skewed pairs (the long row at least kProbeMinLong entries and kProbeRatio
// times the short one) look the short row up in the long one.
constexpr int kProbeMinLong = 256;
constexpr int kProbeRatio = 8;

struct WindowCtl {
  int f, e, R;     // first group not committed; end of the evaluated groups; groups of the iteration
  int p;           // end of the batch being committed
  int take;        // groups to keep evaluated ahead
  int nsmall, nbig, ndirty;
  long long members, pairs;  // of the listed big groups
  unsigned long long work;   // queue of the evaluation kernel
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
};
constexpr int kGroupStatWords = 13;

// Part of a long row (b < 0: its sums, `up` the approximate old cost) or of a
// pair with a long row (the pair's two words).
struct LongUnit {
  unsigned long long* up;
  unsigned long long* down;
  int a, b;  // supernodes
  int at;    // first entry (of the shorter row)
  int ri;    // group, -1: nothing to do
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
  WindowCtl* ctl;
  GroupStats* gs;
  int* conflict;        // per group position: first later group its pairs touch (INT_MAX: none)
  LongUnit* units;
  int* dirty;           // per group position: stamp of the last commit that touched it
  int* list_dirty;
  int* list_small;
  int* list_big;
  long long* moff;      // member / pair prefixes over list_big
  long long* poff;
  const long long* mat_off;
  unsigned char* mat;
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
  unsigned long long* stats;
  DevError* err;
  volatile int* host_f;  // mapped: the frontier, and the lists made so far
};

__device__ __forceinline__ bool WindowSmall(int g, unsigned entries) {
  return g <= kEvalSmall && entries <= static_cast<unsigned>(kSmallStage);
}

// ------------------------------------------------------------ lists

// Per active supernode its group position, per group position the end of its
// block and a clean mark, and the number of blocks.
__global__ void WindowSetupKernel(const int* order, const int* group_of, const int* ri_of, int count, const int* real,
                                  int R, int batch, int* node_ri, int* blk_end, int* dirty, WindowCtl* ctl) {
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
    dirty[i] = 0;
    if (i == 0 || real[i - 1] / batch != b) atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->blocks), 1ull);
  }
}

// The next evaluation's lists, by one CTA of kHugeThreads: the touched groups
// and those that the window takes in. `done`: groups [f, p) are committed.
struct ListSum {
  long long members, pairs;
  int small, big;
};
struct ListSumOp {
  __device__ __forceinline__ ListSum operator()(const ListSum& a, const ListSum& b) const {
    return ListSum{a.members + b.members, a.pairs + b.pairs, a.small + b.small, a.big + b.big};
  }
};

__device__ __noinline__ void BuildLists(const WindowParams& P) {
  using Scan = cub::BlockScan<ListSum, kHugeThreads, cub::BLOCK_SCAN_WARP_SCANS>;
  __shared__ typename Scan::TempStorage tmp;
  __shared__ ListSum carry;
  __shared__ int s_e0, s_e1, s_dirty;
  WindowCtl* c = P.ctl;
  if (threadIdx.x == 0) {
    const int committed = c->p - c->f;
    // twice what the last rounds committed is kept evaluated: evaluations
    // further ahead are likely to be touched before their turn
    int take = c->p == c->e ? 2 * c->take : 2 * committed;
    if (c->R == 0 || c->p == 0) take = c->take;  // the iteration's first lists
    take = take < kWindowMinGroups ? kWindowMinGroups : take > kWindowMaxGroups ? kWindowMaxGroups : take;
    c->take = take;
    c->f = c->p;
    int e = c->f + take;
    e = e >= c->R ? c->R : e == 0 ? 0 : P.blk_end[e - 1];
    s_e0 = c->e;
    s_e1 = e > c->e ? e : c->e;
    s_dirty = c->ndirty;
    carry = ListSum{0, 0, 0, 0};
  }
  __syncthreads();
  const int n = s_dirty + (s_e1 - s_e0);
  for (int base = 0; base < n; base += kHugeThreads) {
    const int i = base + threadIdx.x;
    int ri = -1, g = 0;
    ListSum v{0, 0, 0, 0};
    if (i < n) {
      ri = i < s_dirty ? P.list_dirty[i] : s_e0 + (i - s_dirty);
      const int gid = P.real[ri];
      g = P.glen[gid];
      if (WindowSmall(g, P.gent[gid])) {
        v.small = 1;
      } else {
        v.big = 1;
        v.members = g;
        v.pairs = static_cast<long long>(g) * (g - 1) / 2;
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
      P.list_big[c0.big + ex.big] = ri;
      P.moff[c0.big + ex.big] = c0.members + ex.members;
      P.poff[c0.big + ex.big] = c0.pairs + ex.pairs;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry = ListSumOp()(c0, total);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    P.moff[carry.big] = carry.members;
    P.poff[carry.big] = carry.pairs;
    c->nsmall = carry.small;
    c->nbig = carry.big;
    c->members = carry.members;
    c->pairs = carry.pairs;
    c->ndirty = 0;
    c->work = 0;
    c->units = 0;
    c->e = s_e1;
    P.host_f[0] = c->f;
    __threadfence_system();
    P.host_f[1] = ++c->rounds;
  }
}

__global__ void __launch_bounds__(kHugeThreads) WindowBeginKernel(WindowParams P, int R) {
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
      if (!GainFromSums(A, B, pi, 1, &gp)) {
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

// Entries [k0, k1) of a row, by a warp (sums of the whole warp on return).
__device__ __forceinline__ void SumEntries(const QuotientView& Q, const Entry* row, int k0, int k1, int rep,
                                           long long si, RowPart* out) {
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int k = k0 + lane; k < k1; k += 32) {
    const Entry e = row[k];
    const long long c = EntCnt(e);
    const long long st = Q.size[EntNb(e)];
    out->old += EncodeCostForPair(rep, si, EntNb(e), st, c);
    if (HeavyEntry(si, st, c)) out->heavy.Add(st, c); else out->light += c;
  }
  out->old = WarpSum(out->old);
  out->light = WarpSum(out->light);
  out->heavy.WarpReduce();
}

// Member i of a big group by one warp: its row sums and approximate old cost.
__device__ void EvalMember(const WindowParams& P, int ri, int i) {
  const int lane = threadIdx.x & 31;
  const QuotientView& Q = P.Q;
  const int gid = P.real[ri];
  const long long g = P.glen[gid];
  const int rep = P.order[P.gstart[gid] + i];
  const long long si = Q.size[rep];
  const int len = Q.len[rep];
  const long long internal = Q.internal[rep];
  const long long own = internal > 0 ? EncodeCostForPair(rep, si, rep, si, 2 * internal) : 0;
  long long* old_out = reinterpret_cast<long long*>(P.mat + P.mat_off[ri] + OldCostOffset(g * g)) + i;
  if (lane == 0) atomicAdd(&P.gs[ri].entries, static_cast<unsigned long long>(len));
  RowPart r;
  if (len > kLongRow) {
    LongUnit u{reinterpret_cast<unsigned long long*>(old_out), nullptr, rep, -1, 0, ri};
    if (PushUnits(P, u, len, kLongRowUnit)) {
      // the units add their entries
      if (lane == 0) {
        StoreRowSums(&P.rc[rep], 0, 0, HeavyAcc(), internal, static_cast<int>(si), len);
        *old_out = own;
      }
      return;
    }
  }
  SumEntries(Q, Q.ent + Q.off[rep], 0, len, rep, si, &r);
  if (lane == 0) {
    StoreRowSums(&P.rc[rep], r.old, r.light, r.heavy, internal, static_cast<int>(si), len);
    *old_out = r.old + own;
  }
}

// Members a < b of a big group by one warp: the pair's words, from a merge of
// the two rows (32 entries of each per step, every entry up to the smaller of
// the two tiles' last neighbours final in its step) or, where one row is far
// longer, a search of the short one's entries in it. Returns the shared
// targets found here.
struct PairRows {
  int ra, rb, sa, sb, la, lb;
  long long offa, offb;
};

__device__ int EvalPair(const WindowParams& P, int ri, const PairRows& R, unsigned long long* up,
                        unsigned long long* down) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr Entry kPadEntry = static_cast<Entry>(0x7fffffffull) << 32;
  const int lane = threadIdx.x & 31;
  const QuotientView& Q = P.Q;
  const int ra = R.ra, rb = R.rb;
  const long long sa = R.sa, sb = R.sb;
  const Entry* pa_row = Q.ent + R.offa;
  const Entry* pb_row = Q.ent + R.offb;
  const int la = R.la, lb = R.lb;
  long long delta = 0, corr = 0;
  unsigned ea = 0, eb = 0;
  int ovl = 0;
  bool any_bad = false;
  auto shared = [&](int x, long long ca, long long cb) {
    bool bad;
    const SharedTerm t = TermOf(sa, sb, Q.size[x], ca, cb, &bad);
    delta += t.delta;
    corr += t.corr;
    any_bad |= bad;
    ++ovl;
  };
  const bool a_long = la >= lb;
  const int ll = a_long ? la : lb, ls = a_long ? lb : la;
  const bool probe = ll >= kProbeMinLong && ll >= kProbeRatio * ls;
  if (probe ? ls > kLongProbe : la + lb > kLongRow) {
    if (PushUnits(P, LongUnit{up, down, ra, rb, 0, ri}, ls, kLongPairUnit)) {
      // the units add what they find
      if (lane == 0) {
        *up = 0;
        *down = 0;
      }
      return 0;
    }
  }
  if (probe) {
    const Entry* lr = a_long ? pa_row : pb_row;
    const Entry* sr = a_long ? pb_row : pa_row;
    const int long_rep = a_long ? ra : rb, short_rep = a_long ? rb : ra;
    unsigned e_long = 0, e_short = 0;
    for (int k = lane; k < ls + 1; k += 32) {
      // the lane past the short row looks for it in the long one
      const Entry e = k < ls ? sr[k] : MakeEnt(short_rep, 0);
      const int x = EntNb(e);
      if (x == long_rep) {
        e_short = static_cast<unsigned>(EntCnt(e));
        continue;
      }
      const int at = RowLowerBound(lr, ll, x);
      if (at < ll && EntNb(lr[at]) == x) {
        const long long cl = EntCnt(lr[at]);
        if (k == ls) {
          e_long = static_cast<unsigned>(cl);
        } else {
          shared(x, a_long ? cl : EntCnt(e), a_long ? EntCnt(e) : cl);
        }
      }
    }
    ea = a_long ? e_long : e_short;
    eb = a_long ? e_short : e_long;
  } else {
    int pa = 0, pb = 0;
    while (pa < la || pb < lb) {
      const bool va = pa + lane < la, vb = pb + lane < lb;
      const Entry xe = va ? pa_row[pa + lane] : kPadEntry;
      const Entry ye = vb ? pb_row[pb + lane] : kPadEntry;
      const int xa = EntNb(xe), xb = EntNb(ye);
      const int last_a = __shfl_sync(kFull, xa, 31);
      const int last_b = __shfl_sync(kFull, xb, 31);
      const int lim = last_a < last_b ? last_a : last_b;
      int pos = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const int probe = __shfl_sync(kFull, xb, pos + step - 1);
        if (probe < xa) pos += step;
      }
      const Entry ce = __shfl_sync(kFull, ye, pos);
      const bool fin_a = va && xa <= lim, fin_b = vb && xb <= lim;
      if (fin_a) {
        if (xa == rb) {
          ea = static_cast<unsigned>(EntCnt(xe));
        } else if (EntNb(ce) == xa) {
          shared(xa, EntCnt(xe), EntCnt(ce));
        }
      }
      if (fin_b && xb == ra) eb = static_cast<unsigned>(EntCnt(ye));
      pa += __popc(__ballot_sync(kFull, fin_a));
      pb += __popc(__ballot_sync(kFull, fin_b));
    }
  }
  ovl = WarpSumInt(ovl);
  ea = __reduce_max_sync(kFull, ea);
  eb = __reduce_max_sync(kFull, eb);
  const bool bad = __any_sync(kFull, any_bad);
  unsigned long long word = 0, low = 0;
  if (ovl > 0) {  // most pairs of a group share nothing
    delta = WarpSum(delta);
    corr = WarpSum(corr);
    word = static_cast<unsigned long long>(delta) + static_cast<unsigned long long>(ovl) * kOvlOne;
    low = static_cast<unsigned long long>(bad ? kCorrBad : corr);
  }
  if (ea) word += ea | kRowILists;
  if (eb) word |= kRowJLists;
  if (lane == 0) {
    *up = word;
    *down = low;
  }
  return ovl;
}

// Work items in one queue: the members and pairs of the big groups (the longer
// ones), then the small groups. One warp each.
__global__ void __launch_bounds__(kEvalWarps * 32, kEvalCtas) WindowEvalKernel(WindowParams P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  EvalWarpSmem& W = reinterpret_cast<EvalSmem*>(smem_raw)->w[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const long long nm = P.ctl->members;
  // pairs per item: as few as keep every warp busy
  const long long warps = static_cast<long long>(gridDim.x) * kEvalWarps;
  long long per = P.ctl->pairs / (2 * warps) + 1;
  per = per < kEvalPairs ? per : kEvalPairs;
  const long long np = (P.ctl->pairs + per - 1) / per;
  const int ns = P.ctl->nsmall, nb = P.ctl->nbig;
  for (;;) {
    long long it = 0;
    if (lane == 0) it = static_cast<long long>(atomicAdd(&P.ctl->work, 1ull));
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it < nm) {
      const int bl = WarpLastLE(P.moff, 0, nb, it);
      EvalMember(P, P.list_big[bl], static_cast<int>(it - P.moff[bl]));
    } else if (it < nm + np) {
      const long long p0 = (it - nm) * per;
      const long long p1 = p0 + per < P.ctl->pairs ? p0 + per : P.ctl->pairs;
      // lane d holds pair p0 + d: its group, its place and its rows' scalars,
      // one chain of loads for all of them
      const int bl0 = WarpLastLE(P.poff, 0, nb, p0);
      int ri = 0, g = 0, a = 0, b = 0;
      PairRows R = {0, 0, 0, 0, 0, 0, 0, 0};
      unsigned long long* pmat = nullptr;
      if (p0 + lane < p1) {
        int bl = bl0;
        while (P.poff[bl + 1] <= p0 + lane) ++bl;
        ri = P.list_big[bl];
        const int gid = P.real[ri];
        g = P.glen[gid];
        const int* q = P.order + P.gstart[gid];
        pmat = reinterpret_cast<unsigned long long*>(P.mat + P.mat_off[ri]);
        TriPair(static_cast<int>(p0 + lane - P.poff[bl]), g, &a, &b);
        R.ra = q[a];
        R.rb = q[b];
        R.sa = P.Q.size[R.ra];
        R.sb = P.Q.size[R.rb];
        R.la = P.Q.len[R.ra];
        R.lb = P.Q.len[R.rb];
        R.offa = P.Q.off[R.ra];
        R.offb = P.Q.off[R.rb];
        unsigned char* fmat = reinterpret_cast<unsigned char*>(pmat) + FlagOffset(static_cast<long long>(g) * g);
        fmat[static_cast<long long>(a) * g + b] = 0;
      }
      unsigned long long* up = pmat + static_cast<long long>(a) * g + b;
      unsigned long long* down = pmat + static_cast<long long>(b) * g + a;
      int examined = 0;
      for (int d = 0; d < static_cast<int>(p1 - p0); ++d) {
        constexpr unsigned kFull = 0xffffffffu;
        PairRows X;
        X.ra = __shfl_sync(kFull, R.ra, d);
        X.rb = __shfl_sync(kFull, R.rb, d);
        X.sa = __shfl_sync(kFull, R.sa, d);
        X.sb = __shfl_sync(kFull, R.sb, d);
        X.la = __shfl_sync(kFull, R.la, d);
        X.lb = __shfl_sync(kFull, R.lb, d);
        X.offa = __shfl_sync(kFull, R.offa, d);
        X.offb = __shfl_sync(kFull, R.offb, d);
        unsigned long long* xu =
            reinterpret_cast<unsigned long long*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(up), d));
        unsigned long long* xd =
            reinterpret_cast<unsigned long long*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(down), d));
        const int n = EvalPair(P, __shfl_sync(kFull, ri, d), X, xu, xd);
        if (lane == d) examined = n;
      }
      if (examined) atomicAdd(&P.gs[ri].examined, static_cast<unsigned long long>(examined));
    } else if (it < nm + np + ns) {
      EvalSmallGroup(P, W, P.list_small[it - nm - np]);
    } else {
      break;
    }
  }
}

// The long units, a warp each: row sums and pair words, added up.
__global__ void __launch_bounds__(kLongThreads) WindowLongKernel(WindowParams P) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kPer = kLongPairUnit / 32;
  const QuotientView& Q = P.Q;
  const int lane = threadIdx.x & 31;
  const unsigned total = P.ctl->units < kLongUnits ? P.ctl->units : kLongUnits;
  const unsigned nw = (gridDim.x * blockDim.x) >> 5;
  for (unsigned t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total; t += nw) {
    const LongUnit u = P.units[t];
    if (u.ri < 0) continue;
    if (u.b < 0) {
      const int len = Q.len[u.a];
      RowPart r;
      SumEntries(Q, Q.ent + Q.off[u.a], u.at, min(u.at + kLongRowUnit, len), u.a, Q.size[u.a], &r);
      if (lane == 0) {
        RowSums* s = &P.rc[u.a];
        atomicAdd(u.up, static_cast<unsigned long long>(r.old));
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
      continue;
    }
    const long long sa = Q.size[u.a], sb = Q.size[u.b];
    const int la = Q.len[u.a], lb = Q.len[u.b];
    const bool a_long = la >= lb;
    const int ll = a_long ? la : lb, ls = a_long ? lb : la;
    const Entry* lr = Q.ent + Q.off[a_long ? u.a : u.b];
    const Entry* sr = Q.ent + Q.off[a_long ? u.b : u.a];
    const int long_rep = a_long ? u.a : u.b, short_rep = a_long ? u.b : u.a;
    const int end = min(u.at + kLongPairUnit, ls);
    // the part of the long row that the unit's ids span
    int edge = 0;
    if (lane < 2) edge = RowLowerBound(lr, ll, EntNb(sr[lane == 0 ? u.at : end - 1]));
    const int lo0 = __shfl_sync(kFull, edge, 0);
    const int hi0 = min(__shfl_sync(kFull, edge, 1) + 1, ll);
    Entry e[kPer];
    int at[kPer], hi[kPer];
#pragma unroll
    for (int d = 0; d < kPer; ++d) {
      const int k = u.at + 32 * d + lane;
      e[d] = k < end ? sr[k] : 0;
      at[d] = lo0;
      hi[d] = k < end ? hi0 : lo0;
    }
    // the lanes' searches side by side
    for (int span = hi0 - lo0; span > 0; span >>= 1) {
#pragma unroll
      for (int d = 0; d < kPer; ++d) {
        if (at[d] < hi[d]) {
          const int mid = (at[d] + hi[d]) >> 1;
          if (EntNb(lr[mid]) < EntNb(e[d])) at[d] = mid + 1; else hi[d] = mid;
        }
      }
    }
    long long delta = 0, corr = 0;
    int ovl = 0;
    bool any_bad = false;
    unsigned e_short = 0, e_long = 0;
#pragma unroll
    for (int d = 0; d < kPer; ++d) {
      const int k = u.at + 32 * d + lane;
      if (k >= end) continue;
      const int x = EntNb(e[d]);
      if (x == long_rep) {
        e_short = static_cast<unsigned>(EntCnt(e[d]));
      } else if (at[d] < ll && EntNb(lr[at[d]]) == x) {
        const long long cl = EntCnt(lr[at[d]]), cs = EntCnt(e[d]);
        bool bad;
        const SharedTerm term = TermOf(sa, sb, Q.size[x], a_long ? cl : cs, a_long ? cs : cl, &bad);
        delta += term.delta;
        corr += term.corr;
        any_bad |= bad;
        ++ovl;
      }
    }
    if (u.at == 0 && lane == 0) e_long = static_cast<unsigned>(RowLookup(lr, ll, short_rep));
    ovl = WarpSumInt(ovl);
    e_short = __reduce_max_sync(kFull, e_short);
    e_long = __reduce_max_sync(kFull, e_long);
    const bool bad = __any_sync(kFull, any_bad);
    unsigned long long word = 0;
    if (ovl > 0) {
      delta = WarpSum(delta);
      corr = WarpSum(corr);
      word = static_cast<unsigned long long>(delta) + static_cast<unsigned long long>(ovl) * kOvlOne;
    }
    const unsigned ea = a_long ? e_long : e_short, eb = a_long ? e_short : e_long;
    if (ea) word += ea | kRowILists;
    if (eb) word |= kRowJLists;
    if (lane == 0) {
      if (word) atomicAdd(u.up, word);
      if (ovl > 0 && (bad || corr != 0)) atomicAdd(u.down, static_cast<unsigned long long>(bad ? kCorrBad : corr));
      if (ovl > 0) atomicAdd(&P.gs[u.ri].examined, static_cast<unsigned long long>(ovl));
    }
  }
}

// Members of the big groups, a warp each: the member's top_k partners, and the
// gains of the pairs that no other member's warp has taken yet (the first to
// set a pair's flag scores it). Keys of the pairs that pass go to the group's
// list.
__global__ void __launch_bounds__(256, 2) WindowScoreKernel(WindowParams P) {
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
    const int ri = P.list_big[bl];
    const int gid = P.real[ri];
    const int g = P.glen[gid];
    const int i = static_cast<int>(w - P.moff[bl]);
    const int* q = P.order + P.gstart[gid];
    unsigned char* mat = P.mat + P.mat_off[ri];
    const unsigned long long* pmat = reinterpret_cast<const unsigned long long*>(mat);
    unsigned* flags = reinterpret_cast<unsigned*>(mat + FlagOffset(static_cast<long long>(g) * g));
    if (lane == 0) nkept[warp] = 0;
    __syncwarp();
    RankMember(g, i, q, mat, P.top_k, cand_j[warp], [&](int a, int b) {
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
        sums = GainFromSums(A, B, pi, 1, &gp);
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
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned long long* skeys = reinterpret_cast<unsigned long long*>(smem_raw);
  __shared__ MatchSmem M;
  __shared__ unsigned long long s_gain, s_work;
  __shared__ int s_conflict;
  const QuotientView& Q = P.Q;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nb = P.ctl->nbig;
  for (int bl = blockIdx.x; bl < nb; bl += gridDim.x) {
    const int ri = P.list_big[bl];
    GroupStats* gs = P.gs + ri;
    const int m = static_cast<int>(gs->positive);
    if (m == 0) {  // most groups
      if (tid == 0) {
        gs->rejected = gs->cand;
        P.sel_cnt[ri] = 0;
      }
      continue;
    }
    const int gid = P.real[ri];
    const int g = P.glen[gid];
    const int* q = P.order + P.gstart[gid];
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
    const int ns = MatchKeys(M, keys, spare, m, g);
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
  __shared__ int s_min;
  __shared__ unsigned long long acc[kGroupStatWords + 3];  // + groups, member pairs, largest group
  const int tid = threadIdx.x, lane = tid & 31;
  const int f = P.ctl->f, e = P.ctl->e;
  if (f >= e) {
    if (blockIdx.x == 0 && tid == 0) P.ctl->p = f;
    return;
  }
  if (tid == 0) s_min = e;
  if (tid < kGroupStatWords + 3) acc[tid] = 0;
  __syncthreads();
  int first = e;
#pragma unroll 4
  for (int ri = f + tid; ri < e; ri += kMarkThreads) first = min(first, P.conflict[ri]);
  first = __reduce_min_sync(0xffffffffu, first);
  if (lane == 0) atomicMin(&s_min, first);
  __syncthreads();
  int p = s_min;
  if (p < e) {
    // the start of its block: the first position whose block ends after it
    int lo = f, hi = p;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (P.blk_end[mid] <= p) lo = mid + 1; else hi = mid;
    }
    p = lo;
  }
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
