// A group of medium size by one CTA, from its rows to its selected pairs:
// candidates (src/sweg.cpp:1598-1727, 1800-1999), exact gains
// (src/quotient_graph.cpp:340-462), threshold and g0 selection
// (src/sweg.cpp:2146-2281) without a word of it in global memory in between.
// Included by merge.cu only.
//
// Groups of more than a warp's share but with at most kMedGroup members and
// kMedStage row entries took five launches over tables in global memory
// (prepare, member ranking, output, scoring, selection), each a CTA or a warp
// per member that waits for loads most of the time. Here the group's entries,
// pair sums and keys stay in 68 KB of shared memory, three CTAs to an SM.
// Pairs that share a target are found by hashing the entries' targets into
// runs; every entry visits the earlier ones of its run, so the work is the
// number of shared targets, not of member pairs times row length.
#pragma once


constexpr int kMedGroup = 64;
constexpr int kMedStage = 2048;
constexpr int kMedThreads = 256;
constexpr int kMedPairs = kMedGroup * (kMedGroup - 1) / 2;
constexpr int kMedSlots = 2 * kMedStage;
constexpr int kMedCtas = 3;  // per SM
// Blocks with fewer medium groups than this keep the five launches: a CTA's
// chain through one group (20 us, 100 at most) is longer than theirs, and pays
// when there is a wave or more of groups. (R-MAT 19, some 900 medium groups an
// iteration, is even; Chung-Lu 1M, 14,000 to 25,000, 138 -> 116 ms a run; the
// 16,384-group blocks of the grid + Chung-Lu union, a handful, 335 -> 354 ms.)
constexpr int kMedMinGroups = 2 * 152;
// An iteration planned on the device goes by its groups of all sizes instead,
// which the host knows before the plan; the medium ones among them would tell
// better. 20 iterations without the kernel -> with it, groups of iteration 1 and
// medium groups an iteration: Chung-Lu (degree 17) 3,493 / 370 15.8 -> 16.0 ms,
// 10,409 / 1,090 22.2 -> 21.4, 35,682 / 3,560 38.9 -> 34.9, 92,925 / 8,830 73.1
// -> 61.0; R-MAT 15 and 17 (edge factor 8) 19,549 / 170 17.0 -> 17.8 and 82,247 /
// 620 27.1 -> 27.6; R-MAT 18 and 19 (edge factor 2) 205,762 / 450 21.65 -> 21.97
// and 418,211 / 890 27.8 -> 27.5; the union of 0.26 M nodes in blocks of 16,384
// groups, 190 medium an iteration, 51.8 -> 55.5.
constexpr long long kMedMinAll = 1 << 16;

__host__ __device__ __forceinline__ bool MediumFits(int g, unsigned entries) {
  return g <= kMedGroup && entries <= static_cast<unsigned>(kMedStage);
}

// Pair sums, upper triangle by TriIndex(a, b): proxy << 32 | corr, and the
// number of shared targets, two to a word (16 bits each).
struct MediumPairsSmem {
  unsigned long long pc[kMedPairs];
  unsigned ovl[(kMedPairs + 1) / 2];
};
static_assert(2 * (sizeof(MediumPairsSmem::ovl) / sizeof(unsigned)) >= kMedPairs, "a half word per pair");
static_assert(kMedStage / 2 < 1 << 16, "two rows share at most half of the staged entries");

struct MediumSmem {
  // the members' rows (the names the staged-row helpers use)
  Entry ent[kMedStage];  // afterwards: the selection keys
  long long old[kMedGroup];
  long long off[kMedGroup];
  HeavyAcc heavy[kMedGroup];
  RowSums rs[kMedGroup];
  int tsz[kMedStage];
  unsigned light[kMedGroup];
  int q[kMedGroup];
  int sz[kMedGroup];
  int start[kMedGroup + 1];
  unsigned short order[kMedStage];  // entries by target
  unsigned char row[kMedStage];     // member of the entry; bit 7: its target is a member
  unsigned char rank[kMedStage];    // place in the target's run, by position in order
  union {
    struct {
      int key[kMedSlots];
      unsigned cnt[kMedSlots / 2];  // two to a word: entries of the slot, then its run's start
    } hash;
    MediumPairsSmem pairs;
  } u;
  unsigned keep[kMedGroup][2];  // kept partners b > a of member a
  int cj[kMedThreads / 32][32];
  int rows_end[2];  // entries of the first and the last 32 members
  MatchSmem<kMedGroup> match;
  unsigned long long acc[10];
  int nkeys, err[3], bad;
};
static_assert(kMedCtas * (sizeof(MediumSmem) + kSmemReserved) <= kSmemPerSm, "kMedCtas of them fit an SM");

struct MediumParams {
  QuotientView Q;
  const int* order;
  const int* gstart;
  const int* glen;
  const int* group_of;
  const int* idx_in_group;
  const int* real;
  const int* list;  // group positions
  int list0;
  int top_k;
  double threshold;
  ThresholdBits thr;
  int use_threshold;
  int strict;
  const long long* sel_off;
  int* sel_keep;
  int* sel_rem;
  long long* sel_gain;
  int* sel_cnt;
  int* stamp;
  int* partner;
  int* seq;
  int* sel_list;
  BlockCtl* ctl;
  int block_stamp;
  unsigned long long* stats;
  DevError* err;
};

// Member i's top_k partners by one warp, two candidates to a lane. cj: 32 words
// of the warp's own.
template <typename ProxyFn, typename KeepFn>
__device__ __forceinline__ void MediumTopK(const MediumSmem& S, int g, int i, int top_k, int* cj, ProxyFn proxy_of,
                                           KeepFn keep) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (top_k < 1) top_k = 1;
  long long pg[2], dn[2];
  float rf[2];  // within 3 * 2^-24 of the ratio (relative); 0: no candidate
  int cnt = 0;
  bool large = false;
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int j = lane + 32 * t;
    pg[t] = 0;
    dn[t] = 1;
    rf[t] = 0.0f;
    if (j < g && j != i) pg[t] = j < i ? proxy_of(j, i) : proxy_of(i, j);
    if (pg[t] > 0) {
      dn[t] = S.old[i] + S.old[j];
      if (dn[t] < 1) dn[t] = 1;
      rf[t] = __fdiv_rn(static_cast<float>(pg[t]), static_cast<float>(dn[t]));
    } else {
      pg[t] = 0;
    }
    large |= pg[t] >= kExactRatio || dn[t] >= kExactRatio;
    cnt += __popc(__ballot_sync(kFull, pg[t] > 0));
  }
  if (cnt <= top_k) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int j = lane + 32 * t;
      if (pg[t] > 0) keep(i < j ? i : j, i < j ? j : i);
    }
    return;
  }
  // a bound that at least top_k candidates reach, by bisection, until one
  // lane's worth is left
  float cut = 0.0f;
  if (cnt > 32 && top_k <= 28) {
    unsigned lo = 0, hi = 0x7f800000u;
    int left = cnt;
    while (hi - lo > 1 && left > 30) {
      const unsigned mid = lo + ((hi - lo) >> 1);
      const int c = __popc(__ballot_sync(kFull, __float_as_uint(rf[0]) >= mid)) +
                    __popc(__ballot_sync(kFull, __float_as_uint(rf[1]) >= mid));
      if (c >= top_k) {
        lo = mid;
        left = c;
      } else {
        hi = mid;
      }
    }
    cut = __uint_as_float(lo) * (1.0f - 9.5367431640625e-7f);
  }
  const bool in0 = pg[0] > 0 && rf[0] >= cut, in1 = pg[1] > 0 && rf[1] >= cut;
  const unsigned b0 = __ballot_sync(kFull, in0), b1 = __ballot_sync(kFull, in1);
  const int npass = __popc(b0) + __popc(b1);
  large = __any_sync(kFull, large);
  if (npass <= 32 && !large) {
    const unsigned lt = (1u << lane) - 1u;
    if (in0) cj[__popc(b0 & lt)] = lane;
    if (in1) cj[__popc(b0) + __popc(b1 & lt)] = lane + 32;
    __syncwarp();
    RankCand c[1] = {{0u, 1u, 0}};
    int j = 0;
    if (lane < npass) {
      j = cj[lane];
      const long long p = j < i ? proxy_of(j, i) : proxy_of(i, j);
      long long d = S.old[i] + S.old[j];
      if (d < 1) d = 1;
      c[0] = RankCand{static_cast<unsigned>(p), static_cast<unsigned>(d), S.q[j]};
    }
    int r[1];
    ExactRanks(c, r);
    if (lane < npass && r[0] < top_k) keep(i < j ? i : j, i < j ? j : i);
    __syncwarp();
    return;
  }
  int rank[2] = {0, 0};
  if (!large) {
    RankCand c[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      c[t] = RankCand{static_cast<unsigned>(pg[t]), static_cast<unsigned>(dn[t]), pg[t] > 0 ? S.q[lane + 32 * t] : 0};
    }
    ExactRanks(c, rank);
  } else {
    // the rounded quotients themselves
    for (int o = 0; o < g; ++o) {
      const long long op = __shfl_sync(kFull, o < 32 ? pg[0] : pg[1], o & 31);
      const long long od = __shfl_sync(kFull, o < 32 ? dn[0] : dn[1], o & 31);
      if (op <= 0) continue;
      const double oq = static_cast<double>(op) / static_cast<double>(od);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (pg[t] <= 0) continue;
        const double mq = static_cast<double>(pg[t]) / static_cast<double>(dn[t]);
        const bool better = oq != mq ? oq > mq : op != pg[t] ? op > pg[t] : S.q[o] < S.q[lane + 32 * t];
        rank[t] += better ? 1 : 0;
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int j = lane + 32 * t;
    if (pg[t] > 0 && rank[t] < top_k) keep(i < j ? i : j, i < j ? j : i);
  }
}

__device__ void MediumGroup(const MediumParams& P, MediumSmem& S, int ri) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kPer = kMedStage / kMedThreads;
  using BlockScan = cub::BlockScan<unsigned, kMedThreads, cub::BLOCK_SCAN_WARP_SCANS>;
  __shared__ typename BlockScan::TempStorage scan_tmp;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const QuotientView& Q = P.Q;
  const int gid = P.real[ri];
  const int g = P.glen[gid];
  const int npairs = g * (g - 1) / 2;
  auto& T = S.u.pairs;
  // ---- rows
  if (tid < kMedGroup) {
    int len = 0;
    if (tid < g) {
      const int rep = P.order[P.gstart[gid] + tid];
      S.q[tid] = rep;
      S.sz[tid] = Q.size[rep];
      len = Q.len[rep];
      S.off[tid] = Q.off[rep];
      S.heavy[tid] = HeavyAcc();
      S.old[tid] = 0;
      S.light[tid] = 0;
      S.keep[tid][0] = S.keep[tid][1] = 0;
    }
    int incl = len;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += y;
    }
    if (tid < g) S.start[tid] = incl - len;
    if (lane == 31) S.rows_end[warp] = incl;
  }
  if (tid < 10) S.acc[tid] = 0;
  if (tid == 0) {
    S.nkeys = 0;
    S.err[0] = S.err[1] = S.err[2] = 0;
    S.bad = 0;
  }
  __syncthreads();
  if (tid >= 32 && tid < g) S.start[tid] += S.rows_end[0];
  __syncthreads();
  const int E = S.rows_end[0] + S.rows_end[1];
  if (tid == 0) S.start[g] = E;
  int slots = 2 * kMedThreads;  // of the hash table: a power of two, at least twice the entries
  while (slots < 2 * E && slots < kMedSlots) slots <<= 1;
  for (int k = tid; k < slots; k += kMedThreads) S.u.hash.key[k] = -1;
  for (int k = tid; k < slots / 2; k += kMedThreads) S.u.hash.cnt[k] = 0;
  if (E > kMedStage) {  // not by the plan: row entries counted at Divide time only shrink
    if (tid == 0) {
      P.sel_cnt[ri] = 0;
      RaiseError(P.err, kErrSlots, gid, E, 0);
    }
    return;
  }
  __syncthreads();
  long long counts = 0;
  int largest = 0;
#pragma unroll
  for (int d = 0; d < kPer; ++d) {
    const int k = tid + d * kMedThreads;
    if (k >= E) break;
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
  // (each thread reads back its own entries)
  int slot[kPer];
  unsigned rank[kPer];
#pragma unroll
  for (int d = 0; d < kPer; ++d) {
    const int k = tid + d * kMedThreads;
    if (k >= E) break;
    const int t = EntNb(S.ent[k]);
    const int st = Q.size[t];
    S.tsz[k] = st;
    largest = st > largest ? st : largest;
    if (P.group_of[t] == gid) S.row[k] |= 0x80u;
  }
  if (tid < g) largest = max(largest, S.sz[tid]);
  counts = WarpSum(counts);
  largest = __reduce_max_sync(kFull, largest);
  if (lane == 0) {
    atomicAdd(&S.acc[0], static_cast<unsigned long long>(counts));
    atomicMax(&S.bad, largest);
  }
  __syncthreads();
  // 32-bit sums hold; products of two sizes and their sums fit 32 bits too
  const bool wide = static_cast<long long>(S.acc[0]) >= kSmallNarrow;
  const bool fits32 = !wide && S.bad < (1 << 13);
  __syncthreads();
  if (tid == 0) {
    S.acc[0] = 0;
    S.bad = 0;
  }
  // ---- row sums, runs of equal targets
  if (!wide) {
#pragma unroll
    for (int d = 0; d < kPer; ++d) {
      const int k = tid + d * kMedThreads;
      if (k >= E) break;
      const Entry e = S.ent[k];
      const int t = EntNb(e);
      AddRowEntry(S, S.row[k] & 0x7f, EntCnt(e), S.tsz[k]);
      unsigned h = BucketHash(t, static_cast<unsigned>(slots - 1));
      for (;;) {
        const int was = atomicCAS(&S.u.hash.key[h], -1, t);
        if (was == -1 || was == t) break;
        h = (h + 1) & static_cast<unsigned>(slots - 1);
      }
      slot[d] = static_cast<int>(h);
      rank[d] = (atomicAdd(&S.u.hash.cnt[h >> 1], 1u << (16 * (h & 1))) >> (16 * (h & 1))) & 0xffffu;
    }
  }
  __syncthreads();
  if (!wide) {
    const int per = slots / 2 / kMedThreads;  // words of two counters to a thread
    unsigned sum = 0, ex = 0;
    for (int d = 0; d < per; ++d) {
      const unsigned n = S.u.hash.cnt[tid * per + d];
      sum += (n & 0xffffu) + (n >> 16);
    }
    BlockScan(scan_tmp).ExclusiveSum(sum, ex);
    for (int d = 0; d < per; ++d) {
      const unsigned n = S.u.hash.cnt[tid * per + d];
      const unsigned mid = ex + (n & 0xffffu);
      S.u.hash.cnt[tid * per + d] = ex | mid << 16;
      ex = mid + (n >> 16);
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < kPer; ++d) {
      const int k = tid + d * kMedThreads;
      if (k >= E) break;
      const unsigned p = ((S.u.hash.cnt[slot[d] >> 1] >> (16 * (slot[d] & 1))) & 0xffffu) + rank[d];
      S.order[p] = static_cast<unsigned short>(k);
      S.rank[p] = static_cast<unsigned char>(rank[d]);  // a target is in a row once: below kMedGroup
    }
    __syncthreads();
  }
  // ---- pair sums (over the hash table's memory)
  for (int k = tid; k < npairs; k += kMedThreads) T.pc[k] = 0;
  for (int k = tid; k < (npairs + 1) / 2; k += kMedThreads) T.ovl[k] = 0;
  __syncthreads();
  unsigned examined = 0;
  bool any_bad = false;
  if (!wide) {
    for (int p = tid; p < E; p += kMedThreads) {
      const int k = S.order[p], r = S.rank[p];
      const int i = S.row[k] & 0x7f;
      const unsigned c = static_cast<unsigned>(EntCnt(S.ent[k]));
      const int st = S.tsz[k];
      if (S.row[k] & 0x80u) {
        const int j = P.idx_in_group[EntNb(S.ent[k])];
        if (i < j) atomicAdd(reinterpret_cast<unsigned*>(&T.pc[TriIndex(i, j, g)]) + 1, c);
      }
      examined += static_cast<unsigned>(r);
      for (int d = 1; d <= r; ++d) {
        const int k2 = S.order[p - d];
        const int j = S.row[k2] & 0x7f;
        const unsigned c2 = static_cast<unsigned>(EntCnt(S.ent[k2]));
        const int b = i < j ? TriIndex(i, j, g) : TriIndex(j, i, g);
        bool bad;
        int delta, corr;
        if (fits32) {
          TermOf32(S.sz[i], S.sz[j], st, static_cast<int>(c), static_cast<int>(c2), &delta, &corr, &bad);
        } else {
          const SharedTerm x = TermOf(S.sz[i], S.sz[j], st, c, c2, &bad);
          delta = static_cast<int>(x.delta);
          corr = static_cast<int>(x.corr);
        }
        any_bad |= bad;
        if (delta != 0) atomicAdd(reinterpret_cast<unsigned*>(&T.pc[b]) + 1, static_cast<unsigned>(delta));
        if (corr != 0) atomicAdd(reinterpret_cast<int*>(&T.pc[b]), corr);
        atomicAdd(&T.ovl[b >> 1], 1u << (16 * (b & 1)));
      }
    }
    if (any_bad) S.bad = 1;
  } else {
    // too large for 32 bits: a thread per member, a thread per pair
    if (tid < g) WideRow(S, tid);
    for (int pidx = tid; pidx < npairs; pidx += kMedThreads) {
      int a, b;
      TriPair(pidx, g, &a, &b);
      examined += static_cast<unsigned>(SmallMerge(S, a, b).ovl);
    }
  }
  __syncthreads();
  const bool slow = wide || S.bad != 0;  // SmallMerge gives the pairs' sums
  if (tid < g) SmallFinishRow(Q, S, tid, wide, &S.rs[tid]);
  __syncthreads();
  // ---- candidates
  auto proxy_of = [&](int a, int b) {  // a < b
    return slow ? SmallMerge(S, a, b).proxy : static_cast<long long>(T.pc[TriIndex(a, b, g)] >> 32);
  };
  auto keep = [&](int a, int b) { atomicOr(&S.keep[a][b >> 5], 1u << (b & 31)); };
  if (g - 1 <= P.top_k) {
    for (int pidx = tid; pidx < npairs; pidx += kMedThreads) {
      int a, b;
      TriPair(pidx, g, &a, &b);
      if (proxy_of(a, b) > 0) keep(a, b);
    }
  } else {
    for (int i = warp; i < g; i += kMedThreads / 32) MediumTopK(S, g, i, P.top_k, S.cj[warp], proxy_of, keep);
  }
  __syncthreads();
  // ---- gains of the kept pairs, keys of those that pass
  long long uni = 0, ovl = 0, raw_a = 0, raw_b = 0, nnz = 0;
  int cand = 0;
  // (a key takes the place of its pair's sums, read by this thread alone)
#pragma unroll 1
  for (int pidx = tid; pidx < npairs; pidx += kMedThreads) {
    int a, b;
    TriPair(pidx, g, &a, &b);
    if (!((S.keep[a][b >> 5] >> (b & 31)) & 1u)) {
      T.pc[pidx] = ~0ull;
      continue;
    }
    unsigned long long key = ~0ull;
    SmallPair r;
    if (slow) {
      r = SmallMerge(S, a, b);
    } else {
      r.proxy = static_cast<long long>(T.pc[pidx] >> 32);
      r.corr = static_cast<int>(T.pc[pidx] & 0xffffffffull);
      r.ovl = (T.ovl[pidx >> 1] >> (16 * (pidx & 1))) & 0xffff;
      r.bad = false;
    }
    const RowSums &A = S.rs[a], &B = S.rs[b];
    GainParts gp;
    if (!GainFromSums(A, B, SmallPairInfo(S, a, b, r), P.strict, &gp)) {
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
      if (gp.gain > kKeyGainMax) gp.err = kErrKeyRange;
      key = PackKey(gp.gain, a, b);
    }
    T.pc[pidx] = key;
    if (gp.err && atomicCAS(&S.err[0], 0, gp.err) == 0) {
      S.err[1] = S.q[a];
      S.err[2] = S.q[b];
    }
  }
  __syncthreads();  // the rows are read: their memory takes the list of keys
  unsigned long long* kin = S.ent;
  for (int pidx = tid; pidx < npairs; pidx += kMedThreads) {
    if (T.pc[pidx] != ~0ull) kin[atomicAdd(&S.nkeys, 1)] = T.pc[pidx];
  }
  cand = WarpSumInt(cand);
  examined = __reduce_add_sync(kFull, examined);
  uni = WarpSum(uni);
  ovl = WarpSum(ovl);
  raw_a = WarpSum(raw_a);
  raw_b = WarpSum(raw_b);
  nnz = WarpSum(nnz);
  if (lane == 0) {
    if (examined) atomicAdd(&S.acc[0], static_cast<unsigned long long>(examined));
    if (cand) {
      atomicAdd(&S.acc[1], static_cast<unsigned long long>(cand));
      atomicAdd(&S.acc[2], static_cast<unsigned long long>(uni));
      atomicAdd(&S.acc[3], static_cast<unsigned long long>(ovl));
      atomicAdd(&S.acc[4], static_cast<unsigned long long>(raw_a));
      atomicAdd(&S.acc[5], static_cast<unsigned long long>(raw_b));
      atomicAdd(&S.acc[6], static_cast<unsigned long long>(nnz));
    }
  }
  __syncthreads();
  // ---- selection
  const int m = S.nkeys;
  const int ns = m > 0 ? MatchKeys<kMedThreads>(S.match, kin, T.pc, m, g) : 0;
  const long long so = P.sel_off[ri];
  for (int i = warp; i < ns; i += kMedThreads / 32) {
    const unsigned long long k = S.match.chosen[i];
    const int a = static_cast<int>((k >> kKeyIdxBits) & kKeyIdxMask), b = static_cast<int>(k & kKeyIdxMask);
    const int la = S.rs[a].len, lb = S.rs[b].len;
    if (lane == 0) {
      const long long gain = kKeyGainMax - static_cast<long long>(k >> (2 * kKeyIdxBits));
      const int keep_rep = S.q[a], rem_rep = S.q[b];
      P.sel_keep[so + i] = keep_rep;
      P.sel_rem[so + i] = rem_rep;
      P.sel_gain[so + i] = gain;
      P.stamp[keep_rep] = 2 * P.block_stamp;
      P.stamp[rem_rep] = 2 * P.block_stamp + 1;
      P.partner[keep_rep] = rem_rep;
      P.partner[rem_rep] = keep_rep;
      P.seq[rem_rep] = static_cast<int>(so + i);
      P.sel_list[atomicAdd(&P.ctl->sel_total, 1u)] = static_cast<int>(so + i);
      atomicAdd(&S.acc[7], static_cast<unsigned long long>(gain));
      atomicAdd(&S.acc[8], static_cast<unsigned long long>(la + lb));
    }
  }
  __syncthreads();
  if (tid == 0) P.sel_cnt[ri] = ns;
  if (tid < 22) {
    if (tid == 0 && S.err[0]) RaiseError(P.err, S.err[0], S.err[1], S.err[2], 0);
    const unsigned long long um = m, uns = ns, ug = g;
    // one thread per counter
    int k = kStGroupCount;
    unsigned long long v = 0;
    switch (tid) {
      case 0: k = kStGroupCount; v = 1; break;
      case 1: k = kStRawPairCount; v = ug * (ug - 1) / 2; break;
      case 2: k = kStCandAfterPrune; v = S.acc[1]; break;
      case 3: k = kStProxyExamined; v = S.acc[0]; break;
      case 4: k = kStPrepareBytes; v = 12ull * E; break;
      case 5: k = kStExactCalls; v = S.acc[1]; break;
      case 6: k = kStInputNnz; v = S.acc[6]; break;
      case 7: k = kStRawA; v = S.acc[4]; break;
      case 8: k = kStRawB; v = S.acc[5]; break;
      case 9: k = kStUnion; v = S.acc[2]; break;
      case 10: k = kStOverlap; v = S.acc[3]; break;
      case 11: k = kStRejThreshold; v = S.acc[1] - um; break;
      case 12: k = kStPositive; v = um; break;
      case 13: k = kStRejOverlap; v = um - uns; break;
      case 14: k = kStCandPairs; v = um; break;
      case 15: k = kStSelected; v = uns; break;
      case 16: k = kStLocalGain; v = S.acc[7]; break;
      case 17: k = kStValidationCalls; v = uns; break;
      case 18: k = kStValidationWork; v = S.acc[8]; break;
      case 19: k = kStIsolatedGain; v = S.acc[7]; break;
      case 20: k = kStScoreBytes; v = S.acc[1] * (2 * sizeof(RowSums) + sizeof(PairInfo) + 24); break;
      default: break;
    }
    if (v) atomicAdd(&P.stats[k], v);
    if (tid == 21) atomicMax(&P.stats[kStGroupMaxSize], ug);
  }
}

__global__ void __launch_bounds__(kMedThreads, kMedCtas) MediumKernel(MediumParams P) {
  FollowsOn();
  extern __shared__ __align__(64) unsigned char med_smem[];
  MediumSmem& S = *reinterpret_cast<MediumSmem*>(med_smem);
  MediumGroup(P, S, P.list[P.list0 + blockIdx.x]);
}
