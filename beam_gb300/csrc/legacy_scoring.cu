// Legacy-objective pair scoring over a flat per-block CSR: the service behind
// the reference's Sweg::ScoreCandidatesCuda (include/sweg.hpp:656-658,
// src/cuda_scoring.cu:714-885), which --scoring-backend cuda uses with
// --cost-objective legacy (the README's CUDA mode).
//
// Input is the reference's Sweg::FlatAggCSR (include/sweg.hpp:395-403): row i
// has representative row_rep_ids[i], size row_sizes[i], self-loop count
// row_self_loops[i] and the sorted, duplicate-free entries neighbors /
// weights / neighbor_sizes [offsets[i], offsets[i+1]). A candidate pair
// (a_idx, b_idx) names two rows. Output per pair is {gain, before_cost} with
// the legacy encoding cost min(e, 1 + cap - e) (cap = s(s-1)/2 against the
// row's own representative, s * s_x otherwise), summed over the union of the
// two rows plus the two representatives themselves when a row lacks them;
// counts toward a row's own representative drop its self-loops first
// (src/cuda_scoring.cu:146-252, 282-357).
//
// GB300 form: one warp per pair. Lanes take 32 entries of row a at a time, four
// steps in flight, and find each neighbour in row b by binary search; then the
// entries of row b, skipping those present in row a. Pairs of more than
// kFlatLong entries are shared by the CTA's eight warps once each warp has done
// its own: a hub row of 1,600 entries is two chains of loads instead of 50,
// which were most of the kernel's time. Terms are summed per lane and
// reduced once per pair. A call packs the host inputs into one pinned buffer,
// copies it with one H2D, runs one kernel and copies 16 bytes per pair back.

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "beam_gb300.h"
#include "engine.h"

namespace beam {
namespace {

constexpr int kLegacyThreads = 256;

struct FlatView {
  const int* off;
  const int* rep;
  const int* nb;
  const long long* wt;
  const long long* nsz;
  const long long* rsz;
  const long long* self;
};

// Positions of four keys in the sorted flat row [s, e) (lower bounds), searched
// side by side.
constexpr int kFlatDeep = 4;
constexpr int kFlatLong = 256;

__device__ __forceinline__ void FlatLowerBounds(const int* nb, int s, int e, const int (&key)[kFlatDeep],
                                                int (&lo)[kFlatDeep]) {
  int hi[kFlatDeep];
#pragma unroll
  for (int d = 0; d < kFlatDeep; ++d) {
    lo[d] = s;
    hi[d] = e;
  }
  for (int span = e - s; span > 0; span >>= 1) {
#pragma unroll
    for (int d = 0; d < kFlatDeep; ++d) {
      if (lo[d] < hi[d]) {
        const int mid = lo[d] + ((hi[d] - lo[d]) >> 1);  // up to 2^31 - 1 entries in a call
        if (nb[mid] < key[d]) lo[d] = mid + 1; else hi[d] = mid;
      }
    }
  }
}

struct LegacyPair {
  int ra, rb;
  long long sa, sb, sm, la, lb;
};

// The before and after terms of one neighbour x of the pair.
__device__ __forceinline__ void LegacyTerm(const LegacyPair& p, int x, long long sx, long long ea_raw,
                                           long long eb_raw, long long* before, long long* after) {
  long long ea = ea_raw;
  if (x == p.ra) ea = ea_raw - p.la > 0 ? ea_raw - p.la : 0;
  long long eb = eb_raw;
  if (x == p.rb) eb = eb_raw - p.lb > 0 ? eb_raw - p.lb : 0;
  *before += EncodeCostForPair(p.ra, p.sa, x, sx, ea) + EncodeCostForPair(p.rb, p.sb, x, sx, eb);
  const int mrep = x == p.rb ? p.ra : x;
  const long long msz = x == p.rb ? p.sm : sx;
  *after += EncodeCostForPair(p.ra, p.sm, mrep, msz, ea + eb);
}

// The pair's terms over entries first, first + stride, ... of both rows (unsigned
// positions: the steps may pass 2^31 beyond a last entry near it).
struct LegacySums {
  long long before = 0, after = 0;
  bool seen_a = false, seen_b = false;
};

__device__ __forceinline__ void LegacyRows(const FlatView& F, const LegacyPair& p, int a0, int a1, int b0, int b1,
                                           unsigned first, unsigned stride, LegacySums* s) {
  const unsigned end_a = static_cast<unsigned>(a1), end_b = static_cast<unsigned>(b1);
  for (unsigned k0 = static_cast<unsigned>(a0) + first; k0 < end_a; k0 += stride * kFlatDeep) {
    int x[kFlatDeep], at[kFlatDeep];
#pragma unroll
    for (int d = 0; d < kFlatDeep; ++d) x[d] = k0 + d * stride < end_a ? F.nb[k0 + d * stride] : 0x7fffffff;
    FlatLowerBounds(F.nb, b0, b1, x, at);
#pragma unroll
    for (int d = 0; d < kFlatDeep; ++d) {
      const unsigned k = k0 + d * stride;
      if (k >= end_a) continue;
      const long long eb = at[d] < b1 && F.nb[at[d]] == x[d] ? F.wt[at[d]] : 0;
      LegacyTerm(p, x[d], F.nsz[k], F.wt[k], eb, &s->before, &s->after);
      s->seen_a |= x[d] == p.ra;
      s->seen_b |= x[d] == p.rb;
    }
  }
  for (unsigned k0 = static_cast<unsigned>(b0) + first; k0 < end_b; k0 += stride * kFlatDeep) {
    int x[kFlatDeep], at[kFlatDeep];
#pragma unroll
    for (int d = 0; d < kFlatDeep; ++d) x[d] = k0 + d * stride < end_b ? F.nb[k0 + d * stride] : 0x7fffffff;
    FlatLowerBounds(F.nb, a0, a1, x, at);
#pragma unroll
    for (int d = 0; d < kFlatDeep; ++d) {
      const unsigned k = k0 + d * stride;
      if (k >= end_b || (at[d] < a1 && F.nb[at[d]] == x[d])) continue;
      LegacyTerm(p, x[d], F.nsz[k], 0, F.wt[k], &s->before, &s->after);
      s->seen_a |= x[d] == p.ra;
      s->seen_b |= x[d] == p.rb;
    }
  }
}

__global__ void __launch_bounds__(kLegacyThreads) LegacyFlatScoreKernel(FlatView F, const int2* pairs,
                                                                         long long count, long long* out) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kWarps = kLegacyThreads / 32;
  __shared__ int is_long[kWarps];
  __shared__ long long part[kWarps][2];
  __shared__ int seen[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (long long w0 = static_cast<long long>(blockIdx.x) * kWarps; w0 < count;
       w0 += static_cast<long long>(gridDim.x) * kWarps) {
    // pass 0: a warp per pair; then the long ones of the eight, all warps on each
    for (int pass = 0; pass <= kWarps; ++pass) {
      const int which = pass == 0 ? warp : pass - 1;
      const long long w = w0 + which;
      if (pass > 0 && !is_long[which]) continue;
      LegacySums s;
      LegacyPair p = {0, 0, 0, 0, 0, 0, 0};
      bool mine = false;  // summed here
      if (w < count) {
        const int2 pr = pairs[w];
        const int a0 = F.off[pr.x], a1 = F.off[pr.x + 1];
        const int b0 = F.off[pr.y], b1 = F.off[pr.y + 1];
        mine = pass > 0 || static_cast<long long>(a1 - a0) + (b1 - b0) <= kFlatLong;
        if (mine) {
          p.ra = F.rep[pr.x];
          p.rb = F.rep[pr.y];
          p.sa = F.rsz[pr.x];
          p.sb = F.rsz[pr.y];
          p.sm = p.sa + p.sb;
          p.la = F.self[pr.x];
          p.lb = F.self[pr.y];
          LegacyRows(F, p, a0, a1, b0, b1, pass > 0 ? static_cast<int>(threadIdx.x) : lane,
                     pass > 0 ? kLegacyThreads : 32, &s);
        }
      }
      s.before = WarpSum(s.before);
      s.after = WarpSum(s.after);
      s.seen_a = __any_sync(kFull, s.seen_a);
      s.seen_b = __any_sync(kFull, s.seen_b);
      if (pass > 0) {
        if (lane == 0) {
          part[warp][0] = s.before;
          part[warp][1] = s.after;
          seen[warp] = (s.seen_a ? 1 : 0) | (s.seen_b ? 2 : 0);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          for (int k = 1; k < kWarps; ++k) {
            s.before += part[k][0];
            s.after += part[k][1];
            s.seen_a |= (seen[k] & 1) != 0;
            s.seen_b |= (seen[k] & 2) != 0;
          }
        }
      }
      if (mine && lane == 0 && (pass == 0 || warp == 0)) {
        // a row that does not list its own representative still pays for it
        if (!s.seen_a) LegacyTerm(p, p.ra, p.sa, 0, 0, &s.before, &s.after);
        if (p.rb != p.ra && !s.seen_b) LegacyTerm(p, p.rb, p.sb, 0, 0, &s.before, &s.after);
        out[2 * w] = s.before - s.after;
        out[2 * w + 1] = s.before;
      }
      if (pass == 0 && lane == 0) is_long[warp] = w < count && !mine ? 1 : 0;
      __syncthreads();
    }
    // A pass that is skipped has no barrier: without this one a warp could write
    // the next eight pairs' flags while another still reads these.
    if (w0 + static_cast<long long>(gridDim.x) * kWarps < count) __syncthreads();
  }
}

thread_local std::string g_flat_error;

size_t AlignUp(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace
}  // namespace beam

struct beam_flat_scorer {
  int device = 0;
  beam::OwnedStream stream;
  beam::DevBuf<unsigned char> d_in;
  beam::DevBuf<long long> d_out;
  beam::PinnedBuf<unsigned char> h_in;
  beam::PinnedBuf<long long> h_out;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  beam_flat_scorer_stats stats{};
  ~beam_flat_scorer() {
    for (cudaEvent_t e : ev) {
      if (e) cudaEventDestroy(e);
    }
    if (stream.s) cudaStreamSynchronize(stream.s);
    d_in.release();
    d_out.release();
  }
};

namespace {

int FlatFail(const std::string& msg) {
  beam::g_flat_error = msg;
  return -1;
}

}  // namespace

extern "C" {

const char* beam_flat_scorer_last_error(void) { return beam::g_flat_error.c_str(); }

int beam_flat_scorer_create(int32_t device, beam_flat_scorer** out) {
  if (!out) return FlatFail("null output handle");
  *out = nullptr;
  try {
    auto* s = new beam_flat_scorer();
    s->device = device;
    beam::CheckCuda(cudaSetDevice(device), "cudaSetDevice");
    beam::CheckCuda(cudaStreamCreateWithFlags(&s->stream.s, cudaStreamNonBlocking), "cudaStreamCreate");
    for (cudaEvent_t& e : s->ev) beam::CheckCuda(cudaEventCreate(&e), "cudaEventCreate");
    *out = s;
    return 0;
  } catch (const std::exception& ex) {
    return FlatFail(ex.what());
  }
}

void beam_flat_scorer_destroy(beam_flat_scorer* s) {
  if (!s) return;
  cudaSetDevice(s->device);
  delete s;
}

int beam_flat_scorer_memory_budget(beam_flat_scorer* s, int64_t* bytes) {
  if (!s || !bytes) return FlatFail("null argument");
  size_t free_b = 0, total_b = 0;
  cudaError_t st = cudaSetDevice(s->device);
  if (st == cudaSuccess) st = cudaMemGetInfo(&free_b, &total_b);
  if (st != cudaSuccess) return FlatFail(std::string("cudaMemGetInfo: ") + cudaGetErrorString(st));
  *bytes = static_cast<int64_t>(std::min<size_t>(free_b / 4, size_t{4} << 30));
  return 0;
}

int beam_flat_scorer_get_stats(const beam_flat_scorer* s, beam_flat_scorer_stats* out) {
  if (!s || !out) return FlatFail("null argument");
  *out = s->stats;
  return 0;
}

int beam_flat_scorer_score(beam_flat_scorer* s, const int32_t* pairs, int64_t count, const int32_t* offsets,
                           const int32_t* row_rep_ids, const int64_t* row_sizes, const int64_t* row_self_loops,
                           int32_t rows, const int32_t* neighbors, const int64_t* weights,
                           const int64_t* neighbor_sizes, int64_t entries, int64_t* gain, int64_t* before_cost) {
  using namespace beam;
  if (!s) return FlatFail("null scorer");
  if (count < 0 || rows < 0 || entries < 0) return FlatFail("negative size");
  if (count == 0) return 0;
  if (!pairs || !gain || !before_cost || !offsets || !row_rep_ids || !row_sizes || !row_self_loops ||
      (entries > 0 && (!neighbors || !weights || !neighbor_sizes))) {
    return FlatFail("null input or output pointer");
  }
  if (entries > INT32_MAX) return FlatFail("entries exceed the int offsets of FlatAggCSR");
  // the layout the kernel relies on: offsets rising from 0 to entries, rows
  // sorted by neighbour without repeats, pair indices naming rows
  if (offsets[0] != 0 || offsets[rows] != entries) return FlatFail("offsets must rise from 0 to entries");
  for (int32_t i = 0; i < rows; ++i) {
    if (offsets[i] > offsets[i + 1]) return FlatFail("offsets must rise from 0 to entries");
    unsigned falls = 0;  // no branch in the loop: it vectorises
    for (int32_t k = offsets[i] + 1; k < offsets[i + 1]; ++k) falls |= neighbors[k - 1] >= neighbors[k] ? 1u : 0u;
    if (falls) return FlatFail("row " + std::to_string(i) + " is not sorted by neighbour without repeats");
  }
  uint32_t largest = 0;  // a negative index is a large one
  for (int64_t p = 0; p < 2 * count; ++p) largest = std::max(largest, static_cast<uint32_t>(pairs[p]));
  if (largest >= static_cast<uint32_t>(rows)) {
    for (int64_t p = 0; p < count; ++p) {
      if (pairs[2 * p] < 0 || pairs[2 * p] >= rows || pairs[2 * p + 1] < 0 || pairs[2 * p + 1] >= rows) {
        return FlatFail("pair " + std::to_string(p) + " names a row outside [0, rows)");
      }
    }
  }
  try {
    CheckCuda(cudaSetDevice(s->device), "cudaSetDevice");
    AllocScope alloc(s->stream.s);
    // packed input: offsets | reps | neighbours | pairs (4-byte) then
    // weights | neighbour sizes | row sizes | self loops (8-byte)
    const size_t r1 = static_cast<size_t>(rows) + 1;
    const size_t ur = static_cast<size_t>(rows);
    const size_t ue = static_cast<size_t>(entries);
    const size_t up = static_cast<size_t>(count);
    size_t at = 0;
    const size_t o_off = at;
    at += 4 * r1;
    const size_t o_rep = at;
    at += 4 * ur;
    const size_t o_nb = at;
    at += 4 * ue;
    const size_t o_pair = at = AlignUp(at, 8);
    at += 8 * up;
    const size_t o_wt = at;
    at += 8 * ue;
    const size_t o_nsz = at;
    at += 8 * ue;
    const size_t o_rsz = at;
    at += 8 * ur;
    const size_t o_self = at;
    at += 8 * ur;
    const size_t total = at;
    s->h_in.ensure(total);
    s->d_in.ensure(total);
    s->h_out.ensure(2 * up);
    s->d_out.ensure(2 * up);
    unsigned char* h = s->h_in.p;
    std::memcpy(h + o_off, offsets, 4 * r1);
    std::memcpy(h + o_rep, row_rep_ids, 4 * ur);
    if (ue) std::memcpy(h + o_nb, neighbors, 4 * ue);
    std::memcpy(h + o_pair, pairs, 8 * up);
    if (ue) std::memcpy(h + o_wt, weights, 8 * ue);
    if (ue) std::memcpy(h + o_nsz, neighbor_sizes, 8 * ue);
    std::memcpy(h + o_rsz, row_sizes, 8 * ur);
    std::memcpy(h + o_self, row_self_loops, 8 * ur);
    cudaStream_t st = s->stream.s;
    unsigned char* d = s->d_in.p;
    CheckCuda(cudaMemcpyAsync(d, h, total, cudaMemcpyHostToDevice, st), "h2d flat block");
    FlatView F{reinterpret_cast<const int*>(d + o_off), reinterpret_cast<const int*>(d + o_rep),
               reinterpret_cast<const int*>(d + o_nb), reinterpret_cast<const long long*>(d + o_wt),
               reinterpret_cast<const long long*>(d + o_nsz), reinterpret_cast<const long long*>(d + o_rsz),
               reinterpret_cast<const long long*>(d + o_self)};
    const int grid = static_cast<int>(std::min<int64_t>((count + 7) / 8, 152 * 16));
    CheckCuda(cudaEventRecord(s->ev[0], st), "event");
    LegacyFlatScoreKernel<<<grid, kLegacyThreads, 0, st>>>(F, reinterpret_cast<const int2*>(d + o_pair), count,
                                                            s->d_out.p);
    CheckCuda(cudaGetLastError(), "legacy scoring launch");
    CheckCuda(cudaEventRecord(s->ev[1], st), "event");
    CheckCuda(cudaMemcpyAsync(s->h_out.p, s->d_out.p, 16 * up, cudaMemcpyDeviceToHost, st), "d2h results");
    CheckCuda(cudaStreamSynchronize(st), "sync");
    float ms = 0.f;
    CheckCuda(cudaEventElapsedTime(&ms, s->ev[0], s->ev[1]), "event elapsed");
    for (size_t p = 0; p < up; ++p) {
      gain[p] = s->h_out.p[2 * p];
      before_cost[p] = s->h_out.p[2 * p + 1];
    }
    s->stats.calls += 1;
    s->stats.kernel_launches += 1;
    s->stats.pairs += count;
    s->stats.h2d_bytes += static_cast<int64_t>(total);
    s->stats.d2h_bytes += static_cast<int64_t>(16 * up);
    s->stats.kernel_ms += ms;
    s->stats.max_pairs_per_launch = std::max<int64_t>(s->stats.max_pairs_per_launch, count);
    return 0;
  } catch (const std::exception& ex) {
    return FlatFail(ex.what());
  }
}

}  // extern "C"
