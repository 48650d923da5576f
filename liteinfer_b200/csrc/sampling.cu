// Sampling: a row of logits is an arg-max, or a draw from what temperature, top-k and top-p leave of it.
//
// Order of operations as liteinfer/sampling/sampler.py:50-63: logits / temperature
// -> top-k (exactly k survive; ties at the boundary do not widen it, :76-83)
// -> softmax -> top-p on those probabilities (an entry is dropped when the mass
// before it, in descending order, exceeds p: the entry that crosses p is kept,
// :86-97) -> one draw.  temperature == 0 or top_k == 1 is the arg-max (:36).
//
// The draw takes a uniform number in [0, 1) that the host supplies per row, so a
// request's stream of draws does not depend on what else is in the batch.  All
// arithmetic is 32-bit; the selections use exact integer sums (counts, and
// probabilities in 2^-32 fixed point), so a given row always gives the same
// token.  Among equal values the lower index comes first.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace li {

constexpr int kThreads = 1024;

__device__ __forceinline__ uint32_t ordered_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

__device__ ArgMax block_argmax(ArgMax mine, ArgMax* scratch /* 32 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax other{__shfl_xor_sync(0xffffffffu, mine.v, o), __shfl_xor_sync(0xffffffffu, mine.i, o)};
    mine = better(mine, other);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = mine;
  __syncthreads();
  ArgMax r = scratch[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = better(r, scratch[w]);
  return r;
}

// ---- the sampling kernel --------------------------------------------------------------------------
// A row belongs to a cluster of blocks (one per 8,192 columns, at most eight), each with its share of the columns in its
// shared memory, so the logits are read once.  Every later pass runs over shared memory; what the blocks of a row must agree on (the maximum, a
// histogram, a running weight) they read from one another's shared memory behind a cluster barrier, and each works
// the answer out for itself.
//
// Top-k and top-p are the same selection: in descending order, keep the elements whose preceding weight (1 each, or
// the probability) is within a limit.  The first histogram bins by the distance below the row's maximum, in steps of
// 1/73 for 14 units (counts: see kCountsPerUnit): the interesting values spread over hundreds of bins, so the atomics rarely meet, and the
// last bin takes the rest, whose weight is added up in registers.  Elements above the boundary bin are in, those below are out.  The walk
// behind the histogram lists what can still be chosen, in the order of the columns, and picks out what has to be told apart:
// the boundary bin, or for a top-k that leaves few (most_sorted), everything.  Those few are sorted, by every block for
// itself (top-p), or by one block that then finishes the row alone, top-p and draw included (top-k).  Where they are more (equal
// values, a flat row, a share of 2^16 columns) histograms over ever narrower ranges of keys tell them apart, each a meeting of the blocks.
//
// Bound by the walks over the whole row (load and maximum 6,400 cycles, histogram 5,000 to 16,000, listing 5,000 to 12,000 for
// 16,000 columns a block) and by what a meeting costs: a cluster barrier and the reads of eight blocks' memory behind it, 2,000
// to 6,000 cycles.  Walks take four columns a lane, so that one trip's latencies cover four columns and what is kept of them is
// placed by three ballots; all that a lane needs from other blocks is asked for before the first of it is used.
// Measured on B200, 128,256 bfloat16 columns, 48 rows: all kinds of parameters 55.9 us (85.2 with a histogram per level of keys,
// one column a lane), top-k 50 37.1 (47.4), top-p 0.9 68.9 (98.5), both 45.7 (86.9); one row 22.8 (33.0), 37.1 (47.4), 28.7 (49.4).
constexpr int kSampleThreads = 512, kSampleWarps = kSampleThreads / 32;
constexpr int kMostRanks = 8;      // blocks of a row's cluster
// A row of no more columns is one block's, and so on.  The passes over a share get longer, but there are fewer blocks to meet at
// every barrier, and more rows at once: 48 rows of 32,000 columns, top-p 0.9, take 27 us in four blocks each and 43 in eight.  Where the
// launch's blocks have an SM each all the same, half as many columns: 12 rows of 16,000, top-p 0.9, 22.0 us in two blocks each
// and 17.2 in four, of 32,000 23.5 in four and 19.7 in eight.
constexpr int kRankColumns = 8192;
constexpr int kBins = 1024;
constexpr int kListed = 512;       // columns that a warp can list; where one has more its block goes on walking its whole share
constexpr int kCandidates = 1024;  // elements of a row that are sorted at once, two a thread
constexpr int kSampleMostSmem = 200 << 10;
constexpr size_t kSmemOfSm = 228 << 10, kReservedSmem = 1 << 10;      // an SM's shared memory, and what it keeps of it for a block
constexpr float kBinsPerUnit = 73.f;   // by weight: the last bin holds all that lies 14 and more below the maximum
// By count (top-k) what lies far below the maximum counts as much as what is near it, so a bin holds 1/46 of a unit for 14 units and then one
// unit up to 393: the k-th value of a row with a low temperature or few large values is in a bin of a few columns, too.  With the bins of
// the weights 24 rows of 262,144 columns, top-k 50 at a temperature of 0.2, took 124 us (36 now), 12 of 1,000 20 (10.7).
constexpr float kCountsPerUnit = 46.f, kFar = 14.f, kFarFrom = kFar * (kCountsPerUnit - 1.f);      // (where the second line cuts zero)
static_assert(kFarFrom < kBins - 2, "the lines meet within the histogram");
// A top-k is finished by sorting where no more than this many columns can be chosen, which costs two sorts and saves the histograms that tell the
// boundary bin's columns apart and, with a top-p behind it, those of the second selection.  In a row of one block, which meets nobody, a
// histogram is cheap: 8,192 float32 columns, top-k 50 alone 15.5 us by sorts and 12.4 by histograms, with top-p 0.9 16.3 and 17.6, top-k 200 with
// it 20.0 and 17.9.  In a cluster's: 32,000 bfloat16, top-k 100 alone 19.3 and 20.3, 200 21.3 and 20.6, 800 41 and 21; with top-p 400 26
// and 30, 800 42 and 30.
__host__ __device__ constexpr unsigned most_sorted(bool alone, bool weights_follow) { return alone ? (weights_follow ? 128 : 0) : weights_follow ? 512 : 128; }
static_assert(most_sorted(false, true) <= kCandidates, "a block holds what is sorted");

struct Keep {        // the surviving set: key > beta, or key == beta and index <= tie_cut
  uint32_t beta;
  int tie_cut;
  __device__ __forceinline__ bool has(uint32_t key, int i) const { return key > beta || (key == beta && i <= tie_cut); }
};

struct SampleSmem {
  // Two histograms in turn: kBins counts, or the sums of the weights' lower 16 bits and, behind them, of the bits above;
  // for a share of 2^16 columns or more, where those could overflow, kBins 64-bit sums.  Behind the row's barrier that follows, the one just
  // summed is read by nobody any more, and the other one has been free since the barrier before: see `candidates`.
  alignas(16) uint32_t bins[2][2 * kBins];
  unsigned long long exchange[8];           // what other blocks of the cluster read, one slot per exchange
  unsigned long long warp[kSampleWarps];
  ArgMax warp_best[32];
  ArgMax best[kMostRanks];                  // of every block of the row
  unsigned long long before, mass;          // of the boundary bin
  int chosen;
  int found;                                // entries of `cand`, or more where it did not hold them all
  Keep keep;
  uint16_t list[kSampleWarps][kListed];
  // This block's elements of the boundary bin (top-k: and of those above it), in the histogram whose turn is next: every block has read
  // what it held before it came to the barrier in front of the sums that found the boundary.  In 8 KB of their own they left an SM
  // room for one block of a row of 151,936 columns where there had been two.
  __device__ __forceinline__ unsigned long long* candidates(int turn) { return reinterpret_cast<unsigned long long*>(bins[turn]); }
};
static_assert(sizeof(uint32_t[2 * kBins]) == kCandidates * sizeof(unsigned long long), "candidates lie in a histogram");

// One block's share of a row: columns [base, base + n) of it, whose element i lies at data[i] (in shared memory, or the row
// itself where a share does not fit).  The walks over a share go warp by warp: each warp has a run of columns, and once
// `listed` is set a list of those of its columns that still count, so a walk is in the order of the columns.
template <typename S, bool kStaged>
struct Share {
  const S* data;
  const uint16_t* list;      // this warp's list
  int n, base;
  int from, to;              // this warp's columns, or the length of its list (from 0)
  bool listed;
  bool undivided;            // data holds value, not value / temperature
  bool wide;                 // the row's shares have 2^16 columns or more
  float temp, row_max;
  float bin_max, bin_scale;  // the maximum as it is stored in `data`, and bins per unit of what is stored there
  uint32_t max_key;
  __device__ __forceinline__ int column(int j) const { return listed ? list[j] : j; }
  // Four neighbours as they are stored, i a multiple of four (what lies behind the share's end has no meaning).
  __device__ __forceinline__ void four(int i, float (&f)[4]) const {
    if constexpr (kStaged) {
      if constexpr (sizeof(S) == 4) {
        const float4 v = *reinterpret_cast<const float4*>(data + i);
        f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
      } else {
        const uint2 v = *reinterpret_cast<const uint2*>(data + i);
        f[0] = __uint_as_float(v.x << 16), f[1] = __uint_as_float(v.x & 0xffff0000u);
        f[2] = __uint_as_float(v.y << 16), f[3] = __uint_as_float(v.y & 0xffff0000u);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) f[e] = i + e < n ? to_float(data[i + e]) : 0.f;
    }
  }
  __device__ __forceinline__ float quotient(float stored) const {
    if constexpr (kStaged && sizeof(S) == 4) return stored;
    else return undivided ? stored / temp : stored;
  }
  __device__ __forceinline__ float value(int i) const { return quotient(to_float(data[i])); }
  __device__ __forceinline__ unsigned long long weight(float x) const {
    const float scaled = expf(x - row_max) * 4294967296.0f;
    return scaled < 4294967296.0f ? (unsigned long long)(uint32_t)scaled : (unsigned long long)scaled;
  }
  // Where a difference from the maximum (as it is stored) lies among the bins of counts (`unit`) or weights.
  template <bool unit>
  __device__ __forceinline__ float place(float d) const {
    const float t = d * bin_scale;
    return fminf(unit ? fminf(t, fmaf(t, 1.f / kCountsPerUnit, kFarFrom)) : t, (float)(kBins - 1));
  }
  // The bin never rises with the value, and equal values divided by the temperature are in one bin.  A difference that is no
  // number (infinities, NaN) goes by the key.
  template <bool unit>
  __device__ __forceinline__ int bin_of(float stored) const {
    const float d = bin_max - stored;
    if (!(d >= 0.f)) return ordered_key(quotient(stored)) >= max_key ? 0 : kBins - 1;
    return (int)place<unit>(d);
  }
  template <bool unit>
  __device__ __forceinline__ int bin(int i) const { return bin_of<unit>(to_float(data[i])); }
  __device__ __forceinline__ void bins_per_unit(float bins) { bin_scale = undivided ? bins / temp : bins; }
};

// The difference from the maximum, in units, at which a bin begins.
template <bool unit>
__device__ __forceinline__ float bin_begin(int bin) {
  const float b = (float)bin;
  return unit ? fmaxf(b * (1.f / kCountsPerUnit), b - kFarFrom) : b * (1.f / kBinsPerUnit);
}

// The barrier of a row's blocks; a row that is one block's (kAlone) has no use for a cluster's.
template <bool kAlone>
__device__ __forceinline__ void row_sync(const cg::cluster_group& cluster) {
  if constexpr (kAlone) __syncthreads();
  else cluster.sync();
}

__device__ __forceinline__ unsigned long long warp_inclusive(unsigned long long v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  return v;
}

// A candidate: its key above its index counted down, so that descending order is the selection's (equal values by ascending
// index).  Zero is none: it sorts last.
__device__ __forceinline__ unsigned long long candidate(uint32_t key, int i) {
  return (unsigned long long)key << 32 | (0xffffffffu - (uint32_t)i);
}
__device__ __forceinline__ float key_value(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

// Sorts a block's numbers in descending order: thread t holds the t-th and, H = 2, the (t + 512)-th of the first `many` (a power
// of two, 32 or more).  A bitonic network; steps within a warp are shuffles, the others meet in `a`.
template <int H>
__device__ __forceinline__ void sort_down_by(unsigned long long (&v)[2], int many, unsigned long long* a) {
  const int t = threadIdx.x;
  const bool active = H == 2 || t < many;            // whole warps
  const auto step = [&](int size, int stride, const unsigned long long (&other)[2]) {
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const bool greater = (((t + h * kSampleThreads) & size) == 0) == ((t & stride) == 0);
      v[h] = (v[h] > other[h]) == greater ? v[h] : other[h];
    }
  };
#pragma unroll 1
  for (int size = 2; size <= many; size <<= 1) {
#pragma unroll 1
    for (int stride = size >> 1; stride >= 32; stride >>= 1) {
      if (H == 2 && stride == kSampleThreads) {
        const unsigned long long hi = max(v[0], v[1]), lo = min(v[0], v[1]);
        v[0] = hi;
        v[1] = lo;
        continue;
      }
      unsigned long long other[2];
      if (active) {
#pragma unroll
        for (int h = 0; h < H; ++h) a[t + h * kSampleThreads] = v[h];
      }
      __syncthreads();
      if (active) {
#pragma unroll
        for (int h = 0; h < H; ++h) other[h] = a[(t ^ stride) + h * kSampleThreads];
      }
      __syncthreads();
      if (active) step(size, stride, other);
    }
    if (active) {
#pragma unroll
      for (int stride = 16; stride > 0; stride >>= 1) {
        if (stride >= size) continue;
        unsigned long long other[2];
#pragma unroll
        for (int h = 0; h < H; ++h) other[h] = __shfl_xor_sync(0xffffffffu, v[h], stride);
        step(size, stride, other);
      }
    }
  }
}
__device__ __noinline__ void sort_down(unsigned long long (&v)[2], int many, unsigned long long* a) {
  if (many > kSampleThreads) sort_down_by<2>(v, many, a);
  else sort_down_by<1>(v, many, a);
}

// Inclusive sums over the first `many` of a block's 1,024 numbers (those behind are zero), thread t holding the t-th and the
// (t + 512)-th; returns the sum of all.
__device__ unsigned long long scan_both(unsigned long long (&v)[2], int many, SampleSmem& sm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long all = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h * kSampleThreads >= many) break;
    v[h] = warp_inclusive(v[h], lane);
    __syncthreads();
    if (lane == 31) sm.warp[w] = v[h];
    __syncthreads();
    unsigned long long start = all;
#pragma unroll
    for (int i = 0; i < kSampleWarps; ++i) {
      const unsigned long long part = sm.warp[i];
      if (i < w) start += part;
      all += part;
    }
    v[h] += start;
  }
  return all;
}

__device__ __forceinline__ int power_above(int n) { return n <= 32 ? 32 : 1 << (32 - __clz(n - 1)); }

// The candidates of all blocks of a row, thread t taking the t-th and the (t + 512)-th.  Behind a barrier of the row.
// Returns how many there are, or more than kCandidates where a block did not hold all of its own.
__device__ int gather_candidates(unsigned long long (&v)[2], int turn, SampleSmem& sm) {
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = (int)cluster.num_blocks();
  int count[kMostRanks], all = 0;
  bool whole = true;
#pragma unroll
  for (int r = 0; r < kMostRanks; ++r) count[r] = r < ranks ? *cluster.map_shared_rank(&sm.found, r) : 0;
#pragma unroll
  for (int r = 0; r < kMostRanks; ++r) {
    whole = whole && count[r] <= kCandidates;
    all += min(count[r], kCandidates);
  }
  v[0] = v[1] = 0;
  if (!whole || all > kCandidates) return kCandidates + 1;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    int at = threadIdx.x + h * kSampleThreads;
    if (at >= all) break;
    int r = 0;
#pragma unroll
    for (int i = 0; i < kMostRanks - 1; ++i) {
      if (r == i && at >= count[i]) {
        at -= count[i];
        ++r;
      }
    }
    v[h] = cluster.map_shared_rank(sm.candidates(turn), r)[at];
  }
  return all;
}

// Sums the blocks' histograms `buf` and finds the last non-empty bin whose preceding weight is within the limit
// (`whole`: the limit is the share `top_p` of the whole sum, and is left in `limit`).  Every thread returns with the bin,
// the weight before it and its own weight.
template <bool unit, bool kAlone>
__device__ void find_boundary(SampleSmem& sm, int buf, bool wide, unsigned long long above, bool whole, float top_p,
                              unsigned long long& limit, int& chosen, unsigned long long& before, unsigned long long& mass) {
  cg::cluster_group cluster = cg::this_cluster();
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (t == 0) sm.chosen = -1;
  row_sync<kAlone>(cluster);
  static_assert(kBins == 2 * kSampleThreads, "two bins a thread");
  unsigned long long a = 0, b = 0;
  const int ranks = (int)cluster.num_blocks();
  if (!unit && wide) {
    for (int r = 0; r < ranks; ++r) {
      const ulonglong2 both = *reinterpret_cast<const ulonglong2*>(cluster.map_shared_rank(&sm.bins[buf][4 * t], r));
      a += both.x;
      b += both.y;
    }
  } else {
    // (Four blocks' sums are asked for before the first is used.)
#pragma unroll
    for (int first = 0; first < kMostRanks; first += 4) {
      if (first >= ranks) break;
      uint2 lo[4], hi[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = first + i;
        lo[i] = hi[i] = make_uint2(0, 0);
        if (r < ranks) {
          lo[i] = *reinterpret_cast<const uint2*>(cluster.map_shared_rank(&sm.bins[buf][2 * t], r));
          if (!unit) hi[i] = *reinterpret_cast<const uint2*>(cluster.map_shared_rank(&sm.bins[buf][kBins + 2 * t], r));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a += lo[i].x + ((unsigned long long)hi[i].x << 16);
        b += lo[i].y + ((unsigned long long)hi[i].y << 16);
      }
    }
  }
  const unsigned long long incl = warp_inclusive(a + b, lane);
  if (lane == 31) sm.warp[w] = incl;
  __syncthreads();
  unsigned long long start = above, total = 0;
#pragma unroll
  for (int i = 0; i < kSampleWarps; ++i) {
    const unsigned long long v = sm.warp[i];
    if (i < w) start += v;
    total += v;
  }
  if (whole) limit = (unsigned long long)((double)top_p * (double)total);
  const unsigned long long first = start + incl - (a + b), second = first + a;
  int mine = -1;
  if (a && first <= limit) mine = 2 * t;
  if (b && second <= limit) mine = 2 * t + 1;
  if (mine >= 0) atomicMax(&sm.chosen, mine);
  __syncthreads();
  if (mine >= 0 && mine == sm.chosen) {
    sm.before = (mine & 1) ? second : first;
    sm.mass = (mine & 1) ? b : a;
  }
  __syncthreads();
  chosen = sm.chosen;       // -1: nothing has any weight (a row whose maximum is infinite)
  before = sm.before;
  mass = sm.mass;
}

// The last selections and the draw of a row whose top-k leaves few elements, by one block: the candidates, all that top-k
// keeps among them, lie over the blocks.  Returns the column.
template <typename S, bool kStaged>
__device__ int draw_from_candidates(const Share<S, kStaged>& share, int k, float top_p, double u, int fallback, int turn, SampleSmem& sm) {
  const int t = threadIdx.x;
  unsigned long long* table = sm.candidates(turn ^ 1);      // what was summed last
  unsigned long long v[2];
  const int many = gather_candidates(v, turn, sm);
  sort_down(v, power_above(many), table);
  k = min(k, many);
  unsigned long long weight[2], upto[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    weight[h] = t + h * kSampleThreads < k ? share.weight(key_value((uint32_t)(v[h] >> 32))) : 0;
    upto[h] = weight[h];
  }
  if (top_p > 0.f && top_p < 1.f) {
    const unsigned long long total = scan_both(upto, k, sm);
    const unsigned long long limit = (unsigned long long)((double)top_p * (double)total);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (upto[h] - weight[h] > limit) weight[h] = 0;
  }
  // In the order of the columns: the index, counted down, above the key.
#pragma unroll
  for (int h = 0; h < 2; ++h) v[h] = weight[h] ? v[h] << 32 | v[h] >> 32 : 0;
  __syncthreads();
  sort_down(v, power_above(k), table);
#pragma unroll
  for (int h = 0; h < 2; ++h)
    upto[h] = weight[h] = v[h] && t + h * kSampleThreads < k ? share.weight(key_value((uint32_t)v[h])) : 0;
  const unsigned long long total = scan_both(upto, k, sm);
  unsigned long long target = (unsigned long long)(u * (double)total);
  if (target >= total) target = total ? total - 1 : 0;
  if (t == 0) sm.chosen = fallback;
  __syncthreads();
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (upto[h] > target && upto[h] - weight[h] <= target) sm.chosen = (int)(0xffffffffu - (uint32_t)(v[h] >> 32));
  __syncthreads();
  return sm.chosen;
}

// Among the elements of `within`, in descending order of value (equal values by ascending index), keeps each element
// whose preceding weight sum is within the limit.  `unit` weights count elements (top-k with limit k - 1); otherwise the
// weight is exp(x - row_max) in 2^-32 fixed point (top-p with limit p * total).  `turn`: the histogram to use next;
// `slot`: the next free exchange.  Lists what survives the first histogram.  `few` (top-k, whose `top_p` is what follows it): set where what it keeps lies among
// that many candidates, which one block is to finish with; nothing else is then returned.
template <bool unit, bool kAlone, typename S, bool kStaged>
__device__ Keep select_prefix(Share<S, kStaged>& share, bool all_in, Keep within, unsigned long long limit, float top_p, int vocab,
                              int& turn, int& slot, int& few, SampleSmem& sm) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool wide = share.wide;
  cg::cluster_group cluster = cg::this_cluster();
  int first_bin = -1;
  uint32_t low_key = 0, high_key = 0xffffffffu;
  unsigned long long above = 0, mass = 0;
  for (int level = 0;; ++level) {
    const uint32_t range = high_key - low_key;
    const int shift = level == 0 ? 32 : max(0, 32 - __clz(range) - 10);
    uint32_t* bins = sm.bins[turn];
    for (int i = threadIdx.x; i < 2 * kBins; i += kSampleThreads) bins[i] = 0;
    if (level == 0 && threadIdx.x == 0) sm.found = 0;
    __syncthreads();
    const auto add = [&](int bin, unsigned long long weight) {
      if (unit) {
        atomicAdd(bins + bin, 1u);
      } else if (wide) {
        atomicAdd(reinterpret_cast<unsigned long long*>(bins) + bin, weight);
      } else {
        const uint32_t high = (uint32_t)(weight >> 16);
        atomicAdd(bins + bin, (uint32_t)weight & 0xffffu);
        if (high) atomicAdd(bins + kBins + bin, high);
      }
    };
    if (all_in && level == 0) {
      unsigned long long far = 0;      // the last bin's weight: what many columns have is not added one by one
#pragma unroll 1
      for (int j = share.from + 4 * lane; j < share.to; j += 128) {
        float f[4];
        share.four(j, f);
        int bin[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) bin[e] = share.template bin_of<unit>(f[e]);
        if (unit) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (j + e < share.to) atomicAdd(bins + bin[e], 1u);
        } else {
          unsigned long long weight[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) weight[e] = j + e < share.to ? share.weight(share.quotient(f[e])) : 0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (bin[e] == kBins - 1) far += weight[e];
            else add(bin[e], weight[e]);
          }
        }
      }
      if (!unit) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) far += __shfl_xor_sync(0xffffffffu, far, o);
        if (lane == 0) add(kBins - 1, far);
      }
    } else {
#pragma unroll 2
      for (int j = share.from + lane; j < share.to; j += 32) {
        const int i = share.column(j);
        int bin = share.template bin<unit>(i);
        const float x = share.value(i);
        const uint32_t key = ordered_key(x);
        if (!all_in && !within.has(key, share.base + i)) continue;
        if (level > 0) {
          if (bin != first_bin || key < low_key || key > high_key) continue;
          bin = (int)((high_key - key) >> shift);
        }
        add(bin, unit ? 1ull : share.weight(x));
      }
    }
    int chosen;
    find_boundary<unit, kAlone>(sm, turn, wide, above, !unit && level == 0, top_p, limit, chosen, above, mass);
    turn ^= 1;
    if (chosen < 0) return within;
    if (level == 0) {
      first_bin = chosen;
      const float far = 1.0001f * bin_begin<unit>(chosen + 1), near = 0.9999f * bin_begin<unit>(chosen);
      const float slack = 1e-5f * (fabsf(share.row_max) + 1.f);
      if (chosen > 0) high_key = ordered_key(share.row_max - near + slack);
      if (chosen < kBins - 1) low_key = ordered_key(share.row_max - far - slack);
      if (!(fabsf(share.row_max) < 3.0e38f)) low_key = 0, high_key = 0xffffffffu;
      if (wide) continue;
      // List what the boundary bin and those above it hold, and put what has to be told apart where the other blocks find it.
      const bool collect = !unit || above + mass <= most_sorted(kAlone, top_p > 0.f && top_p < 1.f);
      bool fits = !share.listed;
      int listed = 0;
      const auto put = [&](bool taken, int i, float x) {       // a warp's elements that have to be told apart
        const unsigned votes = __ballot_sync(0xffffffffu, taken);
        if (!votes) return;
        int at = 0;
        if (lane == 0) at = atomicAdd(&sm.found, __popc(votes));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(votes & ((1u << lane) - 1));
        if (taken && at < kCandidates) sm.candidates(turn)[at] = candidate(ordered_key(x), share.base + i);
      };
      if (share.listed) {
        for (int j = share.from; j < share.to && collect; j += 32) {
          const int i = j + lane < share.to ? share.column(j + lane) : 0;
          const int bin = j + lane < share.to ? share.template bin<unit>(i) : kBins;
          const float x = share.value(i);
          put((unit ? bin <= first_bin : bin == first_bin) && (all_in || within.has(ordered_key(x), share.base + i)), i, x);
        }
      } else {
        // For a difference that is a number two comparisons are as good as its bin.
        const float lowest = first_bin == kBins - 1 ? INFINITY : (float)(first_bin + 1), boundary = (float)first_bin;
#pragma unroll 1
        for (int j = share.from; j < share.to && (fits || collect); j += 128) {
          const int i = j + 4 * lane;
          float f[4];
          unsigned in = 0, taken = 0;
          bool odd = false;
          share.four(min(i, share.n - 1) & ~3, f);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float d = share.bin_max - f[e], t = share.template place<unit>(d);
            const bool here = i + e < share.to;
            odd = odd || (here && !(d >= 0.f));
            in |= (unsigned)(here && t < lowest) << e;
            taken |= (unsigned)(here && t < lowest && (unit || t >= boundary)) << e;
          }
          if (__any_sync(0xffffffffu, odd) || !all_in) {
            in = taken = 0;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              if (i + e >= share.to) continue;
              const int bin = share.template bin_of<unit>(f[e]);
              if (bin > first_bin || !(all_in || within.has(ordered_key(share.quotient(f[e])), share.base + i + e))) continue;
              in |= 1u << e;
              if (unit || bin == first_bin) taken |= 1u << e;
            }
          }
          if (!__any_sync(0xffffffffu, in != 0)) continue;
          if (fits) {
            // The lanes' counts, 0 to 4, are added up bit by bit.
            const int many = __popc(in);
            const unsigned below = (1u << lane) - 1, ones = __ballot_sync(0xffffffffu, many & 1),
                           twos = __ballot_sync(0xffffffffu, many & 2), fours = __ballot_sync(0xffffffffu, many & 4);
            const int all = __popc(ones) + 2 * __popc(twos) + 4 * __popc(fours);
            fits = listed + all <= kListed;
            if (fits) {
              int at = listed + __popc(ones & below) + 2 * __popc(twos & below) + 4 * __popc(fours & below);
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (in >> e & 1) sm.list[w][at++] = (uint16_t)(i + e);
              listed += all;
            }
          }
          if (collect && __any_sync(0xffffffffu, taken != 0)) {
#pragma unroll
            for (int e = 0; e < 4; ++e) put(taken >> e & 1, i + e, share.quotient(f[e]));
          }
        }
      }
      if (!share.listed && __syncthreads_and(fits)) {
        share.listed = true;
        share.list = sm.list[w];
        share.from = 0;
        share.to = listed;
      }
      if (!collect) continue;
      row_sync<kAlone>(cluster);
      if (unit) {
        few = (int)(above + mass);
        return within;
      }
      // The few elements of the boundary bin, sorted, tell where the cut falls; every block sorts them for itself.
      unsigned long long v[2], upto[2], weight[2];
      const int many = gather_candidates(v, turn, sm);
      if (many > kCandidates) continue;
      sort_down(v, power_above(many), sm.candidates(turn ^ 1));
#pragma unroll
      for (int h = 0; h < 2; ++h) upto[h] = weight[h] = v[h] ? share.weight(key_value((uint32_t)(v[h] >> 32))) : 0;
      scan_both(upto, many, sm);
      int kept = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        kept += __syncthreads_count((int)threadIdx.x + h * kSampleThreads < many && above + upto[h] - weight[h] <= limit);
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if ((int)threadIdx.x + h * kSampleThreads == kept - 1)
          sm.keep = Keep{(uint32_t)(v[h] >> 32), (int)(0xffffffffu - (uint32_t)v[h])};
      __syncthreads();
      return sm.keep;
    }
    high_key -= (uint32_t)chosen << shift;
    if (shift == 0) break;
    const uint32_t width = (1u << shift) - 1;
    if (high_key - low_key > width) low_key = high_key - width;
  }
  const uint32_t beta = high_key;
  const float beta_value = key_value(beta);
  const unsigned long long each = unit ? 1ull : share.weight(beta_value);
  const unsigned long long count = each ? mass / each : 1ull;
  const unsigned long long ties = each ? min(count, (limit - above) / each + 1) : 1ull;   // above <= limit
  // (Where the cut falls on the value that `within` was cut at, that cut stays.)
  Keep out{beta, beta == within.beta ? within.tie_cut : vocab};
  if (ties < count) {
    // Not every element equal to beta survives: the index of the `ties`-th one, over the blocks in order.
    const int from = share.from, to = share.to;
    int mine = 0;
    for (int j = from; j < to; j += 32) {
      bool in = false;
      if (j + lane < to) {
        const int i = share.column(j + lane);
        const uint32_t key = ordered_key(share.value(i));
        in = key == beta && within.has(key, share.base + i);
      }
      mine += __popc(__ballot_sync(0xffffffffu, in));
    }
    if (lane == 0) sm.warp[w] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long all = 0;
      for (int k = 0; k < kSampleWarps; ++k) all += sm.warp[k];
      sm.exchange[slot] = all;
      sm.exchange[slot + 1] = (unsigned long long)vocab;
    }
    row_sync<kAlone>(cluster);
    unsigned long long before = 0;
    for (unsigned r = 0; r < cluster.block_rank(); ++r) before += *cluster.map_shared_rank(&sm.exchange[slot], r);
    for (int k = 0; k < w; ++k) before += sm.warp[k];
    if (before < ties && ties <= before + mine) {
      int left = (int)(ties - before);
      for (int j = from; j < to; j += 32) {
        int i = 0;
        bool in = false;
        if (j + lane < to) {
          i = share.column(j + lane);
          const uint32_t key = ordered_key(share.value(i));
          in = key == beta && within.has(key, share.base + i);
        }
        const unsigned votes = __ballot_sync(0xffffffffu, in);
        const int here = __popc(votes);
        if (left <= here) {
          if (in && __popc(votes & ((2u << lane) - 1)) == left) sm.exchange[slot + 1] = (unsigned long long)(share.base + i);
          break;
        }
        left -= here;
      }
    }
    row_sync<kAlone>(cluster);
    int cut = vocab;
    for (unsigned r = 0; r < cluster.num_blocks(); ++r) cut = min(cut, (int)*cluster.map_shared_rank(&sm.exchange[slot + 1], r));
    out.tie_cut = cut;
  }
  slot += 2;
  return out;
}

// What a row is sampled with.  A launch of few rows brings it along: no buffer to be pinned and no copy on the stream before
// the kernel (48 rows of 128,256 bfloat16 columns: 66 us a call behind a pinned copy, 55 with it, the time of the kernel).
constexpr int kBroughtAlong = 128;
struct RowParams {
  const float *temperature, *top_p, *uniform;      // on the device; null: the values below
  const int* top_k;
  bool along;
  float values[3][kBroughtAlong];                  // temperature, top_p, uniform
  int counts[kBroughtAlong];                       // top_k
};

// Grid: rows x (cluster size) blocks, a row's in one cluster.  `staged`: a block's share lies in its shared memory behind
// `sm`, as S: the logits as they are, or as float, divided by the temperature.
template <typename T, typename S, bool kAlone, bool kStaged>
__global__ void __launch_bounds__(kSampleThreads, sizeof(S) == 2 ? 3 : 2)
sample_kernel(const T* __restrict__ logits, int vocab, int share_size, const __grid_constant__ RowParams params,
              int* __restrict__ out) {
  extern __shared__ __align__(16) char sample_smem[];
  SampleSmem& sm = *reinterpret_cast<SampleSmem*>(sample_smem);
  S* stage = reinterpret_cast<S*>(sample_smem + (sizeof(SampleSmem) + 15) / 16 * 16);
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks(), r = blockIdx.x / ranks;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const T* row = logits + (size_t)r * vocab;
  const bool along = params.along;
  grid_dependency_wait();
  const float temp = along ? params.values[0][r] : params.temperature ? params.temperature[r] : 0.f;
  const int k = along ? params.counts[r] : params.top_k ? params.top_k[r] : -1;
  const float p = along ? params.values[1][r] : params.top_p ? params.top_p[r] : 1.f;
  const bool greedy = !(temp > 0.f) || k == 1;
  Share<S, kStaged> share;
  share.base = min(vocab, rank * share_size);
  share.n = min(vocab, share.base + share_size) - share.base;
  const T* mine_row = row + share.base;

  if constexpr (!kAlone) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");   // this block runs: its memory may be written
  const bool divide = temp != 1.f;
  ArgMax mine{-INFINITY, 0x7fffffff};
  constexpr int N = Vec16<T>::N;
  int done = 0;
  if (aligned16(mine_row)) {
    done = share.n / N * N;
#pragma unroll 4
    for (int i = threadIdx.x * N; i < done; i += kSampleThreads * N) {
      const Vec16<T> v = load16(mine_row + i);
      float f[N];
      unpack16(v, f);
      float most = f[0];
#pragma unroll
      for (int k = 1; k < N; ++k) most = fmaxf(most, f[k]);
      if (most > mine.v || mine.i == 0x7fffffff) {
#pragma unroll
        for (int k = 0; k < N; ++k) mine = better(mine, ArgMax{f[k], share.base + i + k});
      }
      if (kStaged && !greedy) {
        if constexpr (sizeof(S) == sizeof(T) && sizeof(T) == 2) {
          store16(reinterpret_cast<T*>(stage) + i, v);
        } else {
#pragma unroll
          for (int k = 0; k < N; k += 4) {
            Vec16<float> d;
#pragma unroll
            for (int e = 0; e < 4; ++e) d.set(e, divide ? f[k + e] / temp : f[k + e]);
            store16(reinterpret_cast<float*>(stage) + i + k, d);
          }
        }
      }
    }
  }
  for (int i = done + threadIdx.x; i < share.n; i += kSampleThreads) {
    const T v = mine_row[i];
    if (kStaged && !greedy) stage[i] = from_float<S>(sizeof(S) == 4 ? to_float(v) / temp : to_float(v));
    mine = better(mine, ArgMax{to_float(v), share.base + i});
  }
  const ArgMax block_top = block_argmax(mine, sm.warp_best);
  if constexpr (!kAlone) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (threadIdx.x < ranks) cluster.map_shared_rank(sm.best, threadIdx.x)[rank] = block_top;
  row_sync<kAlone>(cluster);
  ArgMax top = sm.best[0];
  for (int k = 1; k < ranks; ++k) top = better(top, sm.best[k]);

  if (greedy) {
    if (rank == 0 && threadIdx.x == 0) out[r] = top.i;
    return;                             // nothing of this block's is read any more
  }
  const int part_size = (share.n + 4 * kSampleWarps - 1) / (4 * kSampleWarps) * 4;
  share.from = min(share.n, w * part_size);
  share.to = min(share.n, share.from + part_size);
  share.listed = false;
  share.undivided = !(kStaged && sizeof(S) == 4) && temp != 1.f;
  share.wide = share_size >= 1 << 16;
  share.list = nullptr;
  share.temp = temp;
  share.row_max = top.v / temp;
  share.bin_max = share.undivided ? top.v : share.row_max;
  share.max_key = ordered_key(share.row_max);

  if constexpr (kStaged) share.data = stage;
  else share.data = mine_row;
  const bool by_count = k > 0 && k < vocab;
  double u = along ? (double)params.values[2][r] : params.uniform ? (double)params.uniform[r] : 0.5;
  u = u < 0.0 ? 0.0 : (u >= 1.0 ? 0.99999994 : u);
  int turn = 0, slot = 0, few = 0;
  Keep keep{0u, vocab};  // every finite value has a key > 0
  if (by_count) {
    share.bins_per_unit(kCountsPerUnit);
    keep = select_prefix<true, kAlone>(share, true, keep, (unsigned long long)(k - 1), p, vocab, turn, slot, few, sm);
    if (few) {
      if (rank == 0) {
        const int column = draw_from_candidates(share, k, p, u, top.i, turn, sm);
        if (threadIdx.x == 0) out[r] = column;
      }
      row_sync<kAlone>(cluster);        // the others' candidates stay until they have been read
      return;
    }
  }
  if (p > 0.f && p < 1.f) {
    share.bins_per_unit(kBinsPerUnit);
    keep = select_prefix<false, kAlone>(share, !by_count, keep, 0, p, vocab, turn, slot, few, sm);
  }

  // Draw: the first index (ascending) at which the running weight passes uniform * total.
  const int from = share.from, to = share.to;
  unsigned long long part = 0;
  const auto kept_weight = [&](float x, int i) { return keep.has(ordered_key(x), share.base + i) ? share.weight(x) : 0ull; };
  const auto four_weights = [&](int i, unsigned long long (&weight)[4]) {
    float f[4];
    share.four(i, f);
#pragma unroll
    for (int e = 0; e < 4; ++e) weight[e] = i + e < to ? kept_weight(share.quotient(f[e]), i + e) : 0;
  };
  if (share.listed) {
    for (int j = from + lane; j < to; j += 32) part += kept_weight(share.value(share.column(j)), share.column(j));
  } else {
#pragma unroll 2
    for (int j = from + 4 * lane; j < to; j += 128) {
      unsigned long long weight[4];
      four_weights(j, weight);
      part += weight[0] + weight[1] + weight[2] + weight[3];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  __syncthreads();
  if (lane == 0) sm.warp[w] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long all = 0;
    for (int i = 0; i < kSampleWarps; ++i) all += sm.warp[i];
    sm.exchange[slot] = all;
  }
  row_sync<kAlone>(cluster);
  unsigned long long before = 0, total = 0;
  for (int i = 0; i < ranks; ++i) {
    const unsigned long long v = *cluster.map_shared_rank(&sm.exchange[slot], i);
    if (i < rank) before += v;
    total += v;
  }
  for (int i = 0; i < w; ++i) before += sm.warp[i];
  unsigned long long target = (unsigned long long)(u * (double)total);
  if (target >= total) target = total ? total - 1 : 0;
  if (total == 0) {                      // the maximum weighs 2^32: only a row without finite values comes here
    if (rank == 0 && threadIdx.x == 0) out[r] = top.i;
  } else if (part > 0 && before <= target && target < before + part) {
    if (!share.listed) {
      for (int j = from; j < to; j += 128) {
        unsigned long long weight[4] = {0, 0, 0, 0};
        if (j + 4 * lane < to) four_weights(j + 4 * lane, weight);
        const unsigned long long mine = weight[0] + weight[1] + weight[2] + weight[3];
        unsigned long long upto = before + warp_inclusive(mine, lane);
        const unsigned passed = __ballot_sync(0xffffffffu, upto > target);
        if (passed) {
          if (lane == __ffs(passed) - 1) {
            upto -= mine;
            int e = 0;
#pragma unroll
            for (; e < 3; ++e) {
              upto += weight[e];
              if (upto > target) break;
            }
            out[r] = share.base + j + 4 * lane + e;
          }
          break;
        }
        before = __shfl_sync(0xffffffffu, upto, 31);
      }
    } else {
      for (int j = from; j < to; j += 32) {
        const int i = j + lane < to ? share.column(j + lane) : 0;
        const unsigned long long weight = j + lane < to ? kept_weight(share.value(i), i) : 0;
        const unsigned long long upto = before + warp_inclusive(weight, lane);
        const unsigned passed = __ballot_sync(0xffffffffu, upto > target);
        if (passed) {
          if (lane == __ffs(passed) - 1) out[r] = share.base + i;
          break;
        }
        before = __shfl_sync(0xffffffffu, upto, 31);
      }
    }
  }
  row_sync<kAlone>(cluster);            // nobody leaves while another block reads
}

template <typename T, typename S, bool kAlone, bool kStaged>
int launch_sample(const T* logits, int rows, int vocab, int ranks, int share, const RowParams& params, int* out,
                  cudaStream_t stream) {
  const size_t smem = (sizeof(SampleSmem) + 15) / 16 * 16 + (kStaged ? (size_t)share * sizeof(S) : 0);
  const cudaError_t status =
      cudaFuncSetAttribute(sample_kernel<T, S, kAlone, kStaged>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleMostSmem);
  if (status != cudaSuccess) return (int)status;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(rows * ranks);
  config.blockDim = dim3(kSampleThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = ranks;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = pdl_enabled(rows) ? 2 : 1;
  return (int)cudaLaunchKernelEx(&config, sample_kernel<T, S, kAlone, kStaged>, logits, vocab, share, params, out);
}

// Shares in shared memory where they fit.  bfloat16 is staged as divided floats while all of the launch's blocks are resident
// at once that way, two an SM (64 KB of floats beside 33 KB) or, of wide rows, one: the passes then divide nothing.  A wider launch stages the
// logits as they are, three blocks an SM, and divides again in the passes that need the quotient, so that 48 rows of
// 128,256 (384 blocks) still are one wave; two waves would cost each row's chain of barriers twice (24 rows of 151,936, top-k 50: 44 us, in one wave 30).
template <typename T>
int sample_rows(const T* logits, int rows, int vocab, const RowParams& params, int* out, cudaStream_t stream) {
  int ranks = 1;
  while (ranks < kMostRanks && ranks * kRankColumns < vocab) ranks *= 2;
  if (ranks > 1 && ranks < kMostRanks && 2LL * ranks * rows <= 148) ranks *= 2;
  const int share = ((vocab + ranks - 1) / ranks + 7) / 8 * 8;
  if ((long long)rows * ranks > 0x7fffffffll) return LI_ERR_UNSUPPORTED;
  const size_t fixed = (sizeof(SampleSmem) + 15) / 16 * 16, room = kSampleMostSmem - fixed;
  const bool two = 2 * (fixed + (size_t)share * 4 + kReservedSmem) <= kSmemOfSm;      // blocks of floats an SM
  const bool raw = (size_t)share * sizeof(T) <= room;
  const bool floats = sizeof(T) == 4 || ((size_t)share * 4 <= room / 2 && rows * ranks <= (two ? 2 : 1) * 148);
  const auto launch = [&](auto kernel) {
    return kernel(logits, rows, vocab, ranks, share, params, out, stream);
  };
  if (!raw) return launch(launch_sample<T, T, false, false>);
  if (ranks == 1) return floats ? launch(launch_sample<T, float, true, true>) : launch(launch_sample<T, T, true, true>);
  return floats ? launch(launch_sample<T, float, false, true>) : launch(launch_sample<T, T, false, true>);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
argmax_kernel(const T* __restrict__ logits, int vocab, int* __restrict__ out) {
  __shared__ ArgMax scratch[32];
  const T* row = logits + (size_t)blockIdx.x * vocab;
  ArgMax mine{-INFINITY, 0x7fffffff};
  for (int i = threadIdx.x; i < vocab; i += blockDim.x) mine = better(mine, ArgMax{to_float(row[i]), i});
  const ArgMax top = block_argmax(mine, scratch);
  if (threadIdx.x == 0) out[blockIdx.x] = top.i;
}

// A row split over gridDim.y blocks: each finds the best of its chunk and leaves it in scratch; the block
// that arrives last (a counter per row, reset by that block) picks the best of the chunks.
constexpr int kArgmaxThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kArgmaxThreads)
argmax_split_kernel(const T* __restrict__ logits, int vocab, int chunk, float* __restrict__ part_value,
                    int* __restrict__ part_index, unsigned* __restrict__ counters, int* __restrict__ out) {
  __shared__ ArgMax scratch[32];
  __shared__ bool is_last;
  const int r = blockIdx.x, c = blockIdx.y, chunks = gridDim.y;
  grid_launch_dependents();
  grid_dependency_wait();
  const T* row = logits + (size_t)r * vocab;
  const int lo = c * chunk, hi = min(vocab, lo + chunk);
  ArgMax mine{-INFINITY, 0x7fffffff};
  constexpr int N = Vec16<T>::N;
  if ((((size_t)r * vocab + lo) * sizeof(T)) % 16 == 0 && aligned16(logits)) {
    const int vec_hi = lo + (hi - lo) / N * N;
    for (int i = lo + threadIdx.x * N; i < vec_hi; i += kArgmaxThreads * N) {
      const Vec16<T> v = load16(row + i);
#pragma unroll
      for (int k = 0; k < N; ++k) mine = better(mine, ArgMax{v.get(k), i + k});
    }
    for (int i = vec_hi + threadIdx.x; i < hi; i += kArgmaxThreads) mine = better(mine, ArgMax{to_float(row[i]), i});
  } else {
    for (int i = lo + threadIdx.x; i < hi; i += kArgmaxThreads) mine = better(mine, ArgMax{to_float(row[i]), i});
  }
  const ArgMax top = block_argmax(mine, scratch);
  if (threadIdx.x == 0) {
    part_value[(size_t)r * chunks + c] = top.v;
    part_index[(size_t)r * chunks + c] = top.i;
    __threadfence();
    is_last = atomicAdd(&counters[r], 1u) == (unsigned)chunks - 1;
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  if (threadIdx.x == 0) {
    ArgMax best{-INFINITY, 0x7fffffff};
    for (int k = 0; k < chunks; ++k)
      best = better(best, ArgMax{__ldcg(part_value + (size_t)r * chunks + k), __ldcg(part_index + (size_t)r * chunks + k)});
    out[r] = best.i;
    counters[r] = 0;
  }
}

}  // namespace li

using namespace li;

// out[r] = index of the largest logit of row r (the lowest index among equals).
// With scratch (part_value/part_index of rows*32 entries, counters of `rows` zeros) a row is split over
// several blocks; without, one block scans a row.
LI_EXPORT int li_argmax(int dtype, const void* logits, int rows, int vocab, int* out, float* part_value,
                        int* part_index, unsigned* counters, int scratch_rows, cudaStream_t stream) {
  if (rows == 0) return 0;
  int chunks = (vocab + 4095) / 4096;
  if (chunks > 32) chunks = 32;
  if (chunks > 1 && part_value && part_index && counters && rows <= scratch_rows && rows <= 65535) {
    const int chunk = ((vocab + chunks - 1) / chunks + 7) / 8 * 8;
    const dim3 grid(rows, (vocab + chunk - 1) / chunk);
    if (dtype == kFloat32)
      return (int)launch_pdl(rows, argmax_split_kernel<float>, grid, dim3(kArgmaxThreads), 0, stream,
                             (const float*)logits, vocab, chunk, part_value, part_index, counters, out);
    return (int)launch_pdl(rows, argmax_split_kernel<bf16>, grid, dim3(kArgmaxThreads), 0, stream, (const bf16*)logits,
                           vocab, chunk, part_value, part_index, counters, out);
  }
  if (dtype == kFloat32)
    argmax_kernel<float><<<rows, kThreads, 0, stream>>>((const float*)logits, vocab, out);
  else
    argmax_kernel<bf16><<<rows, kThreads, 0, stream>>>((const bf16*)logits, vocab, out);
  LI_LAUNCH_CHECK();
}

// Per row: temperature (<= 0: arg-max), top_k (<= 0 or >= vocab: off), top_p (>= 1: off), uniform in [0, 1).
LI_EXPORT int li_sample(int dtype, const void* logits, int rows, int vocab, const float* temperature,
                        const int* top_k, const float* top_p, const float* uniform, int* out, cudaStream_t stream) {
  if (rows == 0) return 0;
  RowParams params = {};
  params.temperature = temperature;
  params.top_p = top_p;
  params.uniform = uniform;
  params.top_k = top_k;
  if (dtype == kFloat32) return sample_rows((const float*)logits, rows, vocab, params, out, stream);
  return sample_rows((const bf16*)logits, rows, vocab, params, out, stream);
}

// The same with the parameters in host memory, which is read before this returns; at most kBroughtAlong rows.
LI_EXPORT int li_sample_from_host(int dtype, const void* logits, int rows, int vocab, const float* temperature, const int* top_k,
                                  const float* top_p, const float* uniform, int* out, cudaStream_t stream) {
  if (rows == 0) return 0;
  if (rows > kBroughtAlong) return LI_ERR_UNSUPPORTED;
  RowParams params = {};
  params.along = true;
  for (int r = 0; r < rows; ++r) {
    params.values[0][r] = temperature[r];
    params.values[1][r] = top_p[r];
    params.values[2][r] = uniform[r];
    params.counts[r] = top_k[r];
  }
  if (dtype == kFloat32) return sample_rows((const float*)logits, rows, vocab, params, out, stream);
  return sample_rows((const bf16*)logits, rows, vocab, params, out, stream);
}
