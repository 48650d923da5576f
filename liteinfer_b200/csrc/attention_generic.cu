// Paged attention for any batch of (sequence, its newest queries), in plain SIMT
// code: the true 32-bit path, and the path for head sizes and types the tensor-core
// kernels refuse.  One kernel serves whole prompts, portions of prompts and single
// decoded tokens in the same launch; in 32-bit prompts and portions of more than a few tokens have
// a kernel of their own, and the single tokens beside them are a second launch.
//
// Rule (liteinfer/models/attention.py:24-27,81-84): a sequence's queries are the
// last `q_len` positions of its context of `ctx` tokens, so query j has position
// ctx - q_len + j and sees keys 0..position (with a window w: the newest w of
// them).  Query head h reads KV head h / groups (attention.py:69-78).  Scores,
// running maximum, sum and the output accumulator are 32-bit; the softmax is
// the online form (liteinfer/models/paged_kernels.py:216-288).
//
// Options: values of another size than keys (`v_dim`; out then has heads * v_dim columns); with a window, the
// first `keep_first` keys of a sequence stay visible behind it (they are walked first, then the window's keys);
// `softcap` > 0 turns a scaled score s into softcap * tanh(s / softcap) before the softmax; `sink` [heads]
// (float, optional): exp(sink[h]) is one more term of head h's denominator, with no key and no value.
//
// Work split: block = (query tile, KV head, sequence).  A row (query, head-in-group) walks its keys in units of 32 that
// start at multiples of 32, each with a softmax of its own; the units' results are merged in ascending order.  So the order of every sum depends on the row's position only, never on how the batch was cut
// or on who walks a unit: where a block has more rows than warps each warp takes rows in turn and walks all of a row's
// units; where it has fewer (decode) a row belongs to a team of warps, which walk a unit each and meet for the merge.
// Masked keys are not read at all: a page that was never written, or holds another request's tokens, cannot leak
// through a NaN or a stale value.
//
// Bound by the latency of a unit's loads: a lane asks for 64 numbers of its key at once in 16-byte pieces, and for 32 of the
// values' numbers, without a branch between the loads.  Measured on B200 (float32, 12 heads
// on 4, head size 64, a decode step of 12 sequences of 19 to 190): 9 us, against 238 when a warp walked all of a row's keys one load
// after another.
#include "common.cuh"

namespace li {

constexpr int kMaxKeyDim = 1024;
constexpr int kQueriesPerBlock = 8;
constexpr int kUnit = 32;
constexpr int kMostWarps = 16;
constexpr int kSms = 148;

template <typename T>
struct GenericParams {
  const T* q;
  T* out;
  const T *k_pool, *v_pool;
  const int *block_table, *query_start_loc, *context_lens;
  const float* sink;
  int q_row_stride, out_row_stride, table_stride, heads, kv_heads, head_dim, v_dim, page_size, num_pages;
  int window, keep_first;
  float scale, softcap;
  bool vec;      // keys lie on 16 bytes and are a multiple of them long
  bool row_blocks;   // single tokens: a block has one row (blockIdx.x is the head in its group)
  bool only_single;  // sequences that bring more than one token are another launch's
};

// What a walk over keys has so far: the maximum, the sum and the weighted values (lane + 32 i of them in acc[i]).
template <int kDimsPerLane>
struct SoftmaxState {
  float m, l, acc[kDimsPerLane];
  __device__ __forceinline__ void reset() {
    m = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int i = 0; i < kDimsPerLane; ++i) acc[i] = 0.f;
  }
  __device__ __forceinline__ void merge(const SoftmaxState& o) {
    if (o.m == -INFINITY) return;
    if (m == -INFINITY) {
      *this = o;
      return;
    }
    const float top = fmaxf(m, o.m), a = expf(m - top), b = expf(o.m - top);
    m = top;
    l = l * a + o.l * b;
#pragma unroll
    for (int i = 0; i < kDimsPerLane; ++i) acc[i] = acc[i] * a + o.acc[i] * b;
  }
};

// The score of this lane's key: q in shared memory, one accumulator, ascending dimensions.
template <typename T>
__device__ __forceinline__ float key_score(const float* qs, const T* kp, int head_dim, bool vec) {
  float dot = 0.f;
  if (vec) {
    constexpr int N = Vec16<T>::N, kAhead = 64 / N;
    const float4* q4 = reinterpret_cast<const float4*>(qs);
    const int pieces = head_dim / N;
    for (int c = 0; c < pieces; c += kAhead) {
      Vec16<T> v[kAhead];
#pragma unroll
      for (int e = 0; e < kAhead; ++e) v[e] = load16(kp + min(c + e, pieces - 1) * N);      // no branch between the loads
#pragma unroll
      for (int e = 0; e < kAhead; ++e) {
        if (c + e < pieces) {
          float f[N];
          unpack16(v[e], f);
#pragma unroll
          for (int d = 0; d < N; d += 4) {
            const float4 q = q4[((c + e) * N + d) / 4];
            dot += q.x * f[d];
            dot += q.y * f[d + 1];
            dot += q.z * f[d + 2];
            dot += q.w * f[d + 3];
          }
        }
      }
    }
    return dot;
  }
  for (int d = 0; d < head_dim; ++d) dot += qs[d] * to_float(kp[d]);
  return dot;
}

// One unit: the keys lo..hi (inclusive, within one multiple of kUnit) of the row whose query lies in `qs`.
template <typename T, int kDimsPerLane>
__device__ __forceinline__ void walk_unit(const GenericParams<T>& p, const float* qs, const int* table, int kvh, int lo, int hi,
                                          SoftmaxState<kDimsPerLane>& s) {
  const int lane = threadIdx.x & 31;
  s.reset();
  for (int base = lo / 32 * 32; base <= hi; base += 32) {
    const int kpos = base + lane;
    int krow = -1;  // row index of this lane's key inside the pool: (page * kv_heads + kvh) * page_size + slot
    float score = -INFINITY;
    if (kpos >= lo && kpos <= hi) {
      const int page = table[kpos / p.page_size];
      if (page >= 0 && page < p.num_pages) {
        krow = (page * p.kv_heads + kvh) * p.page_size + kpos % p.page_size;
        score = key_score(qs, p.k_pool + (size_t)krow * p.head_dim, p.head_dim, p.vec) * p.scale;
        if (p.softcap > 0.f) score = p.softcap * tanhf(score / p.softcap);
      }
    }
    const float m_new = fmaxf(s.m, warp_max(score));
    if (m_new == -INFINITY) continue;  // nothing visible in this chunk
    const float prob = krow >= 0 ? expf(score - m_new) : 0.f;
    const float alpha = expf(s.m - m_new);  // m = -inf on the first chunk gives 0
    s.l = s.l * alpha + warp_sum(prob);
#pragma unroll
    for (int i = 0; i < kDimsPerLane; ++i) s.acc[i] *= alpha;
    // The probability is rounded to the value type before P.V (paged_kernels.py:282-284).
    const float p_store = round_to<T>(prob);
    const unsigned live = __ballot_sync(0xffffffffu, krow >= 0);
    constexpr int kAhead = kDimsPerLane <= 16 ? 32 / kDimsPerLane : 2;
    for (int j0 = 0; j0 < 32; j0 += kAhead) {
      if (!(live >> j0 & ((1u << kAhead) - 1))) continue;
      T v[kAhead][kDimsPerLane];
      float pj[kAhead];
      // No branch between the loads: a place without a key reads the pool's first row and drops it.
#pragma unroll
      for (int e = 0; e < kAhead; ++e) {
        pj[e] = __shfl_sync(0xffffffffu, p_store, j0 + e);
        const int vr = __shfl_sync(0xffffffffu, krow, j0 + e);
        const T* vp = p.v_pool + (size_t)max(vr, 0) * p.v_dim;
#pragma unroll
        for (int i = 0; i < kDimsPerLane; ++i) v[e][i] = vp[min(lane + 32 * i, p.v_dim - 1)];
      }
#pragma unroll
      for (int e = 0; e < kAhead; ++e) {
        if (live >> (j0 + e) & 1) {
#pragma unroll
          for (int i = 0; i < kDimsPerLane; ++i) s.acc[i] += pj[e] * to_float(v[e][i]);
        }
      }
    }
    s.m = m_new;
  }
}

// kDimsPerLane: a lane keeps this many of a value's dimensions, so values have at most 32 times as many.
// Shared memory: a query per warp, then, for teams, a unit's result per warp.
template <typename T, int kDimsPerLane>
__global__ void __launch_bounds__(kDimsPerLane <= 8 ? 32 * kMostWarps : 256, 1)
paged_attention_generic_kernel(const GenericParams<T> p) {
  extern __shared__ __align__(16) float q_smem[];
  grid_launch_dependents();       // (what follows may be a product that asks for its weights first)
  grid_dependency_wait();
  const int seq = blockIdx.z, kvh = blockIdx.y;
  const int q_begin = p.query_start_loc[seq], q_len = p.query_start_loc[seq + 1] - q_begin;
  const int tile_start = p.row_blocks ? 0 : blockIdx.x * kQueriesPerBlock;
  if (tile_start >= q_len || (p.only_single && q_len > 1)) return;
  const int ctx = p.context_lens[seq];
  const int groups = p.heads / p.kv_heads;
  const int tile_q = min(kQueriesPerBlock, q_len - tile_start);
  const int first_row = p.row_blocks ? blockIdx.x : 0, rows = p.row_blocks ? 1 : tile_q * groups;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int q_stride = (p.head_dim + 3) / 4 * 4;
  float* qs = q_smem + warp * q_stride;
  float* results = q_smem + nwarps * q_stride;       // [warp][2 + 32 * kDimsPerLane]
  constexpr int kResult = 2 + 32 * kDimsPerLane;
  const int* table = p.block_table + (size_t)seq * p.table_stride;
  const int team = max(1, nwarps / rows), teams = nwarps / team, member = warp % team;
  // The most units of any row of the tile: the first tokens that stay visible, then those from the first query's first key.
  const int first_q = ctx - q_len + tile_start, last_q = first_q + tile_q - 1;
  const int tile_first = first_visible(first_q, p.window);
  const int tile_kept = (p.window > 0 && p.keep_first > 0) ? min(p.keep_first, first_visible(last_q, p.window)) : 0;
  const int most_units = (tile_kept + kUnit - 1) / kUnit + last_q / kUnit - tile_first / kUnit + 1;
  // A team has one row, and every warp of the block takes part in its barriers.
  for (int row = warp / team; team > 1 ? row == warp / team : row < rows; row += teams) {
    const bool real = row < rows && warp < teams * team;
    const int qi = tile_start + (real ? (first_row + row) / groups : 0);          // query index within the sequence's queries
    const int head = kvh * groups + (real ? (first_row + row) % groups : 0);
    const int qpos = ctx - q_len + qi;                 // absolute position of this query
    __syncwarp();
    if (real) {
      const T* qrow = p.q + (size_t)(q_begin + qi) * p.q_row_stride + (size_t)head * p.head_dim;
      for (int d = lane; d < p.head_dim; d += 32) qs[d] = to_float(qrow[d]);
    }
    __syncwarp();

    // Two runs of keys: the first tokens that stay visible behind the window, then the window itself.
    const int first = first_visible(qpos, p.window);
    const int kept_end = (p.window > 0 && p.keep_first > 0) ? min(p.keep_first, first) : 0;
    const int kept_units = (kept_end + kUnit - 1) / kUnit, units = kept_units + qpos / kUnit - first / kUnit + 1;
    SoftmaxState<kDimsPerLane> run, mine;
    run.reset();
    for (int u0 = 0; u0 < (team > 1 ? most_units : units); u0 += team) {
      const int u = u0 + member;
      mine.reset();
      if (real && u < units) {
        const bool kept = u < kept_units;
        const int base = kept ? u * kUnit : (first / kUnit + u - kept_units) * kUnit;
        walk_unit<T, kDimsPerLane>(p, qs, table, kvh, max(base, kept ? 0 : first),
                                   min(base + kUnit - 1, kept ? kept_end - 1 : qpos), mine);
      }
      if (team == 1) {
        run.merge(mine);
        continue;
      }
      float* result = results + warp * kResult;
      if (lane == 0) result[0] = mine.m, result[1] = mine.l;
#pragma unroll
      for (int i = 0; i < kDimsPerLane; ++i) result[2 + lane + 32 * i] = mine.acc[i];
      __syncthreads();
      if (member == 0 && real) {
        for (int t = 0; t < team && u0 + t < units; ++t) {
          const float* other = result + t * kResult;
          mine.m = other[0], mine.l = other[1];
#pragma unroll
          for (int i = 0; i < kDimsPerLane; ++i) mine.acc[i] = other[2 + lane + 32 * i];
          run.merge(mine);
        }
      }
      __syncthreads();
    }
    if (member != 0 || !real) continue;
    if (p.sink != nullptr) {      // one more term of the denominator: it has no key, no value, and is not scaled
      const float sk = p.sink[head];
      const float m_new = fmaxf(run.m, sk);
      const float alpha = expf(run.m - m_new);
      run.l = run.l * alpha + expf(sk - m_new);
#pragma unroll
      for (int i = 0; i < kDimsPerLane; ++i) run.acc[i] *= alpha;
    }
    T* orow = p.out + (size_t)(q_begin + qi) * p.out_row_stride + (size_t)head * p.v_dim;
    const float inv = run.l > 0.f ? 1.0f / run.l : 0.f;
#pragma unroll
    for (int i = 0; i < kDimsPerLane; ++i) {
      const int d = lane + 32 * i;
      if (d < p.v_dim) orow[d] = from_float<T>(run.acc[i] * inv);
    }
  }
}

// ---- prompts and portions in 32-bit: a block's queries share its units of keys ---------------------------------------
// The kernel above fetches a unit of keys for every row anew, each lane its own key: 32 lines a load instruction, so a row's unit takes the
// loads some 600 cycles.  Here a block of eight queries (all heads of a KV head's group) copies a unit's keys and values to shared memory
// once (cp.async, the next unit on its way meanwhile), a warp has one query and takes the scores of its rows together.  Bound by
// shared memory's reads, 16 bytes a lane of key and of every row's query.  The sums are those of the kernel above, in its order, to the
// bit.  For 32-bit numbers, head sizes of whole 16 bytes up to 128, groups of up to eight heads; single tokens stay above, where a
// row's units are walked side by side.
// Measured on B200, 12 prompts of 19 to 190 tokens, 12 heads on 4, head size 64: 50 us (136).
constexpr int kPromptWarps = kQueriesPerBlock, kPromptMostDim = 128, kPromptMostRows = 8;

__host__ __device__ constexpr int padded_row(int dim) { return dim + 4; }      // 16-byte reads of 32 rows: off the banks' period
inline size_t prompt_smem(int groups, int head_dim, int v_dim) {
  return sizeof(float) * ((size_t)kPromptWarps * groups * head_dim + 2 * (size_t)kUnit * (padded_row(head_dim) + v_dim + 1));
}

template <int kDimsPerLane, int kRows>
__global__ void __launch_bounds__(32 * kPromptWarps) prompt_attention_kernel(const GenericParams<float> p) {
  extern __shared__ __align__(16) float prompt_smem_raw[];
  grid_launch_dependents();
  grid_dependency_wait();
  const int seq = blockIdx.z, kvh = blockIdx.y, tile_start = blockIdx.x * kQueriesPerBlock;
  const int q_begin = p.query_start_loc[seq], q_len = p.query_start_loc[seq + 1] - q_begin;
  if (q_len <= 1 || tile_start >= q_len) return;
  const int ctx = p.context_lens[seq], groups = p.heads / p.kv_heads, tile_q = min(kQueriesPerBlock, q_len - tile_start);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int key_row = padded_row(p.head_dim);
  float* qs = prompt_smem_raw + warp * groups * p.head_dim;
  float* keys = prompt_smem_raw + kPromptWarps * groups * p.head_dim;        // [stage][key][key_row]
  float* values = keys + 2 * kUnit * key_row;                                // [stage][key][v_dim]
  int* present = reinterpret_cast<int*>(values + 2 * kUnit * p.v_dim);       // [stage][key]: whether the key's page exists
  const int* table = p.block_table + (size_t)seq * p.table_stride;

  const int qi = tile_start + min(warp, tile_q - 1);
  const bool real = warp < tile_q;
  const int qpos = ctx - q_len + qi, first = first_visible(qpos, p.window);
  const int kept_end = (p.window > 0 && p.keep_first > 0) ? min(p.keep_first, first) : 0;
  {
    const float* q = p.q + (size_t)(q_begin + qi) * p.q_row_stride + (size_t)kvh * groups * p.head_dim;
    for (int d = lane; d < groups * p.head_dim; d += 32) qs[d] = q[d];
  }
  // The block's units: those of the first tokens that stay visible behind the last query's window, then from the first query's first key.
  const int first_q = ctx - q_len + tile_start, last_q = first_q + tile_q - 1;
  const int tile_kept = (p.window > 0 && p.keep_first > 0) ? min(p.keep_first, first_visible(last_q, p.window)) : 0;
  const int kept_units = (tile_kept + kUnit - 1) / kUnit, from_unit = first_visible(first_q, p.window) / kUnit;
  const int units = kept_units + last_q / kUnit - from_unit + 1;
  const auto base_of = [&](int u) { return (u < kept_units ? u : from_unit + u - kept_units) * kUnit; };
  const int key = threadIdx.x >> 3, eighth = threadIdx.x & 7;      // eight threads copy a key
  const auto fetch = [&](int u) {
    if (u < units) {
      const int kpos = base_of(u) + key, stage = u & 1;
      int row = -1;
      if (kpos <= last_q) {
        const int page = table[kpos / p.page_size];
        if (page >= 0 && page < p.num_pages) row = (page * p.kv_heads + kvh) * p.page_size + kpos % p.page_size;
      }
      if (eighth == 0) present[stage * kUnit + key] = row >= 0;
      if (row >= 0) {
        const auto copy = [](float* dst, const float* src) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
        };
        for (int d = eighth * 4; d < p.head_dim; d += 32)
          copy(keys + (stage * kUnit + key) * key_row + d, p.k_pool + (size_t)row * p.head_dim + d);
        for (int d = eighth * 4; d < p.v_dim; d += 32)
          copy(values + (stage * kUnit + key) * p.v_dim + d, p.v_pool + (size_t)row * p.v_dim + d);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  SoftmaxState<kDimsPerLane> run[kRows];
#pragma unroll
  for (int g = 0; g < kRows; ++g) run[g].reset();
  fetch(0);
  for (int u = 0; u < units; ++u) {
    fetch(u + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const bool kept = u < kept_units;
    const int base = base_of(u), stage = u & 1, kpos = base + lane;
    const int lo = max(base, kept ? 0 : first), hi = min(base + kUnit - 1, kept ? kept_end - 1 : qpos);
    if (real && lo <= hi) {
      const float4* k4 = reinterpret_cast<const float4*>(keys + (stage * kUnit + lane) * key_row);
      float dot[kRows];
#pragma unroll
      for (int g = 0; g < kRows; ++g) dot[g] = 0.f;
#pragma unroll 4
      for (int c = 0; c < p.head_dim / 4; ++c) {
        const float4 f = k4[c];
#pragma unroll
        for (int g = 0; g < kRows; ++g) {
          if (g >= groups) break;
          const float4 q = reinterpret_cast<const float4*>(qs + g * p.head_dim)[c];
          dot[g] += q.x * f.x;
          dot[g] += q.y * f.y;
          dot[g] += q.z * f.z;
          dot[g] += q.w * f.w;
        }
      }
      const bool live_key = kpos >= lo && kpos <= hi && present[stage * kUnit + lane] != 0;
      const unsigned live = __ballot_sync(0xffffffffu, live_key);
      SoftmaxState<kDimsPerLane> mine[kRows];
      float prob[kRows];
#pragma unroll
      for (int g = 0; g < kRows; ++g) {
        float score = -INFINITY;
        if (live_key) {
          score = dot[g] * p.scale;
          if (p.softcap > 0.f) score = p.softcap * tanhf(score / p.softcap);
        }
        mine[g].reset();
        const float m = warp_max(score);
        prob[g] = live_key && m != -INFINITY ? expf(score - m) : 0.f;
        mine[g].m = m;
        mine[g].l = warp_sum(prob[g]);
      }
#pragma unroll 4
      for (int j = 0; j < kUnit; ++j) {
        if (!(live >> j & 1)) continue;
        float v[kDimsPerLane];
#pragma unroll
        for (int i = 0; i < kDimsPerLane; ++i) v[i] = values[(stage * kUnit + j) * p.v_dim + min(lane + 32 * i, p.v_dim - 1)];
#pragma unroll
        for (int g = 0; g < kRows; ++g) {
          const float pj = __shfl_sync(0xffffffffu, prob[g], j);
#pragma unroll
          for (int i = 0; i < kDimsPerLane; ++i) mine[g].acc[i] += pj * v[i];
        }
      }
#pragma unroll
      for (int g = 0; g < kRows; ++g)
        if (g < groups) run[g].merge(mine[g]);
    }
    __syncthreads();        // the stage is written again with the next fetch
  }
  if (!real) return;
#pragma unroll
  for (int g = 0; g < kRows; ++g) {
    if (g >= groups) break;
    SoftmaxState<kDimsPerLane>& row = run[g];
    const int head = kvh * groups + g;
    if (p.sink != nullptr) {      // one more term of the denominator: it has no key, no value, and is not scaled
      const float sk = p.sink[head], m_new = fmaxf(row.m, sk), alpha = expf(row.m - m_new);
      row.l = row.l * alpha + expf(sk - m_new);
#pragma unroll
      for (int i = 0; i < kDimsPerLane; ++i) row.acc[i] *= alpha;
    }
    float* out = p.out + (size_t)(q_begin + qi) * p.out_row_stride + (size_t)head * p.v_dim;
    const float inv = row.l > 0.f ? 1.0f / row.l : 0.f;
#pragma unroll
    for (int i = 0; i < kDimsPerLane; ++i)
      if (lane + 32 * i < p.v_dim) out[lane + 32 * i] = row.acc[i] * inv;
  }
}

// Whether the portions of a launch bring so few queries that the kernel above is the faster for them: it gives a row's units to several warps,
// where this one has a warp a query, whatever stays idle.  Behind 1,500 keys, microseconds, teams and shared keys: 4 heads on 4 of 64, two
// queries 53 and 137, five 116 and 140, six 148 and 140; 8 on 4, three 148 and 186, four 193 and 186; 12 on 4, two 148 and 255, three
// 308 and 254; 8 on 1, two 376 and 433; of 128, 16 on 16, three 127 and 168, four 169 and 169; 8 on 4, three 254 and 280; 16 on 4, two 351 and
// 350; 16 on 2, two 696 and 580; of 100, 4 on 4, six 171 and 183.  Within one unit of keys groups of one or two heads are
// faster shared (3 queries of 4 heads on 4 of 64: 4.5 and 3.6), wide ones by teams (2 of 16 on 2 of 128 8.5 and 13.0).
inline bool few_queries(int queries, int groups, int head_dim, int v_dim, int max_context) {
  if (max_context > 0 && max_context <= kUnit) return groups > 4 ? queries <= 3 : groups > 2 && queries == 2;
  const bool narrow = v_dim <= 64;
  if (groups == 1) return queries <= (narrow ? 5 : head_dim <= 100 ? 6 : 3);
  if (groups == 2) return queries <= 3;
  return queries == 2 && (narrow || groups <= 4);
}

template <int kDimsPerLane, int kRows>
int launch_prompt(dim3 grid, const GenericParams<float>& p, cudaStream_t stream) {
  const size_t smem = prompt_smem(p.heads / p.kv_heads, p.head_dim, p.v_dim);
  if (smem > 48 * 1024) {
    const cudaError_t status = cudaFuncSetAttribute(prompt_attention_kernel<kDimsPerLane, kRows>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (status != cudaSuccess) return (int)status;
  }
  return (int)launch_pdl(0, prompt_attention_kernel<kDimsPerLane, kRows>, grid, dim3(32 * kPromptWarps), smem, stream, p);
}

template <int kDimsPerLane>
int launch_prompt(dim3 grid, const GenericParams<float>& p, cudaStream_t stream) {
  const int groups = p.heads / p.kv_heads;
  if (groups == 1) return launch_prompt<kDimsPerLane, 1>(grid, p, stream);
  if (groups == 2) return launch_prompt<kDimsPerLane, 2>(grid, p, stream);
  if (groups == 3) return launch_prompt<kDimsPerLane, 3>(grid, p, stream);
  if (groups == 4) return launch_prompt<kDimsPerLane, 4>(grid, p, stream);
  return launch_prompt<kDimsPerLane, 8>(grid, p, stream);
}

template <typename T, int kDimsPerLane>
int launch_generic(dim3 grid, int threads, const GenericParams<T>& p, cudaStream_t stream) {
  const size_t smem = (size_t)(threads / 32) * ((p.head_dim + 3) / 4 * 4 + 2 + 32 * kDimsPerLane) * sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t status = cudaFuncSetAttribute(paged_attention_generic_kernel<T, kDimsPerLane>,
                                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (status != cudaSuccess) return (int)status;
  }
  return (int)launch_pdl(0, paged_attention_generic_kernel<T, kDimsPerLane>, grid, dim3(threads), smem, stream, p);
}

template <typename T>
int launch_generic(dim3 grid, int threads, const GenericParams<T>& p, cudaStream_t stream) {
  if (p.v_dim <= 64) return launch_generic<T, 2>(grid, threads, p, stream);
  if (p.v_dim <= 128) return launch_generic<T, 4>(grid, threads, p, stream);
  if (p.v_dim <= 256) return launch_generic<T, 8>(grid, threads, p, stream);
  return launch_generic<T, 32>(grid, threads, p, stream);
}

template <typename T>
GenericParams<T> typed(const void* q, void* out, const void* k_pool, const void* v_pool) {
  GenericParams<T> p = {};
  p.q = (const T*)q, p.out = (T*)out, p.k_pool = (const T*)k_pool, p.v_pool = (const T*)v_pool;
  return p;
}

}  // namespace li

using namespace li;

// q: [tokens, q_row_stride] with head h of a token at columns [h*head_dim, (h+1)*head_dim).
// out: [tokens, out_row_stride] with head h at columns [h*v_dim, (h+1)*v_dim).  k_pool: [num_pages, kv_heads,
// page_size, head_dim]; v_pool likewise with v_dim.  window: see first_visible (common.cuh).  sink: null or [heads].
// single_tokens: whether sequences may bring one token beside others that bring more.  max_context (0: not known): the most tokens that a
// sequence which brings more than one holds.
LI_EXPORT int li_paged_attention_generic(int dtype, const void* q, int q_row_stride, void* out, int out_row_stride,
                                         const void* k_pool, const void* v_pool, const int* block_table,
                                         int table_stride, const int* query_start_loc, const int* context_lens,
                                         int num_seqs, int max_q_len, int heads, int kv_heads, int head_dim,
                                         int v_dim, int page_size, int num_pages, float scale, int window,
                                         int keep_first, float softcap, const float* sink, int single_tokens, int max_context,
                                         cudaStream_t stream) {
  if (num_seqs == 0 || max_q_len == 0) return 0;
  if (head_dim < 1 || head_dim > kMaxKeyDim || kv_heads < 1 || heads % kv_heads) return LI_ERR_UNSUPPORTED;
  if (v_dim < 1 || v_dim > 32 * 32) return LI_ERR_UNSUPPORTED;
  if (kv_heads > 65535 || num_seqs > 65535) return LI_ERR_UNSUPPORTED;
  const int groups = heads / kv_heads;
  int max_q = max_q_len;
  const bool only_single = max_q_len > 1 && dtype == kFloat32 && head_dim % 4 == 0 && v_dim % 4 == 0 && head_dim <= kPromptMostDim &&
                           v_dim <= kPromptMostDim && groups <= kPromptMostRows && aligned16(k_pool) && aligned16(v_pool) &&
                           !few_queries(max_q_len, groups, head_dim, v_dim, max_context);
  if (only_single) {
    // Prompts and portions by the kernel whose queries share their keys; the single tokens beside them, if any, behind it.
    GenericParams<float> p = typed<float>(q, out, k_pool, v_pool);
    p.block_table = block_table, p.query_start_loc = query_start_loc, p.context_lens = context_lens, p.sink = sink;
    p.q_row_stride = q_row_stride, p.out_row_stride = out_row_stride, p.table_stride = table_stride;
    p.heads = heads, p.kv_heads = kv_heads, p.head_dim = head_dim, p.v_dim = v_dim;
    p.page_size = page_size, p.num_pages = num_pages, p.window = window, p.keep_first = keep_first;
    p.scale = scale, p.softcap = softcap;
    const dim3 grid((max_q_len + kQueriesPerBlock - 1) / kQueriesPerBlock, kv_heads, num_seqs);
    const int status = v_dim <= 64 ? launch_prompt<2>(grid, p, stream) : launch_prompt<4>(grid, p, stream);
    if (status != 0 || !single_tokens) return status;
    max_q = 1;
  }
  // Single tokens of few sequences: a block for every row, whose warps then walk many units at once (12 sequences of 19 to 190
  // keys, 12 heads on 4: 9.2 us a launch, 12.9 with the three rows of a KV head in a block; 64 sequences of 500, whose keys
  // every row's block would fetch again: 72 and 52).
  const bool row_blocks = max_q == 1 && groups > 1 && (long)num_seqs * heads <= 2 * kSms;
  const int rows = row_blocks ? 1 : (max_q < kQueriesPerBlock ? max_q : kQueriesPerBlock) * groups;
  const dim3 grid(row_blocks ? groups : (max_q + kQueriesPerBlock - 1) / kQueriesPerBlock, kv_heads, num_seqs);
  // Few rows a block (decode): as many warps share a row's units as keep an SM busy with the blocks that it gets.  Sixteen warps
  // for every block, however many there are, had most of them wait at the barriers of rows of a unit or two: 256
  // sequences of 16 keys at 16 heads took 120 us (55 with a warp a row; now 22), of 500 keys 383 (248), while 8 sequences of
  // 1,500 keys take 37 us with sixteen warps, 53 with eight and 69 with four.
  const long blocks = (long)grid.x * grid.y * grid.z;
  const int warps = blocks <= kSms ? kMostWarps : blocks <= 2 * kSms ? kMostWarps / 2 : blocks <= 4 * kSms ? kMostWarps / 4 : kMostWarps / 8;
  const int threads = rows >= 8 ? 256 : 32 * (v_dim > 256 && warps > 8 ? 8 : warps);
  const auto run = [&](auto p) {
    p.block_table = block_table, p.query_start_loc = query_start_loc, p.context_lens = context_lens, p.sink = sink;
    p.q_row_stride = q_row_stride, p.out_row_stride = out_row_stride, p.table_stride = table_stride;
    p.heads = heads, p.kv_heads = kv_heads, p.head_dim = head_dim, p.v_dim = v_dim;
    p.page_size = page_size, p.num_pages = num_pages, p.window = window, p.keep_first = keep_first;
    p.scale = scale, p.softcap = softcap, p.row_blocks = row_blocks, p.only_single = only_single;
    p.vec = aligned16(k_pool) && (size_t)head_dim * sizeof(*p.k_pool) % 16 == 0;
    return launch_generic(grid, threads, p, stream);
  };
  if (dtype == kFloat32) return run(typed<float>(q, out, k_pool, v_pool));
  return run(typed<bf16>(q, out, k_pool, v_pool));
}
