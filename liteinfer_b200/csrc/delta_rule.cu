// The gated delta rule and the short convolutions in front of it.
//
//   li_short_conv         y[t, c] = act(b[c] + sum_m w[m, c] * x[t - (K-1-m), c]), b optional: a causal convolution over
//                         time per channel (the taps tap by tap, [K, channels], so that neighbouring channels' weights are
//                         neighbours); inputs before the step come from the request's tail (its last K-1 inputs)
//   li_short_conv_update  moves every request's tail on by the step's inputs
//   li_gated_delta_rule   per request and head a state S [dim, vdim] in 32-bit (kept column by column); per token
//                             S *= g;  u = beta * (v - S^T k);  S += k u^T;  o = S^T q
//                         with q, k made unit vectors (q also times dim^-0.5), beta = sigmoid(raw),
//                         g = exp(-exp(A_log) * softplus(raw + dt_bias))
//
// The recurrence is a chain over the tokens of a sequence, but every column of S is a chain of its own:
// (S^T k)_j, u_j, the update of S[:, j] and o_j touch column j only.  So a block takes 16 or 32 columns of one head of
// one sequence, eight lanes share a column (each keeps dim/8 of its entries in registers for the whole step) and
// add up their parts of the dot products with shuffles.  What does not depend on the state (the unit
// norms, beta, the decay) is computed once per token and head by a kernel in front; the inputs of the next few
// tokens are in flight while one is computed.  Prompts, portions and single tokens go on from the state that the step
// before left.  Heads of 32, 64 and 128 go two tokens at a time, paired from where the step's portion of a sequence
// begins: a cut at an odd place pairs other tokens, which rounds differently (in 32-bit, 1e-7 or so of the
// result), and so does a single token, which is a portion of one beside prompts and another kernel's in a step of
// its like.  Other heads go a token at a time, in one order however a sequence was cut.  Which other sequences a launch
// has changes no bit.  Tokens of padding (sequence -1) and sequences that bring no token touch nothing.
#include <type_traits>

#include "common.cuh"

namespace li {

constexpr int kMaxTaps = 16;

template <typename T>
__global__ void short_conv_kernel(const T* __restrict__ x, size_t x_stride, const T* __restrict__ taps,
                                  const T* __restrict__ tail, const int* __restrict__ seq_of_token,
                                  const int* __restrict__ query_start_loc, const int* __restrict__ state_slots,
                                  T* __restrict__ out, int channels, int K, int act, const float* __restrict__ bias) {
  grid_dependency_wait();
  const int t = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  const int seq = seq_of_token[t];
  if (seq < 0) {
    out[(size_t)t * channels + c] = from_float<T>(0.f);
    return;
  }
  const int j = t - query_start_loc[seq];   // index of the token among its sequence's tokens of this step
  const T* old = tail + (size_t)state_slots[seq] * (K - 1) * channels;
  float acc = bias != nullptr ? bias[c] : 0.f;
  for (int m = 0; m < K; ++m) {
    const int back = K - 1 - m;
    const float in = back <= j ? to_float(x[(size_t)(t - back) * x_stride + c])
                               : to_float(old[(size_t)(K - 1 + j - back) * channels + c]);
    acc = fmaf(to_float(taps[(size_t)m * channels + c]), in, acc);
  }
  if (act) acc = acc / (1.0f + expf(-acc));
  out[(size_t)t * channels + c] = from_float<T>(acc);
}

// The same, a 16-byte vector of neighbouring channels a thread (channels and row strides multiples of the
// vector's length, 16-byte aligned pointers).
template <typename T>
__global__ void short_conv_vec_kernel(const T* __restrict__ x, size_t x_stride, const T* __restrict__ taps,
                                      const T* tail, const int* __restrict__ seq_of_token,
                                      const int* __restrict__ query_start_loc, const int* __restrict__ state_slots,
                                      T* __restrict__ out, int channels, int K, int act, T* move_tail,
                                      const float* __restrict__ bias) {
  // move_tail (only where every sequence of the step brings one token): the tail is also moved on here, by the
  // thread that has just read all of it for its channels (tail and move_tail are the same memory).
  constexpr int N = Vec16<T>::N;
  const int t = blockIdx.x;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * N;
  if (c >= channels) return;
  const int seq = seq_of_token[t];
  Vec16<T> result;
  if (seq < 0) {
    grid_dependency_wait();
#pragma unroll
    for (int e = 0; e < N; ++e) result.set(e, 0.f);
    store16(out + (size_t)t * channels + c, result);
    return;
  }
  const int j = t - query_start_loc[seq];
  const T* old = tail + (size_t)state_slots[seq] * (K - 1) * channels;
  grid_dependency_wait();
  float acc[N];
#pragma unroll
  for (int e = 0; e < N; ++e) acc[e] = bias != nullptr ? bias[c + e] : 0.f;
  for (int m = 0; m < K; ++m) {
    const int back = K - 1 - m;
    const Vec16<T> in = back <= j ? load16(x + (size_t)(t - back) * x_stride + c)
                                  : load16(old + (size_t)(K - 1 + j - back) * channels + c);
    float w[N], v[N];
    unpack16(load16(taps + (size_t)m * channels + c), w);
    unpack16(in, v);
#pragma unroll
    for (int e = 0; e < N; ++e) acc[e] = fmaf(w[e], v[e], acc[e]);
    // A step of one token (j = 0): tap m read tail entry m (or the token itself, m = K - 1), which becomes entry m - 1.
    if (move_tail != nullptr && m >= 1)
      store16(move_tail + ((size_t)state_slots[seq] * (K - 1) + (m - 1)) * channels + c, in);
  }
#pragma unroll
  for (int e = 0; e < N; ++e) {
    // bfloat16 results take the fast exponential and division (relative error about 1e-6, far inside the rounding).
    const float sig = sizeof(T) == 2 ? __fdividef(1.0f, 1.0f + __expf(-acc[e])) : 1.0f / (1.0f + expf(-acc[e]));
    result.set(e, act ? acc[e] * sig : acc[e]);
  }
  store16(out + (size_t)t * channels + c, result);
}

// The same for prompts, kRunTokens neighbouring tokens a thread: the taps of its channels stay in registers, and so do the K - 1 inputs
// before the token at hand, so every input is read once and a half instead of K times, and all of a run's are asked for at once.  2,070
// tokens of 6,144 channels, four taps: 15.9 us (23).
constexpr int kRunTokens = 8;
template <typename T, int K>
__global__ void __launch_bounds__(128)
short_conv_run_kernel(const T* __restrict__ x, size_t x_stride, const T* __restrict__ taps, const T* __restrict__ tail,
                      const int* __restrict__ seq_of_token, const int* __restrict__ query_start_loc,
                      const int* __restrict__ state_slots, T* __restrict__ out, int tokens, int channels, int act,
                      const float* __restrict__ bias) {
  constexpr int N = Vec16<T>::N;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * N;
  if (c >= channels) return;
  grid_dependency_wait();
  const int first = blockIdx.x * kRunTokens;
  Vec16<T> input[kRunTokens];
#pragma unroll
  for (int i = 0; i < kRunTokens; ++i) input[i] = load16(x + (size_t)min(first + i, tokens - 1) * x_stride + c);
  float w[K][N], b[N];
#pragma unroll
  for (int m = 0; m < K; ++m) unpack16(load16(taps + (size_t)m * channels + c), w[m]);
#pragma unroll
  for (int e = 0; e < N; ++e) b[e] = bias != nullptr ? bias[c + e] : 0.f;
  Vec16<T> before[K - 1];       // the inputs K - 1, ..., 1 tokens back
  int current = -1;
#pragma unroll
  for (int i = 0; i < kRunTokens; ++i) {
    const int t = first + i;
    if (t >= tokens) return;
    const int seq = seq_of_token[t];
    Vec16<T> result;
    if (seq < 0) {
#pragma unroll
      for (int e = 0; e < N; ++e) result.set(e, 0.f);
      store16(out + (size_t)t * channels + c, result);
      current = -1;
      continue;
    }
    if (seq != current) {       // a run's first token, or the first of the next sequence
      const int j = t - query_start_loc[seq];
      const T* old = tail + (size_t)state_slots[seq] * (K - 1) * channels;
#pragma unroll
      for (int m = 0; m < K - 1; ++m) {
        const int back = K - 1 - m;
        before[m] = back <= j ? load16(x + (size_t)(t - back) * x_stride + c) : load16(old + (size_t)(K - 1 + j - back) * channels + c);
      }
      current = seq;
    }
    float acc[N], v[N];
#pragma unroll
    for (int e = 0; e < N; ++e) acc[e] = b[e];
#pragma unroll
    for (int m = 0; m < K; ++m) {
      unpack16(m < K - 1 ? before[m < K - 1 ? m : 0] : input[i], v);
#pragma unroll
      for (int e = 0; e < N; ++e) acc[e] = fmaf(w[m][e], v[e], acc[e]);
    }
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const float sig = sizeof(T) == 2 ? __fdividef(1.0f, 1.0f + __expf(-acc[e])) : 1.0f / (1.0f + expf(-acc[e]));
      result.set(e, act ? acc[e] * sig : acc[e]);
    }
    store16(out + (size_t)t * channels + c, result);
#pragma unroll
    for (int m = 0; m + 1 < K - 1; ++m) before[m] = before[m + 1];
    before[K - 2] = input[i];
  }
}

template <typename T>
__global__ void short_conv_update_kernel(const T* __restrict__ x, size_t x_stride, T* __restrict__ tail,
                                         const int* __restrict__ query_start_loc, const int* __restrict__ state_slots,
                                         int channels, int K) {
  grid_dependency_wait();
  const int seq = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  const int begin = query_start_loc[seq], n = query_start_loc[seq + 1] - begin;
  if (n <= 0) return;
  const int keep = K - 1;
  T* mine = tail + (size_t)state_slots[seq] * keep * channels;
  // Entry i becomes the input at index n - keep + i of the step, or the old entry i + n where that lies before the
  // step; ascending i reads only entries that are not yet overwritten.
  for (int i = 0; i < keep; ++i) {
    const int li = n - keep + i;
    mine[(size_t)i * channels + c] = li >= 0 ? x[(size_t)(begin + li) * x_stride + c] : mine[(size_t)(i + n) * channels + c];
  }
}

__device__ __forceinline__ float sum_over_column_lanes(float v) {   // the eight lanes of a column: lane bits 2..4
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  v += __shfl_xor_sync(0xffffffffu, v, 16);
  return v;
}

__device__ __forceinline__ float4 load_piece(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_piece(const bf16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                     __uint_as_float(raw.y & 0xffff0000u));
}

// What of a token does not depend on the state, once per (token, head) instead of once per column of S:
// units [tokens][kv_heads][2][dim] = (q dim^-0.5 / |q|, k / |k|) in float with |x| = sqrt(sum x^2 + 1e-6), and
// gates [tokens][heads][2] = (beta, g) = (sigmoid(raw_b), exp(-exp(A_log) * softplus(raw_a + dt_bias))).  One warp
// a (token, head or kv head).  `products` (optional, [tokens][kv_heads][4]): (q . k, k . k', q . k', 0) of the unit vectors, k' the
// token's before (the launch's first has none); dim is then 4, 8, ... or 128 in whole pieces of four, the rows on their size.
template <typename T>
__global__ void delta_gates_kernel(const T* __restrict__ qkv, size_t row_width, const T* __restrict__ ab,
                                   size_t ab_stride, const float* __restrict__ a_log, const float* __restrict__ dt_bias,
                                   float* __restrict__ scales, float* __restrict__ gates, float* __restrict__ products, int tokens,
                                   int heads, int kv_heads, int dim) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int per_token = kv_heads + (heads + 31) / 32;
  const size_t item = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= (size_t)tokens * per_token) return;
  const size_t t = item / per_token;
  const int what = (int)(item - t * per_token);
  if (what < kv_heads) {
    const T* q = qkv + t * row_width + (size_t)what * dim;
    const T* k = q + (size_t)kv_heads * dim;
    float qq = 0.f, kk = 0.f;
    if (products != nullptr) {
      // A lane's four dimensions at once (dim <= 128).
      const bool mine = 4 * lane < dim;
      const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 a = mine ? load_piece(q + 4 * lane) : none, b = mine ? load_piece(k + 4 * lane) : none;
      const float4 c = mine && t > 0 ? load_piece(k + 4 * lane - (ptrdiff_t)row_width) : none;
      const auto dot = [](const float4& x, const float4& y) { return fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, x.x * y.x))); };
      qq = warp_sum(dot(a, a));
      kk = warp_sum(dot(b, b));
      const float pp = warp_sum(dot(c, c)), qk = warp_sum(dot(a, b)), kp = warp_sum(dot(b, c)), qp = warp_sum(dot(a, c));
      const float q_inv = (1.0f / sqrtf((float)dim)) / sqrtf(qq + 1e-6f), k_inv = 1.0f / sqrtf(kk + 1e-6f);
      const float p_inv = 1.0f / sqrtf(pp + 1e-6f);
      float* unit = scales + (t * kv_heads + what) * 2 * (size_t)dim;
      if (mine) {
        *reinterpret_cast<float4*>(unit + 4 * lane) = make_float4(a.x * q_inv, a.y * q_inv, a.z * q_inv, a.w * q_inv);
        *reinterpret_cast<float4*>(unit + dim + 4 * lane) = make_float4(b.x * k_inv, b.y * k_inv, b.z * k_inv, b.w * k_inv);
      }
      if (lane == 0)
        *reinterpret_cast<float4*>(products + (t * kv_heads + what) * 4) =
            make_float4(qk * (q_inv * k_inv), kp * (k_inv * p_inv), qp * (q_inv * p_inv), 0.f);
      return;
    }
    for (int i = lane; i < dim; i += 32) {
      const float a = to_float(q[i]), b = to_float(k[i]);
      qq = fmaf(a, a, qq);
      kk = fmaf(b, b, kk);
    }
    qq = warp_sum(qq);
    kk = warp_sum(kk);
    const float q_inv = (1.0f / sqrtf((float)dim)) / sqrtf(qq + 1e-6f), k_inv = 1.0f / sqrtf(kk + 1e-6f);
    float* unit = scales + (t * kv_heads + what) * 2 * (size_t)dim;
    for (int i = lane; i < dim; i += 32) {
      unit[i] = to_float(q[i]) * q_inv;
      unit[dim + i] = to_float(k[i]) * k_inv;
    }
  } else {
    const int head = (what - kv_heads) * 32 + lane;
    if (head >= heads) return;
    const float raw_b = to_float(ab[t * ab_stride + head]), raw_a = to_float(ab[t * ab_stride + heads + head]);
    const float z = raw_a + dt_bias[head];
    const float soft = z > 20.f ? z : log1pf(expf(z));
    gates[(t * heads + head) * 2] = 1.0f / (1.0f + expf(-raw_b));
    gates[(t * heads + head) * 2 + 1] = expf(-expf(a_log[head]) * soft);
  }
}

// Which entries of a column of 8 R a lane keeps, where everything is vectors: pieces of four, the eight lanes' pieces side by
// side, so that the lanes of a column read 128 neighbouring bytes at once.
__device__ __forceinline__ int piece_at(int c, int part) { return (c * 8 + part) * 4; }

// A lane's R values of a row as floats: its pieces of the row at p (16-byte aligned) when kVector, else the `live` first of
// the R that start at p.
template <typename T, int R, bool kVector>
__device__ __forceinline__ void load_slice(float (&dst)[R], const T* __restrict__ p, int live, int part) {
  if (kVector) {
#pragma unroll
    for (int c = 0; c < R / 4; ++c) {
      const float4 v = load_piece(p + piece_at(c, part));
      dst[c * 4] = v.x; dst[c * 4 + 1] = v.y; dst[c * 4 + 2] = v.z; dst[c * 4 + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) dst[r] = r < live ? to_float(p[r]) : 0.f;
  }
}

template <int R>
struct DeltaToken {   // what a lane needs of one token: its slices of q and k, its column's v, the head's scalars
  float q[R], k[R], v, q_inv, k_inv, beta, g;
};

// The state is kept column by column: state[slot][head][column][dim], so that the lanes of a column read 128 bytes in a row
// and a warp's four columns are 4 * dim * 4 bytes.
// R: entries of a column that one lane keeps (dim <= 8 R).  kAhead: tokens whose inputs are in flight while one is
// computed (1 for steps of single tokens).  kVector: dim == 8 R and every row is 16-byte aligned.
template <typename T, int R, int kAhead, bool kVector>
__global__ void __launch_bounds__(256)
gated_delta_rule_kernel(const T* __restrict__ qkv, const float* __restrict__ scales, const float* __restrict__ gates,
                        float* __restrict__ state, const int* __restrict__ query_start_loc,
                        const int* __restrict__ state_slots, float* __restrict__ out, int heads, int kv_heads, int dim,
                        int vdim, const T* __restrict__ ab, size_t ab_stride, const float* __restrict__ a_log,
                        const float* __restrict__ dt_bias) {
  grid_dependency_wait();
  const int seq = blockIdx.z, head = blockIdx.y;
  const int begin = query_start_loc[seq], end = query_start_loc[seq + 1];
  if (end <= begin) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = lane >> 2;                                   // which eighth of the column
  const int column = blockIdx.x * 32 + warp * 4 + (lane & 3);
  const bool live = column < vdim;
  const int first = kVector ? 0 : part * R;                     // (a vector's pieces: see piece_at)
  const int mine_dims = min(R, max(0, dim - first));            // entries of this lane's slice that exist
  const int qk_width = kv_heads * dim;
  const size_t row_width = 2 * (size_t)qk_width + (size_t)heads * vdim;
  const int kv_head = head / (heads / kv_heads);
  const size_t q_at = (size_t)kv_head * dim + first, k_at = (size_t)qk_width + q_at;
  const size_t v_at = 2 * (size_t)qk_width + (size_t)head * vdim + (live ? column : 0);
  float* mine = state + (((size_t)state_slots[seq] * heads + head) * vdim + (live ? column : 0)) * dim + first;

  float S[R];
  if (kVector) {
#pragma unroll
    for (int c = 0; c < R / 4; ++c) {
      const float4 v = live ? *reinterpret_cast<const float4*>(mine + piece_at(c, part)) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[c * 4] = v.x; S[c * 4 + 1] = v.y; S[c * 4 + 2] = v.z; S[c * 4 + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r) S[r] = (live && r < mine_dims) ? mine[r] : 0.f;
  }

  DeltaToken<R> ring[kAhead];
  auto fetch = [&](DeltaToken<R>& tok, int t) {
    const T* row = qkv + (size_t)t * row_width;
    tok.v = widen(row[v_at]);
    if (kAhead > 1) {
      // From the kernel in front: q and k as unit vectors in float, and the gates.
      const float* unit = scales + ((size_t)t * kv_heads + kv_head) * 2 * (size_t)dim + first;
      load_slice<float, R, kVector>(tok.q, unit, mine_dims, part);
      load_slice<float, R, kVector>(tok.k, unit + dim, mine_dims, part);
      const float2 ga = *reinterpret_cast<const float2*>(gates + ((size_t)t * heads + head) * 2);
      tok.q_inv = 1.f; tok.k_inv = 1.f; tok.beta = ga.x; tok.g = ga.y;
      return;
    }
    load_slice<T, R, kVector>(tok.q, row + q_at, mine_dims, part);
    load_slice<T, R, kVector>(tok.k, row + k_at, mine_dims, part);
    if (kAhead == 1) {
      // Steps of single tokens: no kernel in front; the block works out the token's scales and gates itself.
      float qq = 0.f, kk = 0.f;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        qq = fmaf(tok.q[r], tok.q[r], qq);
        kk = fmaf(tok.k[r], tok.k[r], kk);
      }
      qq = sum_over_column_lanes(qq);
      kk = sum_over_column_lanes(kk);
      tok.q_inv = (1.0f / sqrtf((float)dim)) / sqrtf(qq + 1e-6f);
      tok.k_inv = 1.0f / sqrtf(kk + 1e-6f);
      const float raw_b = to_float(ab[(size_t)t * ab_stride + head]);
      const float z = to_float(ab[(size_t)t * ab_stride + heads + head]) + dt_bias[head];
      const float soft = z > 20.f ? z : log1pf(expf(z));
      tok.beta = 1.0f / (1.0f + expf(-raw_b));
      tok.g = expf(-expf(a_log[head]) * soft);
    }
  };
  // A token's read-out o = S^T q is not on the chain from token to token, only its S is: the lanes' parts of o
  // are added up together with the next token's parts of S^T k, so a token costs one round of shuffles.
  float o_parts = 0.f, o_scale = 0.f;
  int o_token = -1;
  auto step = [&](const DeltaToken<R>& tok, int t) {
    // With S' = g S:  (S'^T k)_j = g k_inv sum_i S_ij k_i;  S <- g S + k (k_inv u)^T;  o_j = q_inv sum_i S_ij q_i.
    float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
    for (int r = 0; r < R; r += 4) {
      d0 = fmaf(S[r], tok.k[r], d0); d1 = fmaf(S[r + 1], tok.k[r + 1], d1);
      d2 = fmaf(S[r + 2], tok.k[r + 2], d2); d3 = fmaf(S[r + 3], tok.k[r + 3], d3);
    }
    float dsum = (d0 + d1) + (d2 + d3), osum = o_parts;
#pragma unroll
    for (int offset = 4; offset <= 16; offset <<= 1) {
      const float a = __shfl_xor_sync(0xffffffffu, dsum, offset), b = __shfl_xor_sync(0xffffffffu, osum, offset);
      dsum += a;
      osum += b;
    }
    if (o_token >= 0 && live && part == 0)
      out[(size_t)o_token * heads * vdim + (size_t)head * vdim + column] = osum * o_scale;
    const float dot = dsum * (tok.g * tok.k_inv);
    const float c = tok.beta * (tok.v - dot) * tok.k_inv;
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int r = 0; r < R; r += 4) {
      S[r] = fmaf(S[r], tok.g, tok.k[r] * c); S[r + 1] = fmaf(S[r + 1], tok.g, tok.k[r + 1] * c);
      S[r + 2] = fmaf(S[r + 2], tok.g, tok.k[r + 2] * c); S[r + 3] = fmaf(S[r + 3], tok.g, tok.k[r + 3] * c);
      o0 = fmaf(S[r], tok.q[r], o0); o1 = fmaf(S[r + 1], tok.q[r + 1], o1);
      o2 = fmaf(S[r + 2], tok.q[r + 2], o2); o3 = fmaf(S[r + 3], tok.q[r + 3], o3);
    }
    o_parts = (o0 + o1) + (o2 + o3);
    o_scale = tok.q_inv;
    o_token = t;
  };

  // Far ahead of the ring, the lines of a token's inputs are asked into the cache: warp w does it for the tokens
  // whose number is w modulo 8, one lane a 128-byte line (the unit vectors, then v, then the gates).
  constexpr int kFar = 24;
  auto ask_ahead = [&](int t) {
    if (kAhead == 1 || t >= end || ((t - begin) & 7) != warp) return;
    const int unit_lines = (8 * dim + 127) / 128;
    const char* where = nullptr;
    if (lane < unit_lines)
      where = reinterpret_cast<const char*>(scales + ((size_t)t * kv_heads + kv_head) * 2 * (size_t)dim) + lane * 128;
    else if (lane == unit_lines)
      where = reinterpret_cast<const char*>(qkv + (size_t)t * row_width + v_at);
    else if (lane == unit_lines + 1)
      where = reinterpret_cast<const char*>(gates + ((size_t)t * heads + head) * 2);
    if (where != nullptr) asm volatile("prefetch.global.L1 [%0];" ::"l"(where));
  };
  for (int t = begin; t < begin + kFar; ++t) ask_ahead(t);
#pragma unroll
  for (int a = 0; a < kAhead; ++a)
    if (begin + a < end) fetch(ring[a], begin + a);
  for (int t = begin; t < end; t += kAhead) {
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {
      if (t + a < end) {
        ask_ahead(t + a + kFar);
        step(ring[a], t + a);
        if (t + a + kAhead < end) fetch(ring[a], t + a + kAhead);
      }
    }
  }
  {
    const float o = sum_over_column_lanes(o_parts) * o_scale;       // the last token's read-out
    if (live && part == 0) out[(size_t)o_token * heads * vdim + (size_t)head * vdim + column] = o;
  }

  if (!live) return;
  if (kVector) {
#pragma unroll
    for (int c = 0; c < R / 4; ++c)
      *reinterpret_cast<float4*>(mine + piece_at(c, part)) = make_float4(S[c * 4], S[c * 4 + 1], S[c * 4 + 2], S[c * 4 + 3]);
  } else {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < mine_dims) mine[r] = S[r];
  }
}

// Two 32-bit numbers in one register pair: a fused multiply-add of both is one instruction, rounded like two.
typedef unsigned long long pair32;
__device__ __forceinline__ pair32 both(float v) {
  pair32 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ pair32 mul_pair(pair32 a, pair32 b) {
  pair32 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair32 fma_pair(pair32 a, pair32 b, pair32 c) {
  pair32 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float sum_pair(pair32 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}

// The same recurrence for prompts and portions, with the tokens' inputs staged in shared memory: the loads of a
// register ring several tokens deep share a warp's few scoreboards, so a wait for one token's inputs also waits
// for the ones just asked for, and a token cost a whole trip to the second-level cache (0.5 us, whatever the head
// size).  Here a block copies eight tokens at a time (unit q and k in float, gates, the block's values of v)
// with cp.async, whose groups are waited for in order, two chunks in flight, and reads them with shared-memory
// loads.  For heads of 256, vdim a multiple of 16 and 16-byte aligned rows (the kernel behind this one takes the smaller heads).
//
// Bound by instructions: a token is about 90 a warp of four columns, one after the other in a launch of a few hundred warps
// (a prompt or two: each waits for the one before, some 3.5 cycles), and one of several warps' on every scheduler in a wide
// one.  So a multiply-add works on two numbers, a chunk's tokens lie at places known to the compiler, and what a thread copies
// comes from pointers that move on by a constant.
constexpr int kStageTokens = 8;

template <typename T, int R>
__global__ void __launch_bounds__(128)
gated_delta_rule_staged_kernel(const T* __restrict__ qkv, const float* __restrict__ units, const float* __restrict__ gates,
                               float* __restrict__ state, const int* __restrict__ query_start_loc,
                               const int* __restrict__ state_slots, float* __restrict__ out, int heads, int kv_heads,
                               int vdim) {
  extern __shared__ __align__(16) unsigned char staged[];
  constexpr int dim = 8 * R, kColumns = 16, kPieces = R / 4;
  constexpr int kUnitBytes = 8 * dim, kValueBytes = kColumns * (int)sizeof(T);
  constexpr int kTokenBytes = kUnitBytes + 16 + (kValueBytes + 15) / 16 * 16;   // units | gates (8 bytes, padded) | v
  grid_dependency_wait();
  const int seq = blockIdx.z, head = blockIdx.y;
  const int begin = query_start_loc[seq], end = query_start_loc[seq + 1];
  if (end <= begin) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = lane >> 2;                                   // which eighth of the column
  const int local_column = warp * 4 + (lane & 3), column = blockIdx.x * kColumns + local_column;
  const int qk_width = kv_heads * dim;
  const size_t row_width = 2 * (size_t)qk_width + (size_t)heads * vdim;
  const int kv_head = head / (heads / kv_heads);
  const size_t v_at = 2 * (size_t)qk_width + (size_t)head * vdim + (size_t)blockIdx.x * kColumns;
  float* mine = state + (((size_t)state_slots[seq] * heads + head) * vdim + column) * dim;

  pair32 S[kPieces][2];
#pragma unroll
  for (int c = 0; c < kPieces; ++c) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(mine + piece_at(c, part));
    S[c][0] = v.x;
    S[c][1] = v.y;
  }

  // A thread's copies of a chunk: one piece of the unit vectors of every kRound-th token, and for some threads a piece of v
  // or a token's gates.  Where they come from moves on by the same distance every chunk.
  constexpr int kUnitPieces = kUnitBytes / 16, kRound = 128 / kUnitPieces > 0 ? 128 / kUnitPieces : 1;
  constexpr int kValuePieces = kValueBytes / 16 > 0 ? kValueBytes / 16 : 1;
  static_assert(kValueBytes % 16 == 0 && 128 % kUnitPieces == 0 && kStageTokens * kValuePieces <= 128, "a chunk's copies");
  const size_t unit_row = (size_t)kv_heads * 2 * dim;             // of floats, a token
  const int unit_token = threadIdx.x / kUnitPieces, unit_piece = threadIdx.x % kUnitPieces;
  const float* unit_src = units + ((size_t)(begin + unit_token) * kv_heads + kv_head) * 2 * dim + unit_piece * 4;
  const int value_token = threadIdx.x / kValuePieces, value_piece = threadIdx.x % kValuePieces;
  const T* value_src = qkv + (size_t)(begin + value_token) * row_width + v_at + value_piece * (16 / (int)sizeof(T));
  const float* gate_src = gates + ((size_t)(begin + threadIdx.x) * heads + head) * 2;
  const unsigned stage = (unsigned)__cvta_generic_to_shared(staged);
  auto copy_chunk = [&](int chunk) {
    const unsigned buffer = stage + (unsigned)(chunk & 1) * (kStageTokens * kTokenBytes);
    const int left = end - begin - chunk * kStageTokens;          // tokens from the chunk's first on
#pragma unroll
    for (int j = 0; j < kStageTokens; j += kRound)
      if (unit_token + j < left && unit_token + j < kStageTokens)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buffer + (unit_token + j) * kTokenBytes + unit_piece * 16),
                     "l"(unit_src + j * unit_row));
    if (value_token < kStageTokens && value_token < left)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buffer + value_token * kTokenBytes + kUnitBytes + 16 + value_piece * 16),
                   "l"(value_src));
    if (threadIdx.x < kStageTokens && (int)threadIdx.x < left)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(buffer + threadIdx.x * kTokenBytes + kUnitBytes), "l"(gate_src));
    asm volatile("cp.async.commit_group;" ::);
    unit_src += kStageTokens * unit_row;
    value_src += kStageTokens * row_width;
    gate_src += (size_t)kStageTokens * heads * 2;
  };

  // Where the column's read-out of the token before goes.
  const size_t out_row = (size_t)heads * vdim;
  float* out_at = out + (size_t)begin * out_row + (size_t)head * vdim + column - out_row;
  float o_parts = 0.f;
  const int lane_at = part * 16, column_at = kUnitBytes + 16 + local_column * (int)sizeof(T);
  bool stores = false;          // not yet: the first token has none before it
  // One token, whose inputs lie at `tok` (a lane's pieces of a row: see piece_at).
  auto step = [&](const unsigned char* tok) {
    const unsigned char *q = tok + lane_at, *k = q + dim * 4;
    const float2 ga = *reinterpret_cast<const float2*>(tok + kUnitBytes);
    const float v = widen(*reinterpret_cast<const T*>(tok + column_at));
    pair32 kk[kPieces][2], d0, d1, o0, o1;
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
      const ulonglong2 k4 = *reinterpret_cast<const ulonglong2*>(k + c * 128);
      kk[c][0] = k4.x;
      kk[c][1] = k4.y;
      d0 = c == 0 ? mul_pair(S[c][0], k4.x) : fma_pair(S[c][0], k4.x, d0);
      d1 = c == 0 ? mul_pair(S[c][1], k4.y) : fma_pair(S[c][1], k4.y, d1);
    }
    // The read-out of the token before is added up over the lanes together with this token's S^T k.
    float dsum = sum_pair(d0) + sum_pair(d1), osum = o_parts;
#pragma unroll
    for (int offset = 4; offset <= 16; offset <<= 1) {
      const float a = __shfl_xor_sync(0xffffffffu, dsum, offset), b = __shfl_xor_sync(0xffffffffu, osum, offset);
      dsum += a;
      osum += b;
    }
    if (stores) *out_at = osum;
    stores = part == 0;
    out_at += out_row;
    const pair32 g2 = both(ga.y), c2 = both(ga.x * (v - dsum * ga.y));
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
      const ulonglong2 q4 = *reinterpret_cast<const ulonglong2*>(q + c * 128);
      S[c][0] = fma_pair(S[c][0], g2, mul_pair(kk[c][0], c2));
      S[c][1] = fma_pair(S[c][1], g2, mul_pair(kk[c][1], c2));
      o0 = c == 0 ? mul_pair(S[c][0], q4.x) : fma_pair(S[c][0], q4.x, o0);
      o1 = c == 0 ? mul_pair(S[c][1], q4.y) : fma_pair(S[c][1], q4.y, o1);
    }
    o_parts = sum_pair(o0) + sum_pair(o1);
  };

  const int chunks = (end - begin + kStageTokens - 1) / kStageTokens;
  copy_chunk(0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    if (chunk + 1 < chunks) {
      copy_chunk(chunk + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const unsigned char* tok = staged + (size_t)(chunk & 1) * kStageTokens * kTokenBytes;
    const int count = min(kStageTokens, end - begin - chunk * kStageTokens);
    if (count == kStageTokens) {           // at places known when this is compiled
#pragma unroll 4
      for (int j = 0; j < kStageTokens; ++j) step(tok + j * kTokenBytes);
    } else {
#pragma unroll 1
      for (int j = 0; j < count; ++j) step(tok + j * kTokenBytes);
    }
    __syncthreads();     // the buffer is written again two chunks on
  }
  const float total = sum_over_column_lanes(o_parts);
  if (part == 0) *out_at = total;
#pragma unroll
  for (int c = 0; c < kPieces; ++c)
    *reinterpret_cast<ulonglong2*>(mine + piece_at(c, part)) = make_ulonglong2(S[c][0], S[c][1]);
}

// The same for head sizes up to 128: two tokens at a time, C columns a lane (1, or 2 where a launch has blocks enough).  With S the state before a pair of
// tokens, S2 = g1 g2 S + k1 (g2 c1)^T + k2 c2^T, where c1 = beta1 (v1 - g1 S^T k1) and c2 = beta2 (v2 - g2 (g1 S^T k2 + (k1 . k2) c1)):
// all four products with S (k1, k2, q1, q2) are taken at once, what the second token meets of the first is three products of the
// pair's vectors that the kernel in front has made, and the sums over a column's eight lanes are one exchange of eight values
// (seven shuffles, each lane ending with one of them; of four where a lane has one column) instead of four of two.  Two columns share the
// reads of q and k.
//
// Bound by the multiply-adds and shared memory's reads side by side where a launch is wide (56 and 64 cycles of an SM for two tokens of eight
// columns), by the chain of a pair's sums where it is not.  Measured on B200, 16 heads of 128 x 128, the kernel in front included: one
// prompt of 512 tokens 79 us (94 a token at a time in one column a lane; 98 in two), eight of 512 272 (303), eight of 67 to 450 157 (181);
// 8 heads, one of 1,400 198 (240).
template <typename T, int R, int C>
__global__ void __launch_bounds__(128)
gated_delta_rule_pairs_kernel(const T* __restrict__ qkv, const float* __restrict__ units, const float* __restrict__ gates,
                              const float* __restrict__ products, float* __restrict__ state, const int* __restrict__ query_start_loc,
                              const int* __restrict__ state_slots, float* __restrict__ out, int heads, int kv_heads, int vdim) {
  extern __shared__ __align__(16) unsigned char staged[];
  constexpr int dim = 8 * R, kColumns = 16 * C, kPieces = R / 4;
  constexpr int kUnitBytes = 8 * dim, kValueBytes = kColumns * (int)sizeof(T);
  constexpr int kGatesAt = kUnitBytes, kProductsAt = kUnitBytes + 16, kValuesAt = kUnitBytes + 32;
  constexpr int kTokenBytes = kValuesAt + kValueBytes;          // units | gates (8 bytes, padded) | products | v
  grid_dependency_wait();
  const int seq = blockIdx.z, head = blockIdx.y;
  const int begin = query_start_loc[seq], end = query_start_loc[seq + 1];
  if (end <= begin) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = lane >> 2;                                   // which eighth of the columns
  const int local_column = (warp * 4 + (lane & 3)) * C;         // of C
  const int qk_width = kv_heads * dim;
  const size_t row_width = 2 * (size_t)qk_width + (size_t)heads * vdim;
  const int kv_head = head / (heads / kv_heads);
  const size_t v_at = 2 * (size_t)qk_width + (size_t)head * vdim + (size_t)blockIdx.x * kColumns;
  float* mine = state + (((size_t)state_slots[seq] * heads + head) * vdim + blockIdx.x * kColumns + local_column) * dim;

  pair32 S[C][kPieces][2];
#pragma unroll
  for (int j = 0; j < C; ++j)
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(mine + j * dim + piece_at(c, part));
      S[j][c][0] = v.x;
      S[j][c][1] = v.y;
    }

  // A thread's copies of a chunk, as in the kernel above.
  constexpr int kUnitPieces = kUnitBytes / 16, kRound = 128 / kUnitPieces > 0 ? 128 / kUnitPieces : 1;
  constexpr int kValuePieces = kValueBytes / 16;
  static_assert(128 % kUnitPieces == 0 && kStageTokens * kValuePieces <= 128, "a chunk's copies");
  const size_t unit_row = (size_t)kv_heads * 2 * dim;
  const int unit_token = threadIdx.x / kUnitPieces, unit_piece = threadIdx.x % kUnitPieces;
  const float* unit_src = units + ((size_t)(begin + unit_token) * kv_heads + kv_head) * 2 * dim + unit_piece * 4;
  const int value_token = threadIdx.x / kValuePieces, value_piece = threadIdx.x % kValuePieces;
  const T* value_src = qkv + (size_t)(begin + value_token) * row_width + v_at + value_piece * (16 / (int)sizeof(T));
  const int small_token = threadIdx.x & 31;                     // warp 0: gates; warp 1: products
  const float* small_src = threadIdx.x < 32 ? gates + ((size_t)(begin + small_token) * heads + head) * 2
                                            : products + ((size_t)(begin + small_token) * kv_heads + kv_head) * 4;
  const size_t small_step = threadIdx.x < 32 ? (size_t)kStageTokens * heads * 2 : (size_t)kStageTokens * kv_heads * 4;
  const unsigned stage = (unsigned)__cvta_generic_to_shared(staged);
  auto copy_chunk = [&](int chunk) {
    const unsigned buffer = stage + (unsigned)(chunk & 1) * (kStageTokens * kTokenBytes);
    const int left = end - begin - chunk * kStageTokens;
#pragma unroll
    for (int j = 0; j < kStageTokens; j += kRound)
      if (unit_token + j < left && unit_token + j < kStageTokens)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buffer + (unit_token + j) * kTokenBytes + unit_piece * 16),
                     "l"(unit_src + j * unit_row));
    if (value_token < kStageTokens && value_token < left)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buffer + value_token * kTokenBytes + kValuesAt + value_piece * 16),
                   "l"(value_src));
    if (threadIdx.x < 64 && small_token < kStageTokens && small_token < left) {
      if (threadIdx.x < 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(buffer + small_token * kTokenBytes + kGatesAt), "l"(small_src));
      else
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buffer + small_token * kTokenBytes + kProductsAt), "l"(small_src));
    }
    asm volatile("cp.async.commit_group;" ::);
    unit_src += kStageTokens * unit_row;
    value_src += kStageTokens * row_width;
    small_src += small_step;
  };

  const size_t out_row = (size_t)heads * vdim;
  // A lane of the last four eighths (one column: of two of them) stores one of the pair's read-outs: of the first or the second token, of
  // its first or second column.
  const bool second_token = C == 2 ? part & 1 : part & 2, second_column = C == 2 && (part & 2);
  const bool stores = C == 2 ? part >= 4 : part == 4 || part == 6;
  float* out_at = out + (size_t)(begin + second_token) * out_row + (size_t)head * vdim + blockIdx.x * kColumns + local_column + second_column;
  const auto column_values = [&](const unsigned char* tok, float (&v)[C]) {
    const T* at = reinterpret_cast<const T*>(tok + kValuesAt) + local_column;
#pragma unroll
    for (int j = 0; j < C; ++j) v[j] = widen(at[j]);
  };
  // Sums over the eight lanes of a column group: lane `part` returns with the sum of v[part], or with one column of v[part / 2].
  const auto exchange = [&](float (&v)[4 * C]) {
    const bool high = part & 4, mid = part & 2, low = part & 1;
    if constexpr (C == 1) {
      float a[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = (high ? v[i + 2] : v[i]) + __shfl_xor_sync(0xffffffffu, high ? v[i] : v[i + 2], 16);
      const float b = (mid ? a[1] : a[0]) + __shfl_xor_sync(0xffffffffu, mid ? a[0] : a[1], 8);
      return b + __shfl_xor_sync(0xffffffffu, b, 4);
    } else {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = (high ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, high ? v[i] : v[i + 4], 16);
#pragma unroll
    for (int i = 0; i < 2; ++i) b[i] = (mid ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, mid ? a[i] : a[i + 2], 8);
    return (low ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, low ? b[0] : b[1], 4);
    }
  };
  // Which lane has the sums of S^T k of the first or second token, column j.
  const auto holder = [&](int j, int token) { return (C == 2 ? 8 * j + 4 * token : 8 * token) + (lane & 3); };
  // Two tokens whose inputs lie at `tok` and behind it.
  const auto step_two = [&](const unsigned char* tok) {
    const unsigned char *one = tok + part * 16, *two = one + kTokenBytes;
    pair32 k1[kPieces][2], k2[kPieces][2], sum[C][4];
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(one + dim * 4 + c * 128);
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(two + dim * 4 + c * 128);
      const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(one + c * 128), r = *reinterpret_cast<const ulonglong2*>(two + c * 128);
      k1[c][0] = a.x, k1[c][1] = a.y, k2[c][0] = b.x, k2[c][1] = b.y;
#pragma unroll
      for (int j = 0; j < C; ++j) {
        sum[j][0] = c == 0 ? mul_pair(S[j][c][0], a.x) : fma_pair(S[j][c][0], a.x, sum[j][0]);
        sum[j][1] = c == 0 ? mul_pair(S[j][c][0], b.x) : fma_pair(S[j][c][0], b.x, sum[j][1]);
        sum[j][2] = c == 0 ? mul_pair(S[j][c][0], q.x) : fma_pair(S[j][c][0], q.x, sum[j][2]);
        sum[j][3] = c == 0 ? mul_pair(S[j][c][0], r.x) : fma_pair(S[j][c][0], r.x, sum[j][3]);
        sum[j][0] = fma_pair(S[j][c][1], a.y, sum[j][0]);
        sum[j][1] = fma_pair(S[j][c][1], b.y, sum[j][1]);
        sum[j][2] = fma_pair(S[j][c][1], q.y, sum[j][2]);
        sum[j][3] = fma_pair(S[j][c][1], r.y, sum[j][3]);
      }
    }
    const float2 gate1 = *reinterpret_cast<const float2*>(tok + kGatesAt), gate2 = *reinterpret_cast<const float2*>(tok + kTokenBytes + kGatesAt);
    const float own1 = *reinterpret_cast<const float*>(tok + kProductsAt);
    const float4 met = *reinterpret_cast<const float4*>(tok + kTokenBytes + kProductsAt);      // q2 . k2, k2 . k1, q2 . k1
    float v1[C], v2[C];
    column_values(tok, v1);
    column_values(tok + kTokenBytes, v2);
    // By lane: S^T k1 and S^T k2 of the first column, of the second, then S^T q1 and S^T q2 of the first, of the second.
    float parts[4 * C];
#pragma unroll
    for (int j = 0; j < C; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        parts[2 * j + i] = sum_pair(sum[j][i]);
        parts[2 * C + 2 * j + i] = sum_pair(sum[j][2 + i]);
      }
    const float held = exchange(parts);
    const float g1 = gate1.y, g2 = gate2.y, both_decays = g1 * g2;
    float c1[C], c2[C];
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const float d1 = __shfl_sync(0xffffffffu, held, holder(j, 0)), d2 = __shfl_sync(0xffffffffu, held, holder(j, 1));
      c1[j] = gate1.x * (v1[j] - g1 * d1);
      c2[j] = gate2.x * (v2[j] - g2 * fmaf(met.y, c1[j], g1 * d2));
    }
    if (stores) {
      const float first = second_column ? c1[C - 1] : c1[0], second = second_column ? c2[C - 1] : c2[0];
      *out_at = second_token ? fmaf(met.x, second, fmaf(met.z, g2 * first, both_decays * held)) : fmaf(own1, first, g1 * held);
    }
    out_at += 2 * out_row;
    const pair32 decay = both(both_decays);
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const pair32 e1 = both(g2 * c1[j]), e2 = both(c2[j]);
#pragma unroll
      for (int c = 0; c < kPieces; ++c) {
        S[j][c][0] = fma_pair(S[j][c][0], decay, fma_pair(k2[c][0], e2, mul_pair(k1[c][0], e1)));
        S[j][c][1] = fma_pair(S[j][c][1], decay, fma_pair(k2[c][1], e2, mul_pair(k1[c][1], e1)));
      }
    }
  };
  // The last token of an odd number.
  const auto step_one = [&](const unsigned char* tok) {
    const unsigned char* one = tok + part * 16;
    pair32 k1[kPieces][2], sum[C][2];
#pragma unroll
    for (int c = 0; c < kPieces; ++c) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(one + dim * 4 + c * 128), q = *reinterpret_cast<const ulonglong2*>(one + c * 128);
      k1[c][0] = a.x, k1[c][1] = a.y;
#pragma unroll
      for (int j = 0; j < C; ++j) {
        sum[j][0] = c == 0 ? mul_pair(S[j][c][0], a.x) : fma_pair(S[j][c][0], a.x, sum[j][0]);
        sum[j][1] = c == 0 ? mul_pair(S[j][c][0], q.x) : fma_pair(S[j][c][0], q.x, sum[j][1]);
        sum[j][0] = fma_pair(S[j][c][1], a.y, sum[j][0]);
        sum[j][1] = fma_pair(S[j][c][1], q.y, sum[j][1]);
      }
    }
    const float2 gate = *reinterpret_cast<const float2*>(tok + kGatesAt);
    const float own = *reinterpret_cast<const float*>(tok + kProductsAt);
    float v[C];
    column_values(tok, v);
    float parts[4 * C];
#pragma unroll
    for (int j = 0; j < C; ++j) {
      parts[2 * j] = sum_pair(sum[j][0]);
      parts[2 * C + 2 * j] = sum_pair(sum[j][1]);
      parts[2 * j + 1] = parts[2 * C + 2 * j + 1] = 0.f;
    }
    const float held = exchange(parts);
    float c1[C];
#pragma unroll
    for (int j = 0; j < C; ++j) c1[j] = gate.x * (v[j] - gate.y * __shfl_sync(0xffffffffu, held, holder(j, 0)));
    if (stores && !second_token) *out_at = fmaf(own, second_column ? c1[C - 1] : c1[0], gate.y * held);
    const pair32 decay = both(gate.y);
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const pair32 e1 = both(c1[j]);
#pragma unroll
      for (int c = 0; c < kPieces; ++c) {
        S[j][c][0] = fma_pair(S[j][c][0], decay, mul_pair(k1[c][0], e1));
        S[j][c][1] = fma_pair(S[j][c][1], decay, mul_pair(k1[c][1], e1));
      }
    }
  };

  const int chunks = (end - begin + kStageTokens - 1) / kStageTokens;
  copy_chunk(0);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    if (chunk + 1 < chunks) {
      copy_chunk(chunk + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const unsigned char* tok = staged + (size_t)(chunk & 1) * kStageTokens * kTokenBytes;
    const int count = min(kStageTokens, end - begin - chunk * kStageTokens);
    if (count == kStageTokens) {           // at places known when this is compiled
#pragma unroll
      for (int j = 0; j < kStageTokens; j += 2) step_two(tok + j * kTokenBytes);
    } else {
#pragma unroll 1
      for (int j = 0; j + 1 < count; j += 2) step_two(tok + j * kTokenBytes);
    }
    if (count & 1) step_one(tok + (count - 1) * kTokenBytes);
    __syncthreads();     // the buffer is written again two chunks on
  }
#pragma unroll
  for (int j = 0; j < C; ++j)
#pragma unroll
    for (int c = 0; c < kPieces; ++c)
      *reinterpret_cast<ulonglong2*>(mine + j * dim + piece_at(c, part)) = make_ulonglong2(S[j][c][0], S[j][c][1]);
}

// Whether a launch's prompts go two tokens at a time: the sizes and alignments that the kernel above takes.
template <typename T>
bool in_pairs(int dim, int vdim, int heads, int kv_heads, const T* qkv, const float* state, const float* scales) {
  const size_t row_bytes = (2 * (size_t)kv_heads * dim + (size_t)heads * vdim) * sizeof(T);
  return (dim == 32 || dim == 64 || dim == 128) && vdim % 16 == 0 && row_bytes % 16 == 0 && aligned16(qkv) && aligned16(state) &&
         aligned16(scales) && ((size_t)heads * vdim * sizeof(T)) % 16 == 0 && (2 * (size_t)kv_heads * dim * sizeof(T)) % 16 == 0;
}

template <typename T, int R, int C>
int launch_pairs(int tokens, dim3 grid, cudaStream_t stream, const T* qkv, const float* scales, const float* gates, const float* products,
                 float* state, const int* qsl, const int* slots, float* out, int heads, int kv_heads, int vdim) {
  constexpr size_t smem = 2 * (size_t)kStageTokens * (8 * 8 * R + 32 + 16 * C * sizeof(T));
  return (int)launch_pdl(tokens, gated_delta_rule_pairs_kernel<T, R, C>, dim3(vdim / (16 * C), grid.y, grid.z), dim3(128), smem, stream, qkv, scales,
                         gates, products, state, qsl, slots, out, heads, kv_heads, vdim);
}

// Two columns a lane where a launch has blocks enough for that; one where it waits for the chain over its longest sequence's tokens.  What
// counts as a block is a longest sequence's worth of tokens (`tokens` / `max_q_len` of them); a sequence beside those that brings one token
// reads and writes its state and is done, a twelfth of one.  By the number of sequences alone 20 single tokens beside a prompt of 300, 16
// heads of 64 x 64, took 52 us in two columns (43 in one, 49 a token at a time).  The line, by head size: 16 heads of 128 x 128, 4
// prompts of 512 163 us in one and 149 in two, of 32 heads 261 and 250, 8 heads and 300 beside 20 single tokens 50 and 59; 64 x 64, 16 heads, 8 of
// 512 122 and 126, 30 of 64 50 and 48.  At head size 32,
// where the chain is short, 16 heads in float32, 4 of 512 72.5 and 73.2, 8 of 512 89 and 84, 20 single tokens beside 300 39 and 40.
template <typename T, int R>
int launch_pairs(int tokens, int max_q_len, dim3 grid, cudaStream_t stream, const T* qkv, const float* scales, const float* gates,
                 const float* products, float* state, const int* qsl, const int* slots, float* out, int heads, int kv_heads, int vdim) {
  const float sequences = (float)grid.z, whole = max_q_len > 1 ? fminf((float)tokens / (float)max_q_len, sequences) : sequences;
  const float blocks = (float)(vdim / 32 * grid.y) * (R == 4 ? sequences : whole + (sequences - whole) / 12.f);
  const bool wide = vdim % 32 == 0 && blocks > (R == 8 ? 576.f : R == 16 ? 320.f : 64.f);
  return wide ? launch_pairs<T, R, 2>(tokens, grid, stream, qkv, scales, gates, products, state, qsl, slots, out, heads, kv_heads, vdim)
              : launch_pairs<T, R, 1>(tokens, grid, stream, qkv, scales, gates, products, state, qsl, slots, out, heads, kv_heads, vdim);
}

template <typename T, int R>
int launch_delta_r(bool single, bool vector, int tokens, dim3 grid, cudaStream_t stream, const T* qkv, const float* scales,
                   const float* gates, float* state, const int* qsl, const int* slots, float* out, int heads,
                   int kv_heads, int dim, int vdim, const T* ab, size_t ab_stride, const float* a_log,
                   const float* dt_bias) {
  // Tokens in flight: as many as the registers hold beside the state (a token costs 2 R + 5 of them).
  constexpr int kDeep = (2 * R + 5) * 4 + R <= 190 ? 4 : 2;
#define LI_DELTA(AHEAD, VEC)                                                                                          \
  return (int)launch_pdl(tokens, gated_delta_rule_kernel<T, R, AHEAD, VEC>, grid, dim3(256), 0, stream, qkv, scales,  \
                         gates, state, qsl, slots, out, heads, kv_heads, dim, vdim, ab, ab_stride, a_log, dt_bias)
  if (single) {
    if (vector) LI_DELTA(1, true);
    LI_DELTA(1, false);
  }
  if constexpr (R == 32) {      // (smaller heads go two tokens at a time)
    if (vector && vdim % 16 == 0 && aligned16(scales) && (((size_t)heads * vdim) * sizeof(T)) % 16 == 0) {
      constexpr size_t smem = 2 * (size_t)kStageTokens * (8 * 8 * R + 16 + (16 * sizeof(T) + 15) / 16 * 16);
      const dim3 staged_grid(vdim / 16, grid.y, grid.z);
      return (int)launch_pdl(tokens, gated_delta_rule_staged_kernel<T, R>, staged_grid, dim3(128), smem, stream, qkv, scales, gates,
                             state, qsl, slots, out, heads, kv_heads, vdim);
    }
  }
  if (vector) LI_DELTA(kDeep, true);
  LI_DELTA(kDeep, false);
#undef LI_DELTA
}

template <typename T>
int launch_delta(int dim, bool single, int tokens, dim3 grid, cudaStream_t stream, const T* qkv, const float* scales,
                 const float* gates, float* state, const int* qsl, const int* slots, float* out, int heads,
                 int kv_heads, int vdim, const T* ab, size_t ab_stride, const float* a_log, const float* dt_bias) {
  const int R = dim <= 32 ? 4 : dim <= 64 ? 8 : dim <= 128 ? 16 : 32;
  const size_t row_bytes = (2 * (size_t)kv_heads * dim + (size_t)heads * vdim) * sizeof(T);
  const bool vector = dim == 8 * R && row_bytes % 16 == 0 && aligned16(qkv) && aligned16(state) &&
                      (R * sizeof(T)) % 16 == 0;
#define LI_DELTA_R(RR)                                                                                                \
  return launch_delta_r<T, RR>(single, vector, tokens, grid, stream, qkv, scales, gates, state, qsl, slots, out, heads, \
                               kv_heads, dim, vdim, ab, ab_stride, a_log, dt_bias)
  if (R == 4) LI_DELTA_R(4);
  if (R == 8) LI_DELTA_R(8);
  if (R == 16) LI_DELTA_R(16);
  LI_DELTA_R(32);
#undef LI_DELTA_R
}

}  // namespace li

using namespace li;

LI_EXPORT int li_short_conv(int dtype, const void* x, size_t x_stride, const void* taps, const void* tail,
                            const int* seq_of_token, const int* query_start_loc, const int* state_slots, void* out,
                            int tokens, int channels, int K, int act, int move_tail, const float* bias,
                            cudaStream_t stream) {
  if (tokens <= 0 || channels <= 0) return 0;
  if (K < 1 || K > kMaxTaps || (K > 1 && tail == nullptr) || (channels + 127) / 128 > 65535) return LI_ERR_UNSUPPORTED;
  // move_tail: every sequence of the step brings exactly one token and the caller wants the tail moved on by
  // this launch; only the vector kernel does that (LI_ERR_UNSUPPORTED otherwise: the caller then updates apart).
  const int lanes = dtype == kFloat32 ? 4 : 8;     // channels in a 16-byte vector
  if (channels % lanes == 0 && x_stride % lanes == 0 && aligned16(x) && aligned16(out) && aligned16(taps) &&
      (K == 1 || aligned16(tail))) {
    const int vectors = channels / lanes;
    const dim3 vgrid(tokens, (vectors + 127) / 128);
    // Four taps, and tokens enough that every SM still has a few blocks.
    if (K == 4 && !move_tail && (long)(tokens / kRunTokens) * vgrid.y >= 2 * 148) {
      const dim3 rgrid((tokens + kRunTokens - 1) / kRunTokens, vgrid.y);
      if (dtype == kFloat32)
        return (int)launch_pdl(tokens, short_conv_run_kernel<float, 4>, rgrid, dim3(128), 0, stream, (const float*)x, x_stride,
                               (const float*)taps, (const float*)tail, seq_of_token, query_start_loc, state_slots, (float*)out, tokens,
                               channels, act, bias);
      return (int)launch_pdl(tokens, short_conv_run_kernel<bf16, 4>, rgrid, dim3(128), 0, stream, (const bf16*)x, x_stride,
                             (const bf16*)taps, (const bf16*)tail, seq_of_token, query_start_loc, state_slots, (bf16*)out, tokens, channels,
                             act, bias);
    }
    if (dtype == kFloat32)
      return (int)launch_pdl(tokens, short_conv_vec_kernel<float>, vgrid, dim3(128), 0, stream, (const float*)x, x_stride,
                             (const float*)taps, (const float*)tail, seq_of_token, query_start_loc, state_slots,
                             (float*)out, channels, K, act, move_tail ? (float*)tail : (float*)nullptr, bias);
    return (int)launch_pdl(tokens, short_conv_vec_kernel<bf16>, vgrid, dim3(128), 0, stream, (const bf16*)x, x_stride,
                           (const bf16*)taps, (const bf16*)tail, seq_of_token, query_start_loc, state_slots, (bf16*)out,
                           channels, K, act, move_tail ? (bf16*)tail : (bf16*)nullptr, bias);
  }
  if (move_tail) return LI_ERR_UNSUPPORTED;
  const dim3 grid(tokens, (channels + 127) / 128);
  if (dtype == kFloat32)
    return (int)launch_pdl(tokens, short_conv_kernel<float>, grid, dim3(128), 0, stream, (const float*)x, x_stride,
                           (const float*)taps, (const float*)tail, seq_of_token, query_start_loc, state_slots,
                           (float*)out, channels, K, act, bias);
  return (int)launch_pdl(tokens, short_conv_kernel<bf16>, grid, dim3(128), 0, stream, (const bf16*)x, x_stride,
                         (const bf16*)taps, (const bf16*)tail, seq_of_token, query_start_loc, state_slots, (bf16*)out,
                         channels, K, act, bias);
}

LI_EXPORT int li_short_conv_update(int dtype, const void* x, size_t x_stride, void* tail, const int* query_start_loc,
                                   const int* state_slots, int num_seqs, int channels, int K, cudaStream_t stream) {
  if (num_seqs <= 0 || channels <= 0 || K <= 1) return 0;
  if (K > kMaxTaps || num_seqs > 65535) return LI_ERR_UNSUPPORTED;
  const dim3 grid((channels + 127) / 128, num_seqs);
  if (dtype == kFloat32)
    return (int)launch_pdl(num_seqs, short_conv_update_kernel<float>, grid, dim3(128), 0, stream, (const float*)x,
                           x_stride, (float*)tail, query_start_loc, state_slots, channels, K);
  return (int)launch_pdl(num_seqs, short_conv_update_kernel<bf16>, grid, dim3(128), 0, stream, (const bf16*)x, x_stride,
                         (bf16*)tail, query_start_loc, state_slots, channels, K);
}

// qkv [tokens, 2 * kv_heads * dim + heads * vdim]; ab [tokens, >= 2 * heads] with `ab_stride` elements a row; state
// [slots, heads, vdim, dim] (column by column); out [tokens, heads * vdim]; scratch: 2 * tokens * (kv_heads * dim +
// heads) + 4 * tokens * kv_heads + 4 floats.  max_q_len: the most tokens a sequence brings (1 chooses the variant without tokens in flight).
LI_EXPORT int li_gated_delta_rule(int dtype, const void* qkv, const void* ab, size_t ab_stride, int tokens, int num_seqs,
                                  const float* a_log, const float* dt_bias, float* state, const int* query_start_loc,
                                  const int* state_slots, float* out, int heads, int kv_heads, int dim, int vdim,
                                  int max_q_len, float* scratch, cudaStream_t stream) {
  if (tokens <= 0 || num_seqs <= 0) return 0;
  if (heads < 1 || kv_heads < 1 || heads % kv_heads || dim < 1 || dim > 256 || vdim < 1 || heads > 65535 ||
      num_seqs > 65535 || scratch == nullptr)
    return LI_ERR_UNSUPPORTED;
  float* scales = scratch;
  float* gates = scratch + 2 * (size_t)tokens * kv_heads * dim;
  float* room = gates + ((2 * (size_t)tokens * heads + 3) & ~(size_t)3);      // products of neighbouring tokens
  const size_t row_width = 2 * (size_t)kv_heads * dim + (size_t)heads * vdim;
  const size_t items = (size_t)tokens * (kv_heads + (heads + 31) / 32);
  const dim3 gates_grid((unsigned)((items + 7) / 8));
  const dim3 grid((vdim + 31) / 32, heads, num_seqs);
  const bool single = max_q_len == 1;     // the recurrence kernel then works out scales and gates itself
  const auto run = [&](auto* typed) {
    using T = std::remove_cv_t<std::remove_pointer_t<decltype(typed)>>;
    const T* rows = (const T*)qkv;
    const bool pairs = !single && in_pairs(dim, vdim, heads, kv_heads, rows, state, scales);
    if (!single) {
      const int code = (int)launch_pdl(tokens, delta_gates_kernel<T>, gates_grid, dim3(256), 0, stream, rows, row_width, (const T*)ab,
                                       ab_stride, a_log, dt_bias, scales, gates, pairs ? room : (float*)nullptr, tokens, heads, kv_heads, dim);
      if (code) return code;
    }
    if (pairs) {
      if (dim == 32) return launch_pairs<T, 4>(tokens, max_q_len, grid, stream, rows, scales, gates, room, state, query_start_loc, state_slots, out, heads, kv_heads, vdim);
      if (dim == 64) return launch_pairs<T, 8>(tokens, max_q_len, grid, stream, rows, scales, gates, room, state, query_start_loc, state_slots, out, heads, kv_heads, vdim);
      return launch_pairs<T, 16>(tokens, max_q_len, grid, stream, rows, scales, gates, room, state, query_start_loc, state_slots, out, heads, kv_heads, vdim);
    }
    return launch_delta<T>(dim, single, tokens, grid, stream, rows, scales, gates, state, query_start_loc, state_slots, out, heads, kv_heads,
                           vdim, (const T*)ab, ab_stride, a_log, dt_bias);
  };
  return dtype == kFloat32 ? run((float*)nullptr) : run((bf16*)nullptr);
}
