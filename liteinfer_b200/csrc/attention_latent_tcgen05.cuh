// Latent attention over prompts and portions of prompts on the fifth-generation tensor cores (bfloat16, a rotated part
// of 64, latents of 128, 256 and 512, 8 to 128 heads); attention_latent.cu has the formulas, attention_tcgen05.cu the
// scheme that this kernel follows.
//
// A block owns 128 rows, a row being (query token, head): all heads share the cache entries, so the rows of 128 / heads
// consecutive queries walk the same keys, 32 a tile.  Its scores take the whole entry (C + 64 numbers), its values
// at most 256 of the C latent numbers: a row's accumulator of 512 would fill tensor memory.  A latent of 512 therefore
// has two blocks for the same rows, each with all of the scores and half of the values (half as many products again,
// and nothing to exchange).
//
//   loader  (warp 0)    a tile is (C + 64) / 64 sub-tiles of 32 keys x 64 numbers (128-byte swizzle), each one box of the
//                       pool's tensor map per page, four tiles ahead at most; they are the keys and, as an N-major operand, the
//                       values.
//   issuer  (warp 1)    S = Q E^T (128 x 32) of the next tile into one of two score buffers, then O += P E of this one (P
//                       from tensor memory).
//   softmax (warps 2-5) a thread a row, as in attention_tcgen05.cu: lazily moved reference, probabilities over the scores.
//
// At a latent of 512 three quarters of a query lie in tensor memory: all of it in shared memory (147 KB) would leave room for
// two tiles of keys only.  A probability is two bfloat16 numbers (its rounding and the rest): with one, the reference that
// is not the maximum itself made the result's error 3 % larger than the mma.sync kernel's; with two it is 15 % smaller (rms
// against 64 bits over prompts of 130 to 1,300: 2.43e-4, mma.sync 2.87e-4).
//
// What bounds it: a product of 128 x 32 takes some 64 cycles although it has the work of 16, and a tile 36 of them and four
// of P E: 1.57 us a tile.  (A pair of CTAs would halve them: tiles of 64 keys at the same shared memory.)  Measured on B200
// beside the mma.sync kernel, 16 heads, latent 512: prompts of 1,300, 910, 520 and 130 within a window of 1,024 197 against
// 367 us; 2,048 causal 230 against 462; 256 queries over 8,000 keys 393 against 903; portions of 5, 2 and 9 behind contexts of
// up to 1,300 60 against 125; latent 256, twice 1,000: 59 against 174.  What it does before its first tile takes longer, though:
// see `worth`.  The products issued by the whole
// warp with one lane's predicate: 269 to 209 us together with the rotated parts asked for all at once.
#pragma once

#include "attention_mma.cuh"
#include "tcgen05.cuh"

namespace li {
namespace latent_tc {

constexpr int kRows = 128, kKeys = 32, kThreads = 192, kRot = 64;
constexpr int kMinHeads = 8;             // as many as keep the table of cosines (queries x 32 pairs) at 4 KB
constexpr float kLazyLog2 = 8.f;         // how far (in powers of two) a row's maximum may outgrow the reference of its exponentials
constexpr unsigned kSubBytes = kKeys * 64 * 2, kRowSubBytes = kRows * 64 * 2;

struct Params {
  const bf16* q_lat; long q_lat_head_stride; int q_lat_token_stride;
  const bf16* q_raw; int q_raw_token_stride, q_raw_head_stride, q_rot_off;
  bf16* out; long out_head_stride; int out_token_stride;
  const int* block_table; int table_stride;
  const int* query_start_loc; const int* context_lens; const int* seq_index;
  const float* inv_freq; const float* sink;
  int heads, rot_dims, page_size, page_shift, num_pages;
  float scale_log2;
  int window;
  float cs_scale;
  int* error_flag;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// A wait that gave up ends a warp's loop for all of its lanes.
__device__ __forceinline__ bool whole_warp(bool got) { return __all_sync(0xffffffffu, got) != 0; }

// Products and commits of the one lane whose `leader` is not zero, in code that the whole warp runs.
__device__ __forceinline__ void product(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned leader, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(leader) : "memory");
}
__device__ __forceinline__ void product_ts(unsigned d, unsigned a, unsigned long long b, unsigned idesc, unsigned leader, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(leader) : "memory");
}
__device__ __forceinline__ void commit(unsigned bar, unsigned leader) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
               "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(leader) : "memory");
}

template <int C>
struct Sizes {
  static constexpr int kParts = C > 256 ? 2 : 1;            // blocks that share a row's values
  static constexpr int kVal = C / kParts, kValSubs = kVal / 64, kSubs = C / 64 + 1;
  static constexpr int kTmemSubs = C > 256 ? 6 : 0;         // sub-tiles of the queries in tensor memory, 32 columns each
  static constexpr int kStages = 4;
  static constexpr unsigned kStageBytes = kSubs * kSubBytes;
  static constexpr size_t q_bytes = (size_t)(kSubs - kTmemSubs) * kRowSubBytes;
  static constexpr size_t table_bytes = (size_t)(kRows / kMinHeads) * (kRot / 2) * 2 * 4;
  static constexpr size_t total = 1024 + q_bytes + kStages * (size_t)kStageBytes + table_bytes + 8 * (2 * kStages + 8) + 16;
  static_assert(total <= 232448, "more shared memory than a block may have");
};

template <int C>
__global__ void __launch_bounds__(kThreads, 1)
latent_attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map, const Params p) {
  using S = Sizes<C>;
  constexpr int kStages = S::kStages, kSubs = S::kSubs, kValSubs = S::kValSubs, kTmemSubs = S::kTmemSubs;
  constexpr unsigned kStageBytes = S::kStageBytes;
  extern __shared__ unsigned char smem_raw[];
  const unsigned base = (smem_addr(smem_raw) + 1023u) & ~1023u;
  unsigned char* generic_base = smem_raw + (base - smem_addr(smem_raw));
  const unsigned q_smem = base, k_smem = base + (unsigned)S::q_bytes;
  float2* turn = reinterpret_cast<float2*>(generic_base + S::q_bytes + kStages * kStageBytes);     // [queries][pairs] (cos, sin)
  const unsigned bars = k_smem + kStages * kStageBytes + (unsigned)S::table_bytes;
  auto kv_full = [&](int s) { return bars + 8u * s; };
  auto kv_empty = [&](int s) { return bars + 8u * (kStages + s); };
  auto s_full = [&](int b) { return bars + 8u * (2 * kStages + b); };
  auto p_full = [&](int b) { return bars + 8u * (2 * kStages + 2 + b); };
  auto pv_done = [&](int b) { return bars + 8u * (2 * kStages + 4 + b); };
  const unsigned drained = bars + 8u * (2 * kStages + 6);
  const unsigned tmem_slot = bars + 8u * (2 * kStages + 8);

  grid_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seq = p.seq_index ? p.seq_index[blockIdx.y] : blockIdx.y;
  if (seq < 0) return;        // a place of padding in the list of sequences
  const int part = blockIdx.x;
  const int q_begin = p.query_start_loc[seq], q_len = p.query_start_loc[seq + 1] - q_begin;
  const int tq = kRows / p.heads;
  // The last queries see the most keys: they are handed out first, across all sequences.
  const int q0 = (int)(gridDim.z - 1 - blockIdx.z) * tq;
  if (q0 >= q_len) return;
  const int ctx = p.context_lens[seq];
  const int* table = p.block_table + (size_t)seq * p.table_stride;
  const int tile_q = min(tq, q_len - q0), rows_used = tile_q * p.heads;
  const int first_qpos = ctx - q_len + q0, last_qpos = first_qpos + tile_q - 1;
  const int hi = last_qpos + 1;
  const int lo = p.window > 0 ? max(first_qpos - p.window + 1, 0) : 0;
  const int tile_lo = lo / kKeys, ntiles = (hi + kKeys - 1) / kKeys - tile_lo;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * kStages; ++s) mbar_init(bars + 8u * s, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(s_full(b), 1);
      mbar_init(p_full(b), 4);
      mbar_init(pv_done(b), 1);
    }
    mbar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  constexpr unsigned kTmemCols = 512;      // two score buffers of 32 columns, up to 192 of queries, the accumulator from column 256 on
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // The rotation's cosines and sines, a query and pair each (what the step itself brings, not the kernel ahead).
  const int half = p.rot_dims / 2;
  if (warp > 1)
    for (int i = threadIdx.x - 64; i < tile_q * half; i += 128) {
      const float angle = __fmul_rn((float)(first_qpos + i / half), p.inv_freq[i % half]);
      turn[(i / half) * (kRot / 2) + i % half] = make_float2(cosf(angle) * p.cs_scale, sinf(angle) * p.cs_scale);
    }
  // (What follows needs the table of cosines, the barriers and the place in tensor memory.)
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  unsigned tmem_base;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem_base) : "r"(tmem_slot));
  auto tmem_s = [&](int b) { return tmem_base + 32u * b; };
  const unsigned tmem_q = tmem_base + 64u, tmem_o = tmem_base + 256u;
  grid_dependency_wait();   // the queries and the newest entries come from kernels ahead

  // The loader's warp: lane i brings box i % boxes of sub-tile i / boxes.  The block table's entries are in the warp's
  // registers, 32 at a time, the next 32 on their way; a tile's pages lie in one run of 32.
  const int box_rows = min(p.page_size, kKeys), boxes = kKeys / box_rows;
  const unsigned box_bytes = (unsigned)box_rows * 64 * 2;
  int chunk = -1, entries = -1, entries_ahead = -1;
  auto table_chunk = [&](int c) { return c * 32 + lane < p.table_stride ? table[c * 32 + lane] : -1; };
  auto load_tile = [&](int t) -> bool {
    const int stage = t % kStages;
    const unsigned phase = (unsigned)(t / kStages) & 1;
    const int key0 = (tile_lo + t) * kKeys, box = lane % boxes, sub = lane / boxes;
    const int first_page = key0 >> p.page_shift;
    if ((first_page >> 5) != chunk) {
      entries = (first_page >> 5) == chunk + 1 && chunk >= 0 ? entries_ahead : table_chunk(first_page >> 5);
      chunk = first_page >> 5;
      entries_ahead = table_chunk(chunk + 1);
    }
    const int page = __shfl_sync(0xffffffffu, entries, (first_page + box) & 31);
    const int kpos = key0 + box * box_rows;
    const bool wanted = sub < kSubs && kpos < hi && kpos + box_rows > lo && page >= 0 && page < p.num_pages;
    const int row = page * p.page_size + (kpos & (p.page_size - 1));
    const int count = __popc(__ballot_sync(0xffffffffu, wanted));
    bool fine = true;
    if (lane == 0) {
      if (t >= kStages) fine = mbar_wait(kv_empty(stage), phase ^ 1, p.error_flag, 41);
      if (fine) mbar_expect_tx(kv_full(stage), count * box_bytes);
    }
    fine = __shfl_sync(0xffffffffu, fine, 0);
    if (!fine) return false;
    if (wanted) tma_load_2d(k_smem + stage * kStageBytes + sub * kSubBytes + box * box_bytes, &map, kv_full(stage), sub * 64, row);
    return true;
  };
  const int tiles_ahead = min(kStages, ntiles);
  if (warp == 0) {
    __syncwarp();
    for (int t = 0; t < tiles_ahead; ++t) load_tile(t);
  }
  // The rows: row r is head r % heads of query q0 + r / heads, [absorbed query | rotated part]; rows of padding are zero.
  if (warp > 1) {
    // The first sub-tiles go to tensor memory, where the products read them without a trip through shared memory: a thread
    // brings its row's, three at a time.  The others lie in shared memory, swizzled.
    const int row0 = (warp & 3) * 32, own = row0 + lane, own_query = own / p.heads, own_head = own - own_query * p.heads;
    const bool own_used = own < rows_used;
    const uint4* src = reinterpret_cast<const uint4*>(p.q_lat + (own_used ? (size_t)own_head * p.q_lat_head_stride +
                                                                 (size_t)(q_begin + q0 + own_query) * p.q_lat_token_stride : 0));
    // The rotated part, a row at a time by the whole warp: lane j turns pair j where there is one, what does not turn (from
    // 2 * half on) is dealt to the other lanes.  Asked for first, so that it is on its way together with the rest.
    bf16 raw_a[32], raw_b[32];
    const int row0_query = row0 / p.heads, row0_head = row0 - row0_query * p.heads;
    {
      const bf16* from = p.q_raw + (size_t)(q_begin + q0) * p.q_raw_token_stride + p.q_rot_off;
      const int at_a = lane < half ? lane : lane + half, at_b = lane + (lane < half ? half : 32);
      int query = row0_query, head = row0_head;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const bool used = row0 + i < rows_used;
        const bf16* src = from + (used ? (size_t)query * p.q_raw_token_stride + (size_t)head * p.q_raw_head_stride : 0);
        raw_a[i] = src[at_a];
        raw_b[i] = src[at_b];
        if (++head == p.heads) { head = 0; ++query; }
      }
    }
#pragma unroll
    for (int i = 0; i < C / 64 - kTmemSubs; ++i)
#pragma unroll
      for (int c = 0; c < 8; ++c)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(q_smem + i * kRowSubBytes + own * 128 + ((c ^ (own & 7)) << 4)),
                     "l"(src + (kTmemSubs + i) * 8 + c), "r"(own_used ? 16 : 0));
    constexpr int kBatch = 3;
#pragma unroll
    for (int i = 0; i < kTmemSubs; i += kBatch) {
      uint4 v[kBatch][8];
#pragma unroll
      for (int j = 0; j < kBatch; ++j)
#pragma unroll
        for (int c = 0; c < 8; ++c) v[j][c] = own_used ? src[(i + j) * 8 + c] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        unsigned w[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          w[4 * c] = v[j][c].x; w[4 * c + 1] = v[j][c].y; w[4 * c + 2] = v[j][c].z; w[4 * c + 3] = v[j][c].w;
        }
        __syncwarp();
        tmem_store32(tmem_q + ((unsigned)row0 << 16) + (i + j) * 32, w);
      }
    }
    tmem_store_wait();
    auto put = [&](int r, int d, float v) {
      *reinterpret_cast<bf16*>(generic_base + (C / 64 - kTmemSubs) * kRowSubBytes + r * 128 + (((d >> 3) ^ (r & 7)) << 4) + (d & 7) * 2) = __float2bfloat16_rn(v);
    };
    int turn_query = row0_query, turn_head = row0_head;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int r = row0 + i;
      const bool used = r < rows_used;
      const float a = to_float(raw_a[i]), b = to_float(raw_b[i]);
      if (lane < half) {
        const float2 cs = turn[(used ? turn_query : 0) * (kRot / 2) + lane];
        put(r, lane, used ? rotate_lo(a, b, cs.x, cs.y) : 0.f);
        put(r, lane + half, used ? rotate_hi(a, b, cs.x, cs.y) : 0.f);
      } else {
        put(r, lane + half, used ? a : 0.f);
        put(r, lane + 32, used ? b : 0.f);
      }
      if (++turn_head == p.heads) { turn_head = 0; ++turn_query; }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    fence_async_shared();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();

  if (warp == 0) {
    // ------------------------------------------------------------------ loader
    int asked = tiles_ahead;
    while (asked < ntiles && load_tile(asked)) ++asked;
    // Every copy that was asked for has landed before the block ends, also where a wait gave up.
    for (int t = max(0, asked - kStages); t < asked; ++t) mbar_wait(kv_full(t % kStages), (unsigned)(t / kStages) & 1, nullptr, 0);
  } else if (warp == 1) {
    // ------------------------------------------------------------------ issuer
    // The whole warp walks the tiles and one lane's products are issued: descriptors can then stay in uniform registers.
    {
      const unsigned leader = lane == 0;
      // f32 accumulate, bf16 x bf16, M 128, N 32; for P E the second operand is N-major and N the values.
      constexpr unsigned idesc_any = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(kRows >> 4) << 24);
      constexpr unsigned idesc_qk = idesc_any | ((unsigned)(kKeys >> 3) << 17);
      constexpr unsigned idesc_pv = idesc_any | (1u << 16) | ((unsigned)(S::kVal >> 3) << 17);
      const unsigned long long desc_q = umma_desc(q_smem), desc_k = umma_desc(k_smem);
      // The values' sub-tiles of 64 numbers lie kSubBytes apart, which the descriptor's leading offset says.
      const unsigned long long desc_v = (umma_desc(k_smem + part * kValSubs * kSubBytes) & ~(0x3fffULL << 16)) |
                                        ((unsigned long long)((kSubBytes >> 4) & 0x3fff) << 16);
      // S of tile t may overwrite its buffer: see attention_tcgen05.cu.
      auto issue_qk = [&](int t) -> bool {
        const int stage = t % kStages, buf = t & 1;
        const unsigned phase = (unsigned)(t / kStages) & 1;
        const unsigned long long dk = desc_k + (unsigned long long)((stage * kStageBytes) >> 4);
        if (!whole_warp(mbar_wait(kv_full(stage), phase, p.error_flag, 43))) return false;
        tcgen05_fence_after();
#pragma unroll
        for (int k = 0; k < kTmemSubs * 4; ++k)
          product_ts(tmem_s(buf), tmem_q + k * 8u, dk + (unsigned long long)(((k / 4) * kSubBytes + (k % 4) * 32) >> 4), idesc_qk, leader, k > 0);
#pragma unroll
        for (int k = 0; k < (kSubs - kTmemSubs) * 4; ++k)
          product(tmem_s(buf), desc_q + (unsigned long long)(((k / 4) * kRowSubBytes + (k % 4) * 32) >> 4),
                  dk + (unsigned long long)(((kTmemSubs + k / 4) * kSubBytes + (k % 4) * 32) >> 4), idesc_qk, leader, kTmemSubs > 0 || k > 0);
        commit(s_full(buf), leader);
        return true;
      };
      bool ok = ntiles > 0 && issue_qk(0);
      for (int t = 0; ok && t < ntiles; ++t) {
        if (t + 1 < ntiles && !issue_qk(t + 1)) { ok = false; break; }
        const int stage = t % kStages, buf = t & 1;
        if (!whole_warp(mbar_wait(p_full(buf), (unsigned)(t >> 1) & 1, p.error_flag, 45))) { ok = false; break; }
        tcgen05_fence_after();
        const unsigned long long dv = desc_v + (unsigned long long)((stage * kStageBytes) >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k)       // the probabilities' first 16 bits, then what they leave
          product_ts(tmem_o, tmem_s(buf) + k * 8u, dv + (unsigned long long)(((k & 1) * 16 * 128) >> 4), idesc_pv, leader, t > 0 || k > 0);
        commit(kv_empty(stage), leader);
        commit(pv_done(buf), leader);
      }
      // Products are done before tensor memory goes back, also where a wait gave up.
      commit(drained, leader);
      mbar_wait(drained, 0, nullptr, 0);
    }
  } else {
    // ---------------------------------------------------------------- softmax
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const unsigned lane_field = (unsigned)(quarter * 32) << 16;
    const int query = row / p.heads, head = row - query * p.heads;
    const int qpos = row < rows_used ? first_qpos + query : -1;
    float m = -INFINITY, l = 0.f;      // the reference of the exponentials (scores times the scale), their sum
    bool ok = true;
    for (int t = 0; ok && t < ntiles; ++t) {
      const int buf = t & 1, stage = t % kStages, key0 = (tile_lo + t) * kKeys;
      if (!whole_warp(mbar_wait(s_full(buf), (unsigned)(t >> 1) & 1, p.error_flag, 46))) { ok = false; break; }
      tcgen05_fence_after();
      unsigned s[32];
      __syncwarp();
      tmem_load32(tmem_s(buf) + lane_field, s);
      tmem_load_wait();
      float x[32];
      float part_max[4] = {m, m, m, m};
      const bool all_visible = key0 + kKeys - 1 <= first_qpos && (p.window <= 0 || key0 > last_qpos - p.window);
      if (all_visible && qpos >= 0) {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(s[j]) * p.scale_log2;
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int key = key0 + j;
          x[j] = key <= qpos && (p.window <= 0 || key > qpos - p.window) ? __uint_as_float(s[j]) * p.scale_log2 : -INFINITY;
        }
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) part_max[j & 3] = fmaxf(part_max[j & 3], x[j]);
      const float mx = fmaxf(fmaxf(part_max[0], part_max[1]), fmaxf(part_max[2], part_max[3]));
      float m_new = m, alpha = 1.f;
      if (mx - m > kLazyLog2) {       // also when m is still -inf and a score is not
        m_new = mx;
        alpha = ex2(m - mx);
      }
      const bool rescale = alpha != 1.f && m != -INFINITY;   // a row that has seen no key yet holds zeros
      const float ref = m_new == -INFINITY ? 0.f : m_new;
      float sums[4] = {0.f, 0.f, 0.f, 0.f};
      // A probability is kept as two bfloat16 numbers, its rounding and what that leaves: the second half of the
      // products costs two steps of forty, and a probability is exact to 2^-17.
      unsigned packed[32];
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const float e0 = ex2(x[2 * c] - ref), e1 = ex2(x[2 * c + 1] - ref);
        sums[c & 3] += e0 + e1;
        __nv_bfloat162 h = __floats2bfloat162_rn(e0, e1);
        packed[c] = *reinterpret_cast<unsigned*>(&h);
        h = __floats2bfloat162_rn(e0 - __uint_as_float(packed[c] << 16), e1 - __uint_as_float(packed[c] & 0xffff0000u));
        packed[16 + c] = *reinterpret_cast<unsigned*>(&h);
      }
      tmem_store32(tmem_s(buf) + lane_field, packed);
      // The accumulator may be rescaled only between P E of tile t - 1 and that of this tile, which waits for this warp.
      if (t >= 1 && __any_sync(0xffffffffu, rescale)) {
        if (!whole_warp(mbar_wait(pv_done((t - 1) & 1), (unsigned)((t - 1) >> 1) & 1, p.error_flag, 47))) { ok = false; break; }
        tcgen05_fence_after();
        unsigned o[32];
#pragma unroll 1
        for (int i = 0; i < S::kVal / 32; ++i) {
          __syncwarp();
          tmem_load32(tmem_o + lane_field + i * 32, o);
          tmem_load_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_store32(tmem_o + lane_field + i * 32, o);
        }
      }
      tmem_store_wait();
      m = m_new;
      l = l * alpha + (sums[0] + sums[1]) + (sums[2] + sums[3]);
      // Values of keys outside [lo, hi) may hold anything (an unwritten slot): zeros before P E reads them.
      if (key0 < lo || key0 + kKeys > hi) {
        if (!whole_warp(mbar_wait(kv_full(stage), (unsigned)(t / kStages) & 1, p.error_flag, 48))) { ok = false; break; }
        unsigned char* vt = generic_base + S::q_bytes + stage * kStageBytes + part * kValSubs * kSubBytes;
        for (int e = threadIdx.x - 64; e < kValSubs * kKeys * 8; e += 128) {
          const int sub = e / (kKeys * 8), key = (e >> 3) % kKeys, kpos = key0 + key;
          if (kpos < lo || kpos >= hi)
            *reinterpret_cast<uint4*>(vt + sub * kSubBytes + key * 128 + ((e & 7) << 4)) = make_uint4(0, 0, 0, 0);
        }
        fence_async_shared();
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(buf));
    }
    ok = ok && (ntiles <= 0 || mbar_wait(pv_done((ntiles - 1) & 1), (unsigned)((ntiles - 1) >> 1) & 1, p.error_flag, 49));
    tcgen05_fence_after();
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      if (p.sink != nullptr && row < rows_used) l += exp2f(p.sink[head] * kLog2e - m);
      const float inv = l > 0.f ? 1.f / l : 0.f;
      bf16* dst = p.out + (size_t)head * p.out_head_stride + (size_t)(q_begin + q0 + query) * p.out_token_stride + part * S::kVal;
#pragma unroll 1
      for (int i = 0; i < S::kVal / 32; ++i) {
        unsigned o[32];
        __syncwarp();
        tmem_load32(tmem_o + lane_field + i * 32, o);
        tmem_load_wait();
        if (row < rows_used) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            unsigned w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float a = ntiles > 0 ? __uint_as_float(o[v * 8 + 2 * e]) * inv : 0.f;
              const float b = ntiles > 0 ? __uint_as_float(o[v * 8 + 2 * e + 1]) * inv : 0.f;
              __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
              w[e] = *reinterpret_cast<unsigned*>(&h);
            }
            *reinterpret_cast<uint4*>(dst + i * 32 + v * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
}

// The pool [pages, 1, page_size, C + 64] as a map of entries; a box is 64 numbers of `box_rows` entries of one page.
inline bool make_entry_map(CUtensorMap* map, const void* pool, long rows, int box_rows, int entry) {
  EncodeTiledFn encode = encode_tiled();
  if (!encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)entry, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)entry * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, elem[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(pool), dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether the kernel takes a launch over sequences of up to max_q_len queries.
inline bool takes(const Params& p, const void* pool, int num_seqs, int max_q_len, int kv_rank, int rot_dim) {
  return (kv_rank == 128 || kv_rank == 256 || kv_rank == 512) && rot_dim == kRot && p.heads >= kMinHeads && p.heads <= kRows &&
         (p.page_size == 16 || p.page_size == 32 || p.page_size == 64) && max_q_len > 1 &&
         max_q_len / (kRows / p.heads) < 65535 && num_seqs <= 65535 && (p.out_token_stride % 8) == 0 &&
         (p.out_head_stride % 8) == 0 && aligned16(p.out) && aligned16(pool);
}

// Whether it is the faster one there.  Contexts of at most two tiles (`max_context`, 0: not known) it has no use for its faster
// walk: 16 heads of a latent of 512 over one prompt of 16 tokens take 16.0 us here and 13.9 on the mma.sync kernel, eight of 30
// 17.4 and 15.1, sixteen of 33 30.2 and 15.9; 8 heads and eight prompts of 30 18.0 and 11.7; 64 tokens are even.  Unless the
// mma.sync kernel's blocks, of four queries and sixteen heads, need more rounds of the device's SMs: 8 heads and sixteen prompts
// of 64 18.5 and 29.3.
constexpr int kShortContext = 2 * kKeys;
inline bool worth(const Params& p, int num_seqs, int max_q_len, int kv_rank, int max_context) {
  if (max_context <= 0 || max_context > kShortContext) return true;
  const int tq = kRows / p.heads;
  const long here = (long)num_seqs * ((max_q_len + tq - 1) / tq) * (kv_rank > 256 ? 2 : 1);
  const long there = (long)num_seqs * ((max_q_len + 3) / 4) * ((p.heads + 15) / 16);
  return (here + 147) / 148 < (there + 147) / 148;
}

template <int C>
int launch(const Params& p, const CUtensorMap& map, int num_seqs, int max_q_len, cudaStream_t stream) {
  using S = Sizes<C>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(latent_attention_tcgen05_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::total);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int tq = kRows / p.heads;
  const dim3 grid(S::kParts, num_seqs, (max_q_len + tq - 1) / tq);
  return (int)launch_pdl(0, latent_attention_tcgen05_kernel<C>, grid, dim3(kThreads), S::total, stream, map, p);
}

}  // namespace latent_tc
}  // namespace li
