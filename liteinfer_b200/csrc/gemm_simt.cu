// out[M, N] = x[M, K] @ w[N, K]^T (+ bias[N]) in plain FFMA code with 32-bit
// accumulation: the matrix product of the true 32-bit path (tensor cores have no
// full-precision 32-bit mode), also instantiated for bfloat16 storage as the path
// for shapes the tensor-core kernels refuse.
//
// Every output element adds its K products in the same order whatever M and N are, so a row's result does not depend on
// which other rows are in the batch: chunks of 128 k, each two chains of fused multiply-adds in ascending order from zero, of its
// even and its odd k, (which the wide kernel's instruction takes side by side); their sum; and the chunks' sums in ascending order.  Both kernels
// keep that order; the chunks are what lets the narrow one give each to a warp of its own (and the sum of short chains is nearer to
// the exact one: relative error of a product over 768 k 1.55e-7, 2.1e-7 with one chain a chunk).  In bfloat16, where there is the wide
// kernel only, a chunk is one chain.
#include <type_traits>

#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace li {

constexpr int kChunk = 128;

// Two sums side by side, of the even and of the odd k: one instruction multiplies and adds for both.
typedef unsigned long long Pair;
__device__ __forceinline__ Pair multiply_add(Pair a, Pair b, Pair sums) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sums) : "l"(a), "l"(b));
  return sums;
}
__device__ __forceinline__ float both(Pair sums) {
  return __uint_as_float((unsigned)sums) + __uint_as_float((unsigned)(sums >> 32));
}
__device__ __forceinline__ float both(float sum) { return sum; }

struct SimtProduct {
  const void *x, *w, *bias;
  void* out;
  int M, N, K, ldx, ldo;
  long x_batch, w_batch, out_batch;     // one product per blockIdx.z (a plain product is a batch of one)
  bool w_at_rest;       // nothing that is still under way writes w
};

// ---- many rows of x: 64 x 64 tiles, 8 x 4 outputs a thread -------------------------------------------------------
// Bound by shared memory's reads: four k are 64 two-wide multiply-adds a thread on 12 vector loads, and a warp's vector load takes four
// cycles where its multiply-adds take 32 in all.  Rows lie along k in both operands (threads have rows 8 and 16 apart, which with
// rows of 36 words keeps the reads off one another's banks), so two neighbours along k are a pair as they are loaded.  Three steps
// of 32 k are on their way (cp.async) while a fourth is multiplied.  Three blocks of four warps an SM: blocks of this size spread a
// grid of a few hundred over the SMs more evenly than 128 x 64 (1,250 rows of 1280 x 768: 78 us, 97), and half the
// multiply-adds' instructions leave the issue slots to the loads.
// Measured on B200, 1,250 rows: 768 x 2048 132 us (145 with reads just ahead of their use), 4096 x 768 204 us (39 TFLOP/s; 232 in
// tiles of 128 x 64 with one-wide multiply-adds); 400 rows of 768 x 768 33 (37), 256 of 16000 x 768 160 (169).
//
// bfloat16 is widened on its way to shared memory, by loads that a thread waits for: what counts is how many threads do that, and a
// launch's tiles are 128 x 64 (or 64 or 32 x 64) by eight warps, with one-wide multiply-adds in fewer registers, two blocks an SM.  100 rows
// of 4096 x 4096 238 us, 390 by blocks of four warps as above; 12 rows of 2048 x 2048 94 and 99.
constexpr int BN = 64, BK = 32, kTileStages = 4;
template <typename T> constexpr int kTileThreads = sizeof(T) == 4 ? 128 : 256;
constexpr int kTileRow = BK + 4;
template <int BM> constexpr size_t kTileSmem = (size_t)kTileStages * (BM + BN) * kTileRow * sizeof(float);

__device__ __forceinline__ void copy16_async(float* dst, const float* src, int bytes = 16) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes));
}

__device__ __forceinline__ void copy4_async(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}

// Four neighbours along k, `left` of which exist, to shared memory: at once where `vec` (the row lies on 16 bytes).  (What does not
// exist is filled with zeros; the address is then the row's last number's.)  32-bit numbers go asynchronously either way: 3,000 rows
// of 5000 x 770 740 us, 859 when a thread waited for its four, 300 rows of 3072 x 2049 171 and 209.
__device__ __forceinline__ void stage_four(float* dst, const float* src, int left, bool vec) {
  if (vec) {
    copy16_async(dst, left > 0 ? src : src - (4 - left) / 4 * 4, left > 0 ? 16 : 0);   // K is a multiple of four
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) copy4_async(dst + i, src + min(i, left - 1), i < left ? 4 : 0);
}
__device__ __forceinline__ void stage_four(float* dst, const bf16* src, int left, bool vec) {
  if (vec && left > 0) {
    const uint2 raw = *reinterpret_cast<const uint2*>(src);
    *reinterpret_cast<float4*>(dst) = make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                                                  __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) dst[i] = i < left ? widen(src[i]) : 0.f;
}

template <typename T, int BM>
__global__ void __launch_bounds__(kTileThreads<T>, sizeof(T) == 4 ? 3 : 2) gemm_simt_tile_kernel(SimtProduct p, bool vec) {
  constexpr int kThreads = kTileThreads<T>, kApart = kThreads / 16, kRows = BM / kApart;      // a thread's rows of x: kRows, kApart apart
  extern __shared__ __align__(16) float tile_smem[];      // [stage][x rows, then w rows][kTileRow]
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, K = p.K;
  const T* x = static_cast<const T*>(p.x) + blockIdx.z * p.x_batch;
  const T* w = static_cast<const T*>(p.w) + blockIdx.z * p.w_batch;
  T* out = static_cast<T*>(p.out) + blockIdx.z * p.out_batch;
  const T* bias = static_cast<const T*>(p.bias);
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int steps = (K + BK - 1) / BK;
  const int lr = threadIdx.x / 8, lk = threadIdx.x % 8 * 4;   // the first row and the k of this thread's loads

  // Rows beyond a matrix repeat its last one: their outputs are not stored.
  const auto fill = [&](int step) {
    if (step < steps) {
      float* dst = tile_smem + (step % kTileStages) * ((BM + BN) * kTileRow) + lr * kTileRow + lk;
      const int k = step * BK + lk, left = K - k;
#pragma unroll
      for (int r = 0; r < BM; r += kThreads / 8)
        stage_four(dst + r * kTileRow, x + (size_t)min(m0 + lr + r, p.M - 1) * p.ldx + k, left, vec);
#pragma unroll
      for (int r = 0; r < BN; r += kThreads / 8)
        stage_four(dst + (BM + r) * kTileRow, w + (size_t)min(n0 + lr + r, p.N - 1) * K + k, left, vec);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  using Sum = std::conditional_t<sizeof(T) == 4, Pair, float>;
  Sum acc[kRows][4];
  float total[kRows][4];
#pragma unroll
  for (int i = 0; i < kRows; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0, total[i][j] = 0.f;

  for (int step = 0; step < kTileStages - 1; ++step) fill(step);
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kTileStages - 2) : "memory");
    __syncthreads();                   // this step's operands are in place, and everyone is done with the step before
    fill(step + kTileStages - 1);      // into the stage of the step before
    const float* stage = tile_smem + (step % kTileStages) * ((BM + BN) * kTileRow);
    const float* xr = stage + ty * kTileRow;
    const float* wr = stage + (BM + tx) * kTileRow;
    if constexpr (sizeof(T) == 4) {
      // (The next four k are read while these are multiplied.)
      const auto read = [&](int k, ulonglong2 (&a)[kRows], ulonglong2 (&b)[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(wr + j * 16 * kTileRow + k);
#pragma unroll
        for (int i = 0; i < kRows; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xr + i * kApart * kTileRow + k);
      };
      ulonglong2 a[kRows], b[4];
      read(0, a, b);
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
        ulonglong2 next_a[kRows], next_b[4];
        if (k + 4 < BK) read(k + 4, next_a, next_b);
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = multiply_add(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = multiply_add(a[i].y, b[j].y, acc[i][j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = next_b[j];
#pragma unroll
        for (int i = 0; i < kRows; ++i) a[i] = next_a[i];
      }
    } else {
#pragma unroll 2
      for (int k = 0; k < BK; k += 4) {
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(wr + j * 16 * kTileRow + k);
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(xr + i * kApart * kTileRow + k);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[i][j] = fmaf(a.w, b[j].w, fmaf(a.z, b[j].z, fmaf(a.y, b[j].y, fmaf(a.x, b[j].x, acc[i][j]))));
        }
      }
    }
    if ((step + 1) * BK % kChunk == 0 || step + 1 == steps) {
#pragma unroll
      for (int i = 0; i < kRows; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          total[i][j] += both(acc[i][j]);
          acc[i][j] = 0;
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < kRows; ++i) {
    const int m = m0 + ty + kApart * i;
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= p.N) continue;
      float v = total[i][j];
      if (bias) v += to_float(bias[n]);
      out[(size_t)m * p.ldo + n] = from_float<T>(v);
    }
  }
}

// ---- few rows of x (float32): 64 rows of w and one chunk of k a warp -----------------------------------------------
// Bound by reading w (a decode step) and by how much of it is on its way at once: a block copies all of its w, 64 rows of
// one to four chunks, to shared memory before it multiplies anything, and the chunks of a row lie in different warps and
// blocks.  A w that is a model's parameter (`w_at_rest`) it copies before it waits for the kernel ahead, which only x depends on
// then; any other w may be what that kernel is writing, and is read behind the wait.  (Generating 24 tokens for 1, 4, 12 and 16
// sequences at six layers of 768: 5.9, 8.7, 13.4 and 14.6 ms with the early copy, 6.8, 9.9, 14.5 and 16.1 without.)  A lane has two rows of w; x is read as
// broadcasts, R rows a warp, G warps on the same chunk of w.  The chunks' sums meet in the shared memory of the blocks of a
// cluster (along k) and are added in order.
// Measured on B200, 12 rows: 1280 x 768 6.6 us, 768 x 2048 6.9, 16000 x 768 26 (1.9 TB/s); one row of 16384 x 2048 41 us
// (3.3 TB/s).  On the 64 x 64 tiles, a dozen blocks that waited for every 16 k, these took 55, 140, 99 and 252 us.
constexpr int kRowStride = kChunk + 4;     // 16-byte reads of 32 rows at the same k: off the banks' period
constexpr int kRowsN = 64;
constexpr int kMostCluster = 8, kMostChunks = 4, kMostEach = 16;     // blocks along k, chunks of a block at a time, chunks of a block

// Grid: (64 rows of w) x cluster, R * G rows of x, batch.  Block: `chunks` chunks of G warps, `rounds` times.
template <int R, int G>
__global__ void __launch_bounds__(32 * kMostChunks * G) gemm_simt_rows_kernel(SimtProduct p, int chunks, int rounds,
                                                                                          int all_chunks) {
  extern __shared__ __align__(16) float rows_smem[];
  grid_launch_dependents();
  cg::cluster_group cluster = cg::this_cluster();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, mine = warp / G, part = warp % G;
  const int n0 = blockIdx.x / ranks * kRowsN, m0 = blockIdx.y * (R * G);
  const float* x = static_cast<const float*>(p.x) + blockIdx.z * p.x_batch;
  const float* w = static_cast<const float*>(p.w) + blockIdx.z * p.w_batch;
  float* out = static_cast<float*>(p.out) + blockIdx.z * p.out_batch;
  const float* bias = static_cast<const float*>(p.bias);
  float* wt = rows_smem + mine * (kRowsN * kRowStride);
  float* xt = rows_smem + chunks * (kRowsN * kRowStride) + mine * (R * G * kChunk);
  float* sums = rows_smem + chunks * (kRowsN * kRowStride + R * G * kChunk);      // [rounds * chunks][R * G][kRowsN]
  const int rows_w = min(kRowsN, p.N - n0), rows_x = min(R * G, p.M - m0);
  static_assert(kChunk == 128, "a row of a chunk is one 16-byte piece a lane");
  if (!p.w_at_rest) grid_dependency_wait();
  for (int round = 0; round < rounds; ++round) {
    const int place = round * chunks + mine, k0 = (rank * rounds * chunks + place) * kChunk;
    const int fours = max(0, min(kChunk, p.K - k0)) / 4;
    if (round > 0) __syncthreads();        // the warps of a chunk are done with its operands
    // The G warps of a chunk copy its operands between them, a row at a time.
    if (lane < fours) {
#pragma unroll 8
      for (int r = part; r < rows_w; r += G)
        copy16_async(wt + r * kRowStride + 4 * lane, w + (size_t)(n0 + r) * p.K + k0 + 4 * lane);
    }
    if (round == 0) grid_dependency_wait();
    if (lane < fours) {
#pragma unroll 4
      for (int r = part; r < rows_x; r += G)
        copy16_async(xt + r * kChunk + 4 * lane, x + (size_t)(m0 + r) * p.ldx + k0 + 4 * lane);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float sum[R][2];
    const float4* w0 = reinterpret_cast<const float4*>(wt + lane * kRowStride);
    const float4* w1 = reinterpret_cast<const float4*>(wt + (lane + 32) * kRowStride);
    const float4* xr = reinterpret_cast<const float4*>(xt + part * R * kChunk);
    // Two warps on a chunk multiply two-wide (a chunk of 128 k is 32 steps, eight of them in flight): 16 rows 0.94 of the time one k at a time,
    // 8 rows 0.95, 12 0.99.  One warp's few rows take a k at a time, in flight four or eight: one row 0.83 of the time of two in flight, four 0.97.
    if constexpr (G == 2) {
      Pair pairs[R][2];
#pragma unroll
      for (int r = 0; r < R; ++r) pairs[r][0] = pairs[r][1] = 0;
      const ulonglong2 *p0 = reinterpret_cast<const ulonglong2*>(w0), *p1 = reinterpret_cast<const ulonglong2*>(w1),
                       *px = reinterpret_cast<const ulonglong2*>(xr);
#pragma unroll 8
      for (int f = 0; f < fours; ++f) {
        const ulonglong2 b0 = p0[f], b1 = p1[f];
#pragma unroll
        for (int r = 0; r < R; ++r) {        // rows beyond x or w hold what the memory held: their sums are not stored
          const ulonglong2 a = px[r * (kChunk / 4) + f];
          pairs[r][0] = multiply_add(a.y, b0.y, multiply_add(a.x, b0.x, pairs[r][0]));
          pairs[r][1] = multiply_add(a.y, b1.y, multiply_add(a.x, b1.x, pairs[r][1]));
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) sum[r][0] = both(pairs[r][0]), sum[r][1] = both(pairs[r][1]);
    } else {
      float acc[R][2][2];
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r][0][0] = acc[r][0][1] = acc[r][1][0] = acc[r][1][1] = 0.f;
#pragma unroll(R == 1 ? 8 : 4)
      for (int f = 0; f < fours; ++f) {
        const float4 b0 = w0[f], b1 = w1[f];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float4 a = xr[r * (kChunk / 4) + f];
          acc[r][0][0] = fmaf(a.z, b0.z, fmaf(a.x, b0.x, acc[r][0][0]));
          acc[r][0][1] = fmaf(a.w, b0.w, fmaf(a.y, b0.y, acc[r][0][1]));
          acc[r][1][0] = fmaf(a.z, b1.z, fmaf(a.x, b1.x, acc[r][1][0]));
          acc[r][1][1] = fmaf(a.w, b1.w, fmaf(a.y, b1.y, acc[r][1][1]));
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) sum[r][0] = acc[r][0][0] + acc[r][0][1], sum[r][1] = acc[r][1][0] + acc[r][1][1];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float* mine_sums = sums + (place * (R * G) + part * R + r) * kRowsN + lane;
      mine_sums[0] = sum[r][0];
      mine_sums[32] = sum[r][1];
    }
  }
  cluster.sync();
  for (int i = rank * blockDim.x + threadIdx.x; i < rows_x * kRowsN; i += ranks * blockDim.x) {
    const int m = i / kRowsN, n = i % kRowsN;
    if (n >= rows_w) continue;
    const int share = rounds * chunks;
    float total = 0.f;
#pragma unroll 4
    for (int c = 0; c < all_chunks; ++c)
      total += *cluster.map_shared_rank(sums + (c % share * (R * G) + m) * kRowsN + n, c / share);
    if (bias) total += bias[n0 + n];
    out[(size_t)(m0 + m) * p.ldo + n0 + n] = total;
  }
  cluster.sync();        // nobody leaves while another block reads its sums
}

// How a block walks its share of `each` chunks: as many at a time as its shared memory holds beside the sums of all of them.
struct RowsPlan {
  int chunks, rounds;
  size_t smem;
};
constexpr size_t kMostSmem = 227 * 1024;
constexpr RowsPlan rows_plan(int each, int rows) {
  RowsPlan plan = {};
  for (int most = kMostChunks; most > 0; --most) {
    plan.rounds = (each + most - 1) / most;
    plan.chunks = (each + plan.rounds - 1) / plan.rounds;
    plan.smem = sizeof(float) * plan.chunks * (size_t)(kRowsN * kRowStride + rows * (kChunk + plan.rounds * kRowsN));
    if (plan.smem <= kMostSmem) break;
  }
  return plan;
}
constexpr bool every_plan_fits(int rows) {
  for (int each = 1; each <= kMostEach; ++each)
    if (rows_plan(each, rows).smem > kMostSmem) return false;
  return true;
}

template <int R, int G>
int launch_rows(const SimtProduct& p, int batch, cudaStream_t stream) {
  static_assert(every_plan_fits(R * G), "a k that the narrow kernel is chosen for and that its shared memory does not hold");
  const int all_chunks = (p.K + kChunk - 1) / kChunk;
  const RowsPlan plan = rows_plan((all_chunks + kMostCluster - 1) / kMostCluster, R * G);
  const int rounds = plan.rounds, chunks = plan.chunks;
  const int ranks = (all_chunks + rounds * chunks - 1) / (rounds * chunks);
  const size_t smem = plan.smem;
  const long blocks = (long)((p.N + kRowsN - 1) / kRowsN) * ranks, groups = (p.M + R * G - 1) / (R * G);
  if (blocks > 0x7fffffffL || groups > 65535 || batch > 65535) return LI_ERR_UNSUPPORTED;
  const cudaError_t status =
      cudaFuncSetAttribute(gemm_simt_rows_kernel<R, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
  if (status != cudaSuccess) return (int)status;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3((unsigned)blocks, (unsigned)groups, batch);
  config.blockDim = dim3(32 * G * chunks);
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
  config.numAttrs = pdl_enabled(p.M) ? 2 : 1;
  return (int)cudaLaunchKernelEx(&config, gemm_simt_rows_kernel<R, G>, p, chunks, rounds, all_chunks);
}

constexpr int kMostTileRows = 65535 * 128;

template <typename T, int BM>
int launch_tiles(const SimtProduct& p, bool vec, int batch, cudaStream_t stream) {
  if (p.M > kMostTileRows || batch > 65535) return LI_ERR_UNSUPPORTED;
  const cudaError_t status =
      cudaFuncSetAttribute(gemm_simt_tile_kernel<T, BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem<BM>);
  if (status != cudaSuccess) return (int)status;
  // A grid has at most 65,535 tiles along the rows; more of them are another launch's.
  constexpr int kRowsOfGrid = 65535 * BM;
  for (int first = 0; first < p.M; first += kRowsOfGrid) {
    SimtProduct part = p;
    part.M = p.M - first < kRowsOfGrid ? p.M - first : kRowsOfGrid;
    part.x = static_cast<const T*>(p.x) + (size_t)first * p.ldx;
    part.out = static_cast<T*>(p.out) + (size_t)first * p.ldo;
    const dim3 grid((p.N + BN - 1) / BN, (part.M + BM - 1) / BM, batch);
    gemm_simt_tile_kernel<T, BM><<<grid, kTileThreads<T>, kTileSmem<BM>, stream>>>(part, vec);
    const cudaError_t launched = cudaGetLastError();
    if (launched != cudaSuccess) return (int)launched;
  }
  return 0;
}

// Which kernel, by what each was measured to take (B200, microseconds).  float32, the narrow one: 3.6 and 0.12 a row up to 16, and for
// every million weights 0.72 for one row, 0.85 for four, 1.4 for eight, 1.65 for twelve, 2.1 for every group of 16; a fifth more where k
// is more than 2,048.  Tiles take their waves of 148, a whole step each: per 768 k 2 and 12.4 a wave for tiles of 32 rows (a lone wave 17.8),
// 6.5 and 21 a wave for tiles of 64 (768 k, 140 tiles of 32 18.4, 156 27.7, 288 28.7, 300 39.5, 448 52.7, 640 64; of 64 rows 140 29.3, 156
// 48.9, 320 70, 448 91).  By a line through these 257 rows of 4096 x 768 went to 320 tiles of 64 rows, 96 us (59 in 576 of 32).
// Up to 16 rows of one product the narrow kernel is the faster wherever k is not short (16 of 16000 x 768: 29 and 40).
// bfloat16, whose blocks are two an SM: waves in pairs, of 32 rows 46 a pair and 34 for one over (a lone wave 35), of 64 rows 63 and 58 (46.5), of
// 128 rows 106 and 76 (68).  (Without tiles of 64 rows 300 of 2048 x 2048 took 202 us, 170 with them.)
constexpr int kMostRows = 256;
inline float rows_cost(const SimtProduct& p, int batch) {
  if (p.M <= 16 && p.K >= 256 && batch == 1) return 0.f;
  const float each = p.M == 1 ? 0.72f : p.M <= 4 ? 0.85f : p.M <= 8 ? 1.4f : p.M <= 12 ? 1.65f : 2.1f * ((p.M + 15) / 16);
  return 3.6f + 0.12f * (p.M < 16 ? p.M : 16) + 1e-6f * each * (p.K > 2048 ? 1.2f : 1.f) * (float)p.N * p.K * batch;
}
inline float tiles_cost(int dtype, const SimtProduct& p, int batch, int rows) {
  const float tiles = (float)((p.N + BN - 1) / BN) * ((p.M + rows - 1) / rows) * batch, depth = p.K / 768.f;
  const float waves = ceilf(tiles / 148.f);
  if (dtype != kFloat32) {
    const float two = floorf(waves / 2.f), over = waves - 2.f * two;
    const float cost = rows == 32 ? (waves <= 1.f ? 35.f : 46.f * two + 34.f * over) :
                       rows == 64 ? (waves <= 1.f ? 46.5f : 63.f * two + 58.f * over) : waves <= 1.f ? 68.f : 106.f * two + 76.f * over;
    return 1.5f + depth * cost;
  }
  if (rows == 32) return 1.5f + (waves <= 1.f ? 17.8f * depth : 2.f * depth + waves * (0.5f + 11.9f * depth));
  return 2.f + 6.5f * depth + waves * (0.45f + 20.6f * depth);
}

int launch_product(int dtype, const SimtProduct& p, int batch, cudaStream_t stream) {
  const size_t element = dtype == kFloat32 ? 4 : 2, four = 4 * element;
  // Loads of four k at once: every row of x and w starts on their size.
  const bool vec = p.K % 4 == 0 && p.ldx % 4 == 0 && p.x_batch % 4 == 0 && p.w_batch % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(p.x) % four == 0 && reinterpret_cast<uintptr_t>(p.w) % four == 0;
  const float small = tiles_cost(dtype, p, batch, 32), medium = tiles_cost(dtype, p, batch, 64);
  const float large = dtype == kFloat32 ? medium : tiles_cost(dtype, p, batch, 128);
  if (dtype == kFloat32 && vec && p.K > 0 && p.M <= kMostRows && p.K <= kMostEach * kMostCluster * kChunk &&
      batch <= 65535 && rows_cost(p, batch) < fminf(small, large)) {
    if (p.M == 1) return launch_rows<1, 1>(p, batch, stream);
    if (p.M <= 4) return launch_rows<4, 1>(p, batch, stream);
    if (p.M <= 8) return launch_rows<4, 2>(p, batch, stream);
    if (p.M <= 12) return launch_rows<6, 2>(p, batch, stream);
    return launch_rows<8, 2>(p, batch, stream);
  }
  const bool narrow = small < fminf(medium, large) && (p.M + 31) / 32 <= 65535;
  if (dtype == kFloat32) return narrow ? launch_tiles<float, 32>(p, vec, batch, stream) : launch_tiles<float, 64>(p, vec, batch, stream);
  if (narrow) return launch_tiles<bf16, 32>(p, vec, batch, stream);
  return medium < large ? launch_tiles<bf16, 64>(p, vec, batch, stream) : launch_tiles<bf16, 128>(p, vec, batch, stream);
}

}  // namespace li

using namespace li;

// w_at_rest: w is written by nothing that is still under way on the device (a model's parameter), so that it may be read before
// the kernel ahead in the stream is done.
LI_EXPORT int li_gemm_simt(int dtype, const void* x, const void* w, const void* bias, void* out, int M, int N, int K,
                           int w_at_rest, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  return launch_product(dtype, SimtProduct{x, w, bias, out, M, N, K, K, N, 0, 0, 0, w_at_rest != 0}, 1, stream);
}

// A batch of products: out[b][m][n] = sum_k x[b][m][k] * w[b][n][k], b < batch.  x[b] starts at x + b * x_batch
// with `ldx` elements between its rows, w[b] at w + b * w_batch (rows of K), out[b] at out + b * out_batch with
// `ldo` between rows: operands may be slices of wider tensors (a head's columns of a projection).
LI_EXPORT int li_gemm_simt_batched(int dtype, const void* x, const void* w, void* out, int M, int N, int K, int batch,
                                   int ldx, int ldo, long x_batch, long w_batch, long out_batch,
                                   int w_at_rest, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  return launch_product(dtype, SimtProduct{x, w, nullptr, out, M, N, K, ldx, ldo, x_batch, w_batch, out_batch, w_at_rest != 0},
                        batch, stream);
}
