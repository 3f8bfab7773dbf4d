// True 32-bit matrix product for the float32 path: C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]),
// plain FMA on the CUDA cores, no tensor-core mode of reduced precision.
// (The reference's float32 mode is cublasGemmEx with CUBLAS_COMPUTE_32F,
// kernels/cuda/kernels.cu:752-767.)
//
// K is cut into S segments, S a function of N and K alone (`segments`).  Of a segment, each output element accumulates the even and
// the odd k in two chains in ascending order (one packed fma.rn.f32x2, two rounded fused multiply-adds; k and k + 1 lie side by side
// in both operands' rows, so nothing is packed), adds the two, and the segments' sums are added in ascending order, then the bias: a row's
// result does not depend on how many other rows the batch holds, where it stands, or which of the two kernels below computes it.
//
// * Up to 16 rows (decoded tokens): `gemm_f32_skinny_kernel`, bound by reading W once.  A warp streams 32 rows of W through a ring
//   of its own (cp.async, 6 stages of 32 rows x 32 k), a lane per row of W, so nothing but its own copies is waited for.  The
//   S segments of the same 32 rows are the warps of a cluster of CTAs of two warps, so that a matrix of 896 rows still
//   reaches 112 SMs with 40 KB in flight on each; they meet in distributed shared memory.
// * Beyond: `gemm_f32_tile_kernel`, bound by the FMA pipes and by issue slots: tiles of 128, 64 or 32 x 128 or 64, 8 x 8 (4 x 8, 4 x 4) results
//   a thread, a three-stage cp.async ring; the S segments of a tile are the CTAs of a cluster, which add up through distributed shared
//   memory, or where the tiles alone fill the GPU one CTA's, one after the other.  The packed form matters here: it halves the issue slots of the multiply-adds, which leaves room for the loads from shared memory.
//
// Measured (us; floor: W at 6.65 TB/s): 3 rows, 9,728 x 896 10.0 (floor 5.2; 82 with the one 64 x 64 tile form there was before), 896 x 4,864 10.4
// (2.6; 342), 151,936 x 896 93 (82; 503); 543 rows 260 (36 TFLOP/s; 314) and 149 (32; 299); 2,048 rows of 9,728 x 896 844 (42 TFLOP/s of 74; 1,015).
// The tiles are bound by the multiply-add pipes (59 % active) and the reads of shared memory beside them (75 %).
#include <cooperative_groups.h>
#include <stdio.h>

#include "common.cuh"

namespace sllm {

namespace cg = cooperative_groups;

// 16 (or 4) bytes from global to shared memory, `bytes` of them read and the rest zeros
__device__ __forceinline__ void f32_copy16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void f32_copy4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// two fused multiply-adds side by side, each rounded as fmaf's
__device__ __forceinline__ void f32_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float f32_both(unsigned long long acc) {
  return __uint_as_float((unsigned)acc) + __uint_as_float((unsigned)(acc >> 32));
}

// Four consecutive k from `src` (at k of its row) into shared memory; zeros from kend on.  Rows beyond an operand's are staged as its
// last row: nobody reads what they give.
template <bool VEC>
__device__ __forceinline__ void f32_stage4(float* dst, const float* src, int k, int kend) {
  if (VEC) {                               // K and kend are multiples of 4 here, so four k are in or out together
    f32_copy16(dst, src, k < kend ? 16 : 0);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) f32_copy4(dst + i, k + i < kend ? src + i : src, k + i < kend ? 4 : 0);
  }
}

// ---- up to 16 rows ------------------------------------------------------------------------------------------------------

constexpr int SK_WARPS = 2, SK_ROWS = 32, SK_BK = 32, SK_PITCH = SK_BK + 4, SK_STAGES = 6;

__host__ __device__ constexpr int sk_stage_floats(int MT) { return SK_ROWS * SK_PITCH + MT * SK_BK; }

template <int MT, bool VEC>
__global__ void __launch_bounds__(SK_WARPS * 32)
gemm_f32_skinny_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                       int M, int N, int K, int S, int seg) {
  extern __shared__ __align__(16) float sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* ring = sm + warp * (SK_STAGES * sk_stage_floats(MT));
  // S segments of the same rows are S neighbouring warps of the grid
  const int group = (blockIdx.x * SK_WARPS + warp) / S, s = (blockIdx.x * SK_WARPS + warp) % S;
  const int n0 = group * SK_ROWS, k0 = s * seg, kend = min(K, k0 + seg);
  const int steps = kend > k0 && n0 < N ? (kend - k0 + SK_BK - 1) / SK_BK : 0;

  // eight lanes a row: 128 consecutive bytes; the lane's rows are 4 apart
  const int kl = lane % 8 * 4;
  const float* wsrc[SK_ROWS / 4];
#pragma unroll
  for (int i = 0; i < SK_ROWS / 4; ++i) wsrc[i] = W + (size_t)min(n0 + i * 4 + lane / 8, N - 1) * K + kl;
  auto stage_w = [&](int it) {
    float* st = ring + (it % SK_STAGES) * sk_stage_floats(MT) + lane / 8 * SK_PITCH + kl;
    const int k = k0 + it * SK_BK;
#pragma unroll
    for (int i = 0; i < SK_ROWS / 4; ++i) f32_stage4<VEC>(st + i * 4 * SK_PITCH, wsrc[i] + (k + kl < K ? k : 0), k + kl, kend);
  };
  auto stage_a = [&](int it) {
    float* st = ring + (it % SK_STAGES) * sk_stage_floats(MT) + SK_ROWS * SK_PITCH;
    const int k = k0 + it * SK_BK;
#pragma unroll
    for (int r = lane / 8; r < MT; r += 4)
      f32_stage4<VEC>(st + r * SK_BK + kl, A + (size_t)min(r, M - 1) * K + (k + kl < K ? k + kl : 0), k + kl, kend);
  };

  unsigned long long two[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) two[m] = 0;
  // the weights are nobody's output: the first ring of them is on its way before the wait on the step's earlier kernels
#pragma unroll
  for (int p = 0; p < SK_STAGES - 1; ++p)
    if (p < steps) stage_w(p);
  pdl_wait();
#pragma unroll
  for (int p = 0; p < SK_STAGES - 1; ++p) {
    if (p < steps) stage_a(p);
    f32_commit();                                    // (the first group holds all the weights above)
  }
  for (int it = 0; it < steps; ++it) {
    f32_wait<SK_STAGES - 2>();
    __syncwarp();
    const float* wr = ring + (it % SK_STAGES) * sk_stage_floats(MT) + lane * SK_PITCH;
    const float* ar = ring + (it % SK_STAGES) * sk_stage_floats(MT) + SK_ROWS * SK_PITCH;
#pragma unroll
    for (int k = 0; k < SK_BK; k += 4) {
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(wr + k);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(ar + m * SK_BK + k);
        f32_fma2(two[m], a.x, w.x);
        f32_fma2(two[m], a.y, w.y);
      }
    }
    __syncwarp();
    if (it + SK_STAGES - 1 < steps) { stage_w(it + SK_STAGES - 1); stage_a(it + SK_STAGES - 1); }
    f32_commit();
  }
  f32_wait<0>();
  pdl_launch_dependents();
  float acc[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m] = f32_both(two[m]);
  if (S > 1) {
    __syncwarp();
#pragma unroll
    for (int m = 0; m < MT; ++m) ring[m * 32 + lane] = acc[m];       // the warp's own ring, drained
    if (S > SK_WARPS) cg::this_cluster().sync(); else __syncthreads();
    if (s == 0)
      for (int o = 1; o < S; ++o) {
        const float* there = sm + o % SK_WARPS * (SK_STAGES * sk_stage_floats(MT));
        const float* other = S > SK_WARPS ? cg::this_cluster().map_shared_rank(there, o / SK_WARPS) : there;
#pragma unroll
        for (int m = 0; m < MT; ++m) acc[m] += other[m * 32 + lane];
      }
    if (S > SK_WARPS) cg::this_cluster().sync();     // nobody leaves while its sums are being read
    if (s != 0) return;
  }
  const int n = n0 + lane;
  if (n >= N) return;
  const float b = bias ? bias[n] : 0.f;
#pragma unroll
  for (int m = 0; m < MT; ++m)
    if (m < M) C[(size_t)m * N + n] = acc[m] + b;
}

// ---- tiles --------------------------------------------------------------------------------------------------------------

constexpr int TL_BK = 32, TL_PITCH = TL_BK + 4, TL_STAGES = 3;

__host__ __device__ constexpr int tl_stage_floats(int BM, int BN) { return (BM + BN) * TL_PITCH; }
// the ring, and afterwards the tile's partial sums
__host__ __device__ constexpr int tl_smem(int BM, int BN) { return 4 * TL_STAGES * tl_stage_floats(BM, BN); }
static_assert(TL_STAGES * tl_stage_floats(32, 128) >= 32 * 128 && TL_STAGES * tl_stage_floats(128, 128) >= 128 * 128, "the ring holds a tile");
__host__ __device__ constexpr int tl_threads(int BM) { return BM == 32 ? 128 : 256; }

// FOLD: a CTA takes all the segments of its tile, one after the other; else the segments are the CTAs of a cluster (or there is one).
template <int BM, int BN, bool VEC, bool FOLD>
__global__ void __launch_bounds__(tl_threads(BM), BM == 128 ? 1 : 2)
gemm_f32_tile_kernel(const float* A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                     int M, int N, int K, int S, int seg) {
  constexpr int THREADS = tl_threads(BM), TM = BM == 128 ? 8 : 4, TN = BN / 16;
  constexpr int WM = TM * 4, WN = TN * 8;            // a warp's share: lanes 4 x 8, the rows of a lane 4 (of W: 8) apart
  constexpr int WARPS_N = BN / WN;
  static_assert(BM / WM * WARPS_N == THREADS / 32, "the warps' shares are the tile");
  extern __shared__ __align__(16) float sm[];
  // eight consecutive rows are what a quarter of a warp reads, and a pitch of 36 floats puts them on different banks
  const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
  const int mt = warp / WARPS_N * WM + lane / 8, nt = warp % WARPS_N * WN + lane % 8;
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
  pdl_wait();
  const int s = FOLD ? 0 : blockIdx.z, k0 = s * seg, kend = FOLD ? K : min(K, k0 + seg);
  const int steps = kend > k0 ? (kend - k0 + TL_BK - 1) / TL_BK : 0;
  const int fold = FOLD ? seg / TL_BK : 0;           // steps of a segment (a whole number: `launch`)
  unsigned long long two[TM][TN];
  float sum[FOLD ? TM : 1][FOLD ? TN : 1];           // the segments before
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) two[i][j] = 0;
  auto stage = [&](int it) {
    float* st = sm + (it % TL_STAGES) * tl_stage_floats(BM, BN);
    if constexpr (VEC) {                             // eight threads a row
      const int kl = tid % 8 * 4, row = tid / 8, k = k0 + it * TL_BK + kl, from = k < K ? k : 0;
      st += row * TL_PITCH + kl;
#pragma unroll
      for (int i = 0; i < BM; i += THREADS / 8) f32_stage4<true>(st + i * TL_PITCH, A + (size_t)min(m0 + row + i, M - 1) * K + from, k, kend);
#pragma unroll
      for (int i = 0; i < BN; i += THREADS / 8)
        f32_stage4<true>(st + (BM + i) * TL_PITCH, W + (size_t)min(n0 + row + i, N - 1) * K + from, k, kend);
    } else {                                         // a warp a row: neighbouring lanes copy neighbouring numbers
      const int k = k0 + it * TL_BK + lane, from = k < K ? k : 0, bytes = k < kend ? 4 : 0;
      st += warp * TL_PITCH + lane;
#pragma unroll 4
      for (int i = 0; i < BM; i += THREADS / 32) f32_copy4(st + i * TL_PITCH, A + (size_t)min(m0 + warp + i, M - 1) * K + from, bytes);
#pragma unroll 4
      for (int i = 0; i < BN; i += THREADS / 32) f32_copy4(st + (BM + i) * TL_PITCH, W + (size_t)min(n0 + warp + i, N - 1) * K + from, bytes);
    }
  };
#pragma unroll
  for (int p = 0; p < TL_STAGES - 1; ++p) {
    if (p < steps) stage(p);
    f32_commit();
  }
  for (int it = 0; it < steps; ++it) {
    f32_wait<TL_STAGES - 2>();
    __syncthreads();
    if (it + TL_STAGES - 1 < steps) stage(it + TL_STAGES - 1);
    f32_commit();
    const float* as = sm + (it % TL_STAGES) * tl_stage_floats(BM, BN) + mt * TL_PITCH;
    const float* ws = sm + (it % TL_STAGES) * tl_stage_floats(BM, BN) + (BM + nt) * TL_PITCH;
    if (FOLD && it % fold == 0 && it > 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          sum[i][j] = it == fold ? f32_both(two[i][j]) : sum[i][j] + f32_both(two[i][j]);
          two[i][j] = 0;
        }
    }
    const int left = kend - k0 - it * TL_BK;         // (what lies beyond is zeros)
#pragma unroll
    for (int k = 0; k < TL_BK; k += 4) {
      if (!VEC && k >= left) break;
      ulonglong2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + i * 4 * TL_PITCH + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(ws + j * 8 * TL_PITCH + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) f32_fma2(two[i][j], a[i].x, w.x);
#pragma unroll
        for (int i = 0; i < TM; ++i) f32_fma2(two[i][j], a[i].y, w.y);
      }
    }
  }
  f32_wait<0>();
  if (FOLD || S == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + mt + i * 4;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + nt + j * 8;
        if (n >= N) continue;
        float v = f32_both(two[i][j]);
        if constexpr (FOLD) v = sum[i][j] + v;
        C[(size_t)m * N + n] = v + (bias ? bias[n] : 0.f);
      }
    }
    return;
  }
  if constexpr (!FOLD) {
    __syncthreads();                                 // everybody has read the last stage
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) sm[(mt + i * 4) * BN + nt + j * 8] = f32_both(two[i][j]);
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    // each CTA of the cluster adds up its share of the tile's rows, the segments in order
    const int share = BM / S;
    for (int i = tid; i < share * BN; i += THREADS) {
      const int r = s * share + i / BN, c = i % BN;
      if (m0 + r >= M || n0 + c >= N) continue;
      float v = *cl.map_shared_rank(sm + r * BN + c, 0);
      for (int o = 1; o < S; ++o) v += *cl.map_shared_rank(sm + r * BN + c, o);
      C[(size_t)(m0 + r) * N + n0 + c] = v + (bias ? bias[n0 + c] : 0.f);
    }
    cl.sync();                                       // nobody leaves while its sums are being read
  }
}

// Segments of K: as many (1, 2, 4, 8) as give the skinny kernel four warps of 32 rows an SM, none shorter than 64.  A warp is bound by the
// latency of its own steps (about 0.4 us for 4 KB of weights), so warps are what it needs; the tiles gain the finer waves and pay the pass
// over the cluster's sums.  (16 segments: 896 x 4,864 and 3 rows 9.8 -> 7.5 us, 537 rows 209 -> 237; 1,152 x 896 and 3 rows 4.2 -> 7.0.)
static int segments(int N, int K) {
  int S = 1;
  while (S < 8 && (long long)((N + SK_ROWS - 1) / SK_ROWS) * S < 4 * 148 && K / (2 * S) >= 64) S *= 2;
  return S;
}

template <typename Kernel>
static int launch_clusters(Kernel kernel, dim3 grid, int threads, int smem, dim3 cluster, const float* A, const float* W, const float* bias,
                           float* C, int M, int N, int K, int S, int seg, cudaStream_t stream) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  SLLM_REQUIRE(e == cudaSuccess, "gemm_f32: %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster.x;
  attr[0].val.clusterDim.y = cluster.y;
  attr[0].val.clusterDim.z = cluster.z;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, A, W, bias, C, M, N, K, S, seg);
  return launch_status("gemm_f32");
}

template <int MT, bool VEC>
static int launch_skinny(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int S, int seg, cudaStream_t stream) {
  const int warps = (N + SK_ROWS - 1) / SK_ROWS * S;
  const int cluster = S > SK_WARPS ? S / SK_WARPS : 1;       // (S > 1: the warps are then a whole number of clusters)
  return launch_clusters(gemm_f32_skinny_kernel<MT, VEC>, dim3((warps + SK_WARPS - 1) / SK_WARPS), SK_WARPS * 32,
                         4 * SK_WARPS * SK_STAGES * sk_stage_floats(MT), dim3(cluster, 1, 1), A, W, bias, C, M, N, K, S, seg, stream);
}

template <int BM, int BN, bool VEC, bool FOLD>
static int launch_tiles(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int S, int seg, cudaStream_t stream) {
  const int rows = (M + BM - 1) / BM, cols = (N + BN - 1) / BN;
  SLLM_REQUIRE(rows <= 65535, "gemm_f32: M=%d is too large for one launch", M);
  const int parts = FOLD ? 1 : S;
  return launch_clusters(gemm_f32_tile_kernel<BM, BN, VEC, FOLD>, dim3(cols, rows, parts), tl_threads(BM), tl_smem(BM, BN), dim3(1, 1, parts), A, W, bias, C,
                         M, N, K, S, seg, stream);
}

// The forms of the tiles and what they take, us: a step of 32 k of a CTA no less than `wait` (latency) nor than `work` times the CTAs that share its SM; `once` a
// tile; `cluster` the pass over the cluster's sums, times the CTAs an SM; `launch`.  Fitted to 26 matrices of 24 x 1,024 to 32,000 x 512 with 17 to 4,096 rows; without
// whole 16-byte pieces (`vec` false) copies of 4 bytes weigh on every step.
struct TileForm {
  int bm, bn, per_sm, fold;
  float wait[2], work[2], once[2], cluster[2], launch[2], margin;      // [whole pieces]; margin: how much better it must look, the model's error
};
constexpr TileForm TILE_FORMS[] = {
    {32, 64, 4, 0, {0.82f, 0.66f}, {0.46f, 0.47f}, {0.f, 0.f}, {1.68f, 0.88f}, {1.96f, 2.19f}, 1.2f},
    {32, 128, 3, 0, {1.66f, 1.18f}, {0.91f, 0.86f}, {0.f, 0.f}, {3.92f, 2.11f}, {1.48f, 2.37f}, 1.0f},
    {64, 128, 2, 0, {2.38f, 1.95f}, {1.52f, 1.74f}, {0.f, 0.f}, {5.42f, 3.2f}, {0.97f, 2.38f}, 1.0f},
    {64, 64, 2, 1, {1.64f, 1.15f}, {1.32f, 1.03f}, {0.f, 0.f}, {0.f, 0.f}, {0.41f, 1.72f}, 1.2f},
    {64, 128, 2, 1, {2.69f, 2.28f}, {2.12f, 1.85f}, {0.f, 0.f}, {0.f, 0.f}, {0.02f, 3.16f}, 1.1f},
    {128, 128, 1, 1, {3.99f, 3.34f}, {0.04f, 2.43f}, {0.f, 3.7f}, {0.f, 0.f}, {0.f, 0.06f}, 1.1f},
};
// The form that finishes first: waves of CTAs an SM, and never faster than W streams in once per row of tiles (2 TB/s).  (us, one form for all rows before: 64 x
// 64 matrix, 2,048 rows 8.4 -> 3.4; 2,304 x 768, 2,048 rows 243 -> 169 with the segments in turn; 896 x 896, 130 rows 19.3 -> 13.1.)
static int tile_form(int M, int N, int K, int S, int seg, bool vec) {
  const int sms = num_sms();
  int best = 2;
  float least = 0.f;
  for (int f = 0; f < (int)(sizeof(TILE_FORMS) / sizeof(TileForm)); ++f) {
    const TileForm& t = TILE_FORMS[f];
    if (t.fold && S == 1) continue;                  // (that is the form without)
    if (t.bm < 64 && M > 65535 * t.bm) continue;     // (a launch's rows of tiles)
    const long long rows = (M + t.bm - 1) / t.bm, ctas = rows * ((N + t.bn - 1) / t.bn) * (t.fold ? 1 : S), per = (ctas + sms - 1) / sms;
    const float steps = (float)((t.fold || seg > K ? K + TL_BK - 1 : seg) / TL_BK);
    const auto wave = [&](long long n) { return n == 0 ? 0.f : t.once[vec] + steps * fmaxf(t.wait[vec], (float)n * t.work[vec]); };
    float us = t.launch[vec] + (float)(per / t.per_sm) * wave(t.per_sm) + wave(per % t.per_sm) + (S > 1 ? t.cluster[vec] * (float)per : 0.f);
    us = t.margin * fmaxf(us, (float)rows * (float)N * (float)K * 2e-6f);
    if (least == 0.f || us < least) {
      best = f;
      least = us;
    }
  }
  return best;
}

template <bool VEC>
static int launch(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
  const int S = segments(N, K), seg = ((K + S - 1) / S + 31) / 32 * 32;
  if (M <= 1) return launch_skinny<1, VEC>(A, W, bias, C, M, N, K, S, seg, stream);
  if (M <= 2) return launch_skinny<2, VEC>(A, W, bias, C, M, N, K, S, seg, stream);
  if (M <= 4) return launch_skinny<4, VEC>(A, W, bias, C, M, N, K, S, seg, stream);
  if (M <= 8) return launch_skinny<8, VEC>(A, W, bias, C, M, N, K, S, seg, stream);
  if (M <= 16) return launch_skinny<16, VEC>(A, W, bias, C, M, N, K, S, seg, stream);
  switch (tile_form(M, N, K, S, seg, VEC)) {
    case 0: return launch_tiles<32, 64, VEC, false>(A, W, bias, C, M, N, K, S, seg, stream);
    case 1: return launch_tiles<32, 128, VEC, false>(A, W, bias, C, M, N, K, S, seg, stream);
    case 2: return launch_tiles<64, 128, VEC, false>(A, W, bias, C, M, N, K, S, seg, stream);
    case 3: return launch_tiles<64, 64, VEC, true>(A, W, bias, C, M, N, K, S, seg, stream);
    case 4: return launch_tiles<64, 128, VEC, true>(A, W, bias, C, M, N, K, S, seg, stream);
  }
  return launch_tiles<128, 128, VEC, true>(A, W, bias, C, M, N, K, S, seg, stream);
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                              cudaStream_t stream) {
  SLLM_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
  if (M == 0) return SLLM_OK;
  const bool vec = K % 4 == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
  return vec ? launch<true>(A, W, bias, C, M, N, K, stream) : launch<false>(A, W, bias, C, M, N, K, stream);
}
