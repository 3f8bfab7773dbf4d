// Weight-streaming linear layer for few tokens (decoding): y[M, N] = x[M, K] W[N, K]^T with
// M <= 64, bfloat16 operands, float32 accumulation.  At these sizes the product is bound by
// reading W once from HBM, so the kernel is built around that stream:
//
//  * W is the M-side operand of mma.sync m16n8k16 (16 weight rows per warp), the tokens are
//    the N side (8 tokens per MMA), so no tensor-core work is wasted on padding tokens to 16+.
//  * Each thread reads its share of W straight from global memory into the MMA's A-fragment
//    registers with 16-byte loads, two chunks ahead of the math.  Within a 32-wide k block a
//    thread takes 8 consecutive k of two rows; the k order inside the block is permuted
//    identically for W and x (a dot product does not care), so no shuffle or shared-memory
//    staging of W is needed.
//  * The tokens' activations are staged per 128-wide k chunk in shared memory (double
//    buffered with cp.async) and shared by the CTA's 8 warps (128 weight rows).
//  * Small N (the attention and down projections) would leave most SMs idle, so the grid
//    also splits K; the partial sums go to scratch [splits, M, N] and the consumer (the
//    residual add + RMSNorm kernel, or the rotary kernel) adds them in a fixed order.
//  * Epilogues: bias; SiLU(gate)*up for a gate|up matrix whose rows alternate in blocks of 8
//    (rows g and g+8 of a warp's tile are a gate row and its up row, held by one thread).
//
// The reference's device path calls cublasGemmEx for these products
// (kernels/cuda/kernels.cu:752-767; kernels/device_decode.py:294-326) and applies SiLU*up
// in a kernel of its own (kernels.cu:898-919).
#include <stdio.h>

#include "common.cuh"

namespace sllm {

constexpr int LS_KC = 128;                 // k per chunk
constexpr int LS_ROWS = 128;               // weight rows per CTA (8 warps x 16)
constexpr int LS_XSTRIDE = LS_KC + 32;     // bf16 elements: 320 bytes, = 64 mod 128 -> conflict-free 16-byte reads

#define EPI_STORE 0
#define EPI_SILU 1
#define EPI_GELU 2      // the tanh form of GELU in place of SiLU, gate and up each with its bias

constexpr int LS_SSQ_MAX = 608;            // partial sums of squares per token a scaled launch takes (as in linear_ws.cu)

// A norm still owed on the input (see linear_ws.cu, WsNorm): x is bfloat16(stream * gain), ssq [M][stride]
// (stride = parts rounded up to 4) holds partial sums of squares of the stream's rows, and every row of the
// product is multiplied by rsqrt(sum / width + eps) before the epilogue's arithmetic.
struct LsScale {
  const float* ssq = nullptr;
  int parts = 0;
  float eps = 0.f, inv_width = 0.f;
};

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void ls_cp_async_16(void* smem, const void* gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void ls_mma(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                       unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// acc[j][c]: c0,c1 = (row g, tokens 8j+2t, +1); c2,c3 = (row g+8, same tokens) of the 16 rows from n0
template <int NT, int EPI, typename OUT>
__device__ __forceinline__ void ls_finish(const float (&acc)[NT][4], int n0, int g, int t4, const float* __restrict__ bias, OUT* __restrict__ out, int M, int N) {
  const int row_a = n0 + g, row_b = n0 + g + 8;
  if constexpr (EPI == EPI_SILU || EPI == EPI_GELU) {
    // rows g (gate i) and g+8 (up i) of this 16-row tile; the output column is (n0/16)*8 + g
    const int col = (n0 >> 4) * 8 + g;
    const int I = N >> 1;
    if (row_b < N) {
      const float bias_g = (EPI == EPI_GELU && bias) ? bias[row_a] : 0.f, bias_u = (EPI == EPI_GELU && bias) ? bias[row_b] : 0.f;
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int tok = 8 * j + 2 * t4 + c;
          if (tok < M) {
            const float gate = acc[j][c] + bias_g, up = acc[j][c + 2] + bias_u;
            if constexpr (EPI == EPI_GELU)
              out[(size_t)tok * I + col] = from_f32<OUT>(0.5f * gate * (1.0f + tanhf(0.7978845608028654f * (gate + 0.044715f * gate * gate * gate))) * up);
            else
              out[(size_t)tok * I + col] = from_f32<OUT>(gate * (1.0f / (1.0f + expf(-gate))) * up);
          }
        }
    }
  } else {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int tok = 8 * j + 2 * t4 + (c & 1), row = (c & 2) ? row_b : row_a;
        if (tok < M && row < N) out[(size_t)tok * N + row] = from_f32<OUT>(acc[j][c] + (bias ? bias[row] : 0.f));
      }
  }
}

// NT: 8-token tiles (M <= 8*NT).  OUT: float or __nv_bfloat16.  SCALED: the rows of the result are scaled
// (LsScale; unsplit launches only).
template <int NT, int EPI, typename OUT, bool SCALED>
__global__ void __launch_bounds__(256)
linear_stream_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ W,
                     const float* __restrict__ bias, OUT* __restrict__ out, float* __restrict__ partial,
                     int M, int N, int K, int chunks_per_split, const LsScale scale) {
  extern __shared__ __align__(16) unsigned char ls_smem[];
  __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(ls_smem);          // [2][8*NT][LS_XSTRIDE]
  float* ssq_s = reinterpret_cast<float*>(ls_smem + sizeof(__nv_bfloat16) * 2 * 8 * NT * LS_XSTRIDE);   // SCALED: [8*NT][LS_SSQ_MAX]
  __shared__ float row_scale[8 * NT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int n0 = blockIdx.x * LS_ROWS + warp * 16;
  const int split = blockIdx.y;
  const int total_chunks = K / LS_KC;
  const int c_begin = split * chunks_per_split;
  const int c_end = min(total_chunks, c_begin + chunks_per_split);
  const int n_chunks = max(c_end - c_begin, 0);

  // rows past N are clamped for the loads and skipped at the store
  const int r0 = min(n0 + g, N - 1), r1 = min(n0 + g + 8, N - 1);
  const __nv_bfloat16* w0 = W + (size_t)r0 * K + (size_t)c_begin * LS_KC + t4 * 8;
  const __nv_bfloat16* w1 = W + (size_t)r1 * K + (size_t)c_begin * LS_KC + t4 * 8;

  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;

  auto load_x = [&](int chunk, int buf) {
    // [8*NT tokens][128 k] -> 16 sixteen-byte pieces per token
    for (int c = tid; c < 8 * NT * (LS_KC / 8); c += 256) {
      const int tok = c / (LS_KC / 8), piece = c % (LS_KC / 8);
      const bool ok = tok < M;
      const __nv_bfloat16* src = x + (size_t)(ok ? tok : 0) * K + (size_t)(c_begin + chunk) * LS_KC + piece * 8;
      ls_cp_async_16(xs + ((size_t)buf * 8 * NT + tok) * LS_XSTRIDE + piece * 8, src, ok);
    }
  };
  auto load_w = [&](uint4 (&a)[8], int chunk) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      a[2 * b] = ldg_stream(w0 + (size_t)chunk * LS_KC + b * 32);
      a[2 * b + 1] = ldg_stream(w1 + (size_t)chunk * LS_KC + b * 32);
    }
  };
  auto compute = [&](const uint4 (&a)[8], int buf) {
    const __nv_bfloat16* xb = xs + (size_t)buf * 8 * NT * LS_XSTRIDE;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const uint4 ra = a[2 * b], rb = a[2 * b + 1];         // rows g and g+8: 8 consecutive k each
      uint4 xv[NT];
#pragma unroll
      for (int j = 0; j < NT; ++j) xv[j] = *reinterpret_cast<const uint4*>(xb + (size_t)(8 * j + g) * LS_XSTRIDE + b * 32 + t4 * 8);
      // first MMA: k slots (2t,2t+1) <- elements 0,1; slots (2t+8,2t+9) <- elements 2,3; second: elements 4,5 and 6,7.  A tile's second depends on its first, so the tiles'
      // first ones come before their second ones.
#pragma unroll
      for (int j = 0; j < NT; ++j) ls_mma(acc[j], ra.x, rb.x, ra.y, rb.y, xv[j].x, xv[j].y);
#pragma unroll
      for (int j = 0; j < NT; ++j) ls_mma(acc[j], ra.z, rb.z, ra.w, rb.w, xv[j].z, xv[j].w);
    }
  };

  uint4 wa[8], wb[8];
  // weights do not depend on the step's earlier kernels: start the stream (two chunks) now
  if (n_chunks > 0) load_w(wa, 0);
  if (n_chunks > 1) load_w(wb, 1);
  pdl_wait();                          // the activations do
  if (n_chunks > 0) load_x(0, 0);
  if constexpr (SCALED) {
    // the tokens' partial sums of squares come to shared memory with the first activations
    const int stride = (scale.parts + 3) & ~3, pieces = stride >> 2;
    for (int c = tid; c < M * pieces; c += 256) {
      const int tok = c / pieces, piece = c % pieces;
      ls_cp_async_16(ssq_s + (size_t)tok * LS_SSQ_MAX + piece * 4, scale.ssq + (size_t)tok * stride + piece * 4, true);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::);
  for (int c = 0; c < n_chunks; c += 2) {
    // chunk c from wa, chunk c+1 from wb
    if (c + 1 < n_chunks) {
      load_x(c + 1, 1);
      if (c > 0) load_w(wb, c + 1);    // the first pair was fetched before the wait
    }
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
    compute(wa, 0);
    __syncthreads();
    if (c + 1 >= n_chunks) break;
    if (c + 2 < n_chunks) {
      load_x(c + 2, 0);
      load_w(wa, c + 2);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_group 1;\n" ::);
    __syncthreads();
    compute(wb, 1);
    __syncthreads();
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  pdl_launch_dependents();             // the stream is read; the next kernel may begin while the results are stored
  if constexpr (SCALED) {
    // warp w adds the partial sums of tokens w, w + 8, ...: lane l takes l, l + 32, ..., then the lanes are added
    // (the table has been visible to all since the loop's first barrier)
    for (int tok = warp; tok < 8 * NT; tok += 8) {
      float sum = 0.f;
      if (tok < M)
        for (int p = lane; p < scale.parts; p += 32) sum += ssq_s[(size_t)tok * LS_SSQ_MAX + p];
      sum = warp_sum(sum);
      if (lane == 0) row_scale[tok] = rsqrtf(sum * scale.inv_width + scale.eps);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j][c] *= row_scale[8 * j + 2 * t4 + (c & 1)];
  }

  // ---- epilogue ----
  if (gridDim.y > 1) {
    const int row_a = n0 + g, row_b = n0 + g + 8;
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int tok = 8 * j + 2 * t4 + (c & 1), row = (c & 2) ? row_b : row_a;
        if (tok < M && row < N)
          partial[((size_t)split * M + tok) * N + row] = acc[j][c] + ((bias && split == 0) ? bias[row] : 0.f);
      }
    return;
  }
  ls_finish<NT, EPI, OUT>(acc, n0, g, t4, bias, out, M, N);
}

// The same product with all of the activations in shared memory (a short K): no barrier in the stream, so it is bound by the weights in flight alone.  Above, a chunk of 128
// columns waits for its activations from L2 between two barriers, which for 32 tokens and K = 896 was seven round trips of a kernel whose weights take 2.7 us.
// A CTA of four warps takes 64 rows, so that 9,728 rows are 152 CTAs for 148 SMs and a warp's products a quarter of a scheduler's; a warp keeps LR_DEPTH chunks (16 KB) in flight, the
// first of them before the wait; the activations lie in the order the lanes read them, 16 bytes each.  The k order of every sum is that of the form above, so are the bits.
// (In a graph of such products, us, this / the form above: one token, output head 151,936 x 896 42.5 / 48.0; 8 tokens, gate|up with the activation 4,864 x 896 4.5 / 7.6, 8,192 x 1,024 6.1 / 9.0,
// with a norm owed 6.7 / 9.0; 16 tokens 5.2 / 7.9, 7.1 / 9.3, 7.7 / 9.6; 12,288 x 1,536 11.2 / 14.1; 32 tokens with a norm owed 9,728 x 896 12.0 / 13.6, 4,864 x 896 8.5 / 12.2.)
constexpr int LR_WARPS = 4, LR_DEPTH = 4, LR_X_MAX = 100 * 1024;

template <int NT, int EPI, typename OUT, bool SCALED>
__global__ void __launch_bounds__(LR_WARPS * 32)
linear_resident_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias, OUT* __restrict__ out,
                       int M, int N, int K, const LsScale scale) {
  extern __shared__ __align__(16) unsigned char ls_smem[];               // [K / 32][NT][32 lanes] 16 bytes
  __shared__ float row_scale[8 * NT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int n0 = (blockIdx.x * LR_WARPS + warp) * 16;
  const int chunks = K / LS_KC;
  const int r0 = min(n0 + g, N - 1), r1 = min(n0 + g + 8, N - 1);      // rows past N are clamped for the loads and skipped at the store
  const __nv_bfloat16* w0 = W + (size_t)r0 * K + t4 * 8;
  const __nv_bfloat16* w1 = W + (size_t)r1 * K + t4 * 8;
  uint4 w[LR_DEPTH][8];
  auto load_w = [&](uint4 (&a)[8], int chunk) {
    if (chunk >= chunks) return;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      a[2 * b] = ldg_stream(w0 + (size_t)chunk * LS_KC + b * 32);
      a[2 * b + 1] = ldg_stream(w1 + (size_t)chunk * LS_KC + b * 32);
    }
  };
#pragma unroll
  for (int d = 0; d < LR_DEPTH; ++d) load_w(w[d], d);
  pdl_wait();
  for (int e = tid; e < K / 32 * NT * 32; e += LR_WARPS * 32) {
    const int l = e & 31, j = (e >> 5) % NT, b = (e >> 5) / NT, row = 8 * j + (l >> 2);
    if (row < M) ls_cp_async_16(ls_smem + (size_t)e * 16, x + (size_t)row * K + b * 32 + (l & 3) * 8, true);       // (tokens past M: what lies there, in columns that nobody stores)
  }
  asm volatile("cp.async.commit_group;\n" ::);
  if constexpr (SCALED) {              // eight lanes a token, four partial sums a load: every load of a thread is under way before the first is added
    constexpr int LANES = LR_WARPS * 32 / (8 * NT) < 8 ? LR_WARPS * 32 / (8 * NT) : 8;
    const int stride = (scale.parts + 3) & ~3, tok = tid / LANES, q = tid % LANES;
    float sum = 0.f;
    if (tok < M) {
      const float* s = scale.ssq + (size_t)tok * stride;
#pragma unroll 4
      for (int p = q * 4; p < scale.parts; p += LANES * 4) {
        const float4 v = *reinterpret_cast<const float4*>(s + p);
        sum += v.x + (p + 1 < scale.parts ? v.y : 0.f) + (p + 2 < scale.parts ? v.z : 0.f) + (p + 3 < scale.parts ? v.w : 0.f);
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (q == 0 && tok < 8 * NT) row_scale[tok] = rsqrtf(sum * scale.inv_width + scale.eps);
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
  for (int c0 = 0; c0 < chunks; c0 += LR_DEPTH) {
#pragma unroll
    for (int d = 0; d < LR_DEPTH; ++d) {
      const int c = c0 + d;
      if (c >= chunks) break;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const uint4 ra = w[d][2 * b], rb = w[d][2 * b + 1];
        uint4 xv[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) xv[j] = *reinterpret_cast<const uint4*>(ls_smem + ((size_t)((c * 4 + b) * NT + j) * 32 + lane) * 16);
        // (a token tile's two products depend on one another: the tiles' first ones, then their second ones)
#pragma unroll
        for (int j = 0; j < NT; ++j) ls_mma(acc[j], ra.x, rb.x, ra.y, rb.y, xv[j].x, xv[j].y);
#pragma unroll
        for (int j = 0; j < NT; ++j) ls_mma(acc[j], ra.z, rb.z, ra.w, rb.w, xv[j].z, xv[j].w);
      }
      load_w(w[d], c + LR_DEPTH);
    }
  }
  pdl_launch_dependents();
  if constexpr (SCALED) {
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j][c] *= row_scale[8 * j + 2 * t4 + (c & 1)];
  }
  ls_finish<NT, EPI, OUT>(acc, n0, g, t4, bias, out, M, N);
}

// Where the activations fit and this form is the faster one (the bits are the same).  With four token tiles the products of a warp (mma.sync, some 30 cycles each) are what takes the
// time, so there only where the form above is worse off still: a norm owed, whose partial sums it adds token after token behind the stream, or too few rows for its CTAs.  Else by
// how well the CTAs fill the SMs, three an SM (registers) or what the activations leave room for, against the form above with two of 128 rows: as long as all are on the SMs at
// once the shorter CTAs win, in later waves only where they fill them better.  A CTA has 64 KB of loads in flight, which lie in L1: where the activations of an SM's CTAs leave less than
// 92 KB of it, two CTAs an SM at most; less than 60 KB, one on every other SM.  (Us, the form above / this one.  8 tokens: 1,024 x 2,048 16.4 / 7.1, 9,728 x 1,536 13.3 / 9.1, 18,944
// x 1,536 1.25 times as fast, 28,416 rows 1.08, 30,720 (1.1 waves) 0.94, 32,000 18.7 / 20.0, 36,864 0.88, 40,960 (1.4 waves against 1.1 of the other) 1.26, 65,536 1.0, 151,936 x 1,536
// 81.9 / 73.9; K = 256 1,024 rows 1.98 / 1.76, 9,728 2.62 / 2.63, 32,000 4.4 / 5.2.  K = 4,096 9,728 rows 34.4 / 26.9, 24,576 0.98, 32,000 48.3 / 65.1; K = 6,400 4,096 rows 51.2 /
// 39.2, 8,192 52.6 / 55.5, 9,472 53.1 / 64.9; K = 4,864 9,472 rows 40.7 / 23.4, K = 4,608 38.9 / 50.9.
// 16 tokens: 9,728 x 2,048 18.1 / 15.2, 32,000 x 2,048 25.7 / 35.6, 9,728 x 3,200 27.7 / 41.2.  17 tokens: 9,728 x 896 with the activation 9.6 / 10.4, with a norm owed 13.4 / 11.0;
// 4,096 x 1,024 10.3 / 7.2, 6,144 x 1,536 15.3 / 10.3, 8,192 x 1,024 10.6 / 9.8, 32 tokens 10.6 / 11.0.)
constexpr int LR_MANY_TOKENS_ROWS = 7168, LR_CTAS = 3;
static bool ls_resident(int M, int N, int K, int splits, bool gated, bool scaled) {
  const int nt = M <= 8 ? 1 : (M <= 16 ? 2 : 4), bytes = K * 16 * nt;
  if (splits != 1 || M > 32 || bytes > LR_X_MAX || (nt == 4 && !scaled && N > LR_MANY_TOKENS_ROWS)) return false;
  if ((K <= 256 && scaled) || (K < 512 && nt == 4 && gated && !scaled)) return false;       // (two or three chunks: what comes before the stream is all of it)
  const int sms = num_sms(), ctas = (N + LR_WARPS * 16 - 1) / (LR_WARPS * 16);
  const int a_cta = bytes + 1152, fit = 227 * 1024 / a_cta, per_sm = fit < LR_CTAS ? fit : LR_CTAS;
  if (per_sm * a_cta > 196 * 1024) return ctas <= sms / 2;
  if (ctas <= sms) return true;
  if (K <= 256 || (K < 512 && nt == 1 && scaled)) return false;
  if (K < 512 || (nt < 4 && per_sm * a_cta > 164 * 1024) || (nt == 1 && scaled && K < 1536) || (nt == 2 && K < 896)) return ctas <= 2 * sms;
  const long long places = (long long)per_sm * sms, above = (N + LS_ROWS - 1) / LS_ROWS, above_places = 2LL * sms;
  const long long waves = (ctas + places - 1) / places, above_waves = (above + above_places - 1) / above_places;
  return ctas * above_waves * above_places > above * waves * places;
}
// 1: the form with resident activations, 0: the other (epilogue as in sllm_linear_stream; scaled: sllm_linear_stream_silu_scaled)
SLLM_EXPORT int sllm_linear_stream_resident(int M, int N, int K, int epilogue, int scaled) { return ls_resident(M, N, K, 1, epilogue != 0, scaled != 0) ? 1 : 0; }

template <int NT, int EPI, typename OUT, bool SCALED>
static int launch_resident(const __nv_bfloat16* x, const __nv_bfloat16* W, const float* bias, void* out, int M, int N, int K, cudaStream_t stream, const LsScale& scale) {
  static SharedLimit limit;
  if (!limit.raise(linear_resident_kernel<NT, EPI, OUT, SCALED>, LR_X_MAX)) {
    set_error("linear_stream: cannot raise the shared memory limit");
    return SLLM_ERR_LAUNCH;
  }
  launch_kernel(linear_resident_kernel<NT, EPI, OUT, SCALED>, (N + LR_WARPS * 16 - 1) / (LR_WARPS * 16), LR_WARPS * 32, (size_t)K * 16 * NT, stream, x, W, bias, (OUT*)out, M, N, K, scale);
  return launch_status("linear_stream");
}

template <int NT, int EPI, typename OUT, bool SCALED = false>
static int launch_ls(const __nv_bfloat16* x, const __nv_bfloat16* W, const float* bias, void* out, float* partial,
                     int M, int N, int K, int splits, cudaStream_t stream, const LsScale& scale = LsScale{}) {
  if constexpr (NT <= 4) {
    if (ls_resident(M, N, K, splits, EPI != EPI_STORE, SCALED)) return launch_resident<NT, EPI, OUT, SCALED>(x, W, bias, out, M, N, K, stream, scale);
  }
  constexpr size_t smem = sizeof(__nv_bfloat16) * 2 * 8 * NT * LS_XSTRIDE + (SCALED ? sizeof(float) * 8 * NT * LS_SSQ_MAX : 0);
  static SharedLimit limit;
  if (smem + 1024 > 48 * 1024 && !limit.raise(linear_stream_kernel<NT, EPI, OUT, SCALED>, smem)) {      // (the kernel has a little static shared memory too)
    set_error("linear_stream: cannot raise the shared memory limit");
    return SLLM_ERR_LAUNCH;
  }
  const int total_chunks = K / LS_KC;
  const int per = (total_chunks + splits - 1) / splits;
  dim3 grid((N + LS_ROWS - 1) / LS_ROWS, (total_chunks + per - 1) / per);
  launch_kernel(linear_stream_kernel<NT, EPI, OUT, SCALED>, grid, 256, smem, stream, x, W, bias, (OUT*)out, partial, M, N, K, per, scale);
  return launch_status("linear_stream");
}

}  // namespace sllm

using namespace sllm;

// How many k-splits a launch with `splits_wanted` really uses (the scratch needs that many slices).
SLLM_EXPORT int sllm_linear_stream_splits(int K, int splits_wanted) {
  const int total_chunks = K / LS_KC;
  if (total_chunks <= 0) return 1;
  const int s = splits_wanted < 1 ? 1 : (splits_wanted > total_chunks ? total_chunks : splits_wanted);
  const int per = (total_chunks + s - 1) / s;
  return (total_chunks + per - 1) / per;
}

SLLM_EXPORT int sllm_linear_stream_supports(int M, int N, int K) {
  return M >= 1 && M <= 64 && N >= 16 && K >= LS_KC && K % LS_KC == 0;
}

// epilogue 0: out[M, N] (+bias) in out_dtype, or with splits > 1 float32 partial[splits, M, N];
// epilogue 1: out[M, N/2] = silu(gate) * up for rows interleaved in blocks of 8 (splits must be 1);
// epilogue 2: the same with gelu_tanh(gate + bias) * (up + bias), the bias interleaved like the rows.
SLLM_EXPORT int sllm_linear_stream(const void* x, const void* W, const float* bias, void* out, int out_dtype,
                                   float* partial, int M, int N, int K, int splits, int epilogue,
                                   cudaStream_t stream) {
  SLLM_REQUIRE(sllm_linear_stream_supports(M, N, K), "linear_stream: sizes M=%d N=%d K=%d (needs M<=64, K%%128==0)", M, N, K);
  SLLM_REQUIRE(splits >= 1, "linear_stream: splits=%d", splits);
  SLLM_REQUIRE(splits == 1 || partial != nullptr, "linear_stream: k-splits need scratch");
  SLLM_REQUIRE(epilogue == EPI_STORE || (splits == 1 && N % 16 == 0 && out_dtype == SLLM_BF16),
               "linear_stream: the gated epilogues need splits=1, N%%16==0 and a bfloat16 result");
  SLLM_REQUIRE(epilogue >= EPI_STORE && epilogue <= EPI_GELU, "linear_stream: unknown epilogue %d", epilogue);
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)W;
  const int nt = M <= 8 ? 1 : (M <= 16 ? 2 : (M <= 32 ? 4 : 8));
#define GO(NT_)                                                                                              \
  if (epilogue == EPI_SILU) return launch_ls<NT_, EPI_SILU, __nv_bfloat16>(xb, wb, bias, out, partial, M, N, K, splits, stream); \
  if (epilogue == EPI_GELU) return launch_ls<NT_, EPI_GELU, __nv_bfloat16>(xb, wb, bias, out, partial, M, N, K, splits, stream); \
  if (out_dtype == SLLM_BF16) return launch_ls<NT_, EPI_STORE, __nv_bfloat16>(xb, wb, bias, out, partial, M, N, K, splits, stream); \
  return launch_ls<NT_, EPI_STORE, float>(xb, wb, bias, out, partial, M, N, K, splits, stream);
  switch (nt) {
    case 1: GO(1)
    case 2: GO(2)
    case 4: GO(4)
    default: GO(8)
  }
#undef GO
}

// The SiLU epilogue on an input whose norm is still owed: out[M, N/2] = silu(s gate) * (s up) with
// s[token] = rsqrt(sum of ssq[token][0..parts) / width + eps); x is bfloat16(stream * gain).  At most 32 tokens.
SLLM_EXPORT int sllm_linear_stream_silu_scaled(const void* x, const void* W, void* out, int M, int N, int K, const float* ssq,
                                               int parts, float eps, int width, cudaStream_t stream) {
  SLLM_REQUIRE(sllm_linear_stream_supports(M, N, K) && M <= 32 && N % 16 == 0,
               "linear_stream_silu_scaled: sizes M=%d N=%d K=%d (needs M<=32, N%%16==0, K%%128==0)", M, N, K);
  SLLM_REQUIRE(ssq != nullptr && ((uintptr_t)ssq & 15) == 0 && parts >= 1 && parts <= LS_SSQ_MAX && width >= 1,
               "linear_stream_silu_scaled: a table of %d partial sums (at most %d) over width %d", parts, LS_SSQ_MAX, width);
  LsScale sc;
  sc.ssq = ssq; sc.parts = parts; sc.eps = eps; sc.inv_width = 1.0f / (float)width;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)W;
  if (M <= 8) return launch_ls<1, EPI_SILU, __nv_bfloat16, true>(xb, wb, nullptr, out, nullptr, M, N, K, 1, stream, sc);
  if (M <= 16) return launch_ls<2, EPI_SILU, __nv_bfloat16, true>(xb, wb, nullptr, out, nullptr, M, N, K, 1, stream, sc);
  return launch_ls<4, EPI_SILU, __nv_bfloat16, true>(xb, wb, nullptr, out, nullptr, M, N, K, 1, stream, sc);
}

// ---------------------------------------------------------------------------------------------
// Products of fewer than 16 columns (a router's logits): out[M, N] = x[M, K] W[N, K]^T (+ bias).  A warp a (token, column), 16 bytes a load, the first LN_AHEAD * 256 of a column's
// weights in registers before the wait on the step's earlier kernels.  Bound by latency: one round trip for every LN_AHEAD * 256 columns of K (weights and activations together behind
// the first), a sum over the warp; and for few tokens by what one SM draws from L2, so a CTA there has few columns
// (ln_columns).  (In a graph of such products, us, with eight columns a CTA in two rounds and a loop behind K = 4,096 / so / the library's: 16 tokens, 8 columns, K = 2,048 3.1 / 1.7 / 4.6;
// 48 tokens, 9 columns, K = 2,048 4.3 / 2.0 / 17.9; one token, 9 columns, K = 4,096 6.1 / 1.8 / 3.8, 15 columns, K = 11,008 16.0 / 3.9 / 4.1; 128 tokens, 15 columns, K = 8,192 15.7 / 6.6 /
// 18.8, 10 columns 13.5 / 4.5 / 7.4.)
// ---------------------------------------------------------------------------------------------
namespace sllm {

constexpr int LN_MAX_N = 15, LN_COLS = 4 /* of a CTA, at most */, LN_AHEAD = 16;

__device__ __forceinline__ float ln_dot(const uint4& a, const uint4& b, float sum) {
  const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162*>(&a), *q = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 u = __bfloat1622float2(p[i]), v = __bfloat1622float2(q[i]);
    sum = fmaf(u.x, v.x, sum);
    sum = fmaf(u.y, v.y, sum);
  }
  return sum;
}

template <typename OUT>
__global__ void __launch_bounds__(LN_COLS * 32)
linear_narrow_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias, OUT* __restrict__ out, int N, int K) {
  const int lane = threadIdx.x & 31, n = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  pdl_launch_dependents();
  uint4 w[LN_AHEAD], v[LN_AHEAD];
  auto load = [&](uint4 (&a)[LN_AHEAD], const __nv_bfloat16* row, int k0) {
#pragma unroll
    for (int i = 0; i < LN_AHEAD; ++i) {
      const int k = k0 + (lane + 32 * i) * 8;
      a[i] = n < N && k < K ? *reinterpret_cast<const uint4*>(row + k) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  load(w, W + (size_t)n * K, 0);
  pdl_wait();
  float sum = 0.f;
  for (int k0 = 0; k0 < K; k0 += LN_AHEAD * 256) {
    if (k0 > 0) load(w, W + (size_t)n * K, k0);
    load(v, x + (size_t)blockIdx.x * K, k0);
#pragma unroll
    for (int i = 0; i < LN_AHEAD; ++i)
      if (k0 + (lane + 32 * i) * 8 < K) sum = ln_dot(v[i], w[i], sum);
  }
  sum = warp_sum(sum);
  if (lane == 0 && n < N) out[(size_t)blockIdx.x * N + n] = from_f32<OUT>(sum + (bias ? bias[n] : 0.f));
}

// Columns of a CTA: as few as make two CTAs an SM, at most (each reads the token's row again).
static int ln_columns(int M, int N) {
  int cols = 1;
  while (cols < LN_COLS && (long long)M * ((N + cols - 1) / cols) > 2 * num_sms()) ++cols;
  return cols < N ? cols : N;
}

}  // namespace sllm

SLLM_EXPORT int sllm_linear_narrow(const void* x, const void* W, const float* bias, void* out, int out_dtype, int M, int N, int K, cudaStream_t stream) {
  SLLM_REQUIRE(M >= 1 && N >= 1 && N <= LN_MAX_N && K >= 8 && K % 8 == 0, "linear_narrow: sizes M=%d N=%d K=%d (needs N<=15, K%%8==0)", M, N, K);
  SLLM_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)W & 15) == 0, "linear_narrow: operands must be 16-byte aligned");
  const int cols = ln_columns(M, N);
  const dim3 grid(M, (N + cols - 1) / cols);
  if (out_dtype == SLLM_BF16)
    launch_kernel(linear_narrow_kernel<__nv_bfloat16>, grid, cols * 32, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)W, bias, (__nv_bfloat16*)out, N, K);
  else
    launch_kernel(linear_narrow_kernel<float>, grid, cols * 32, 0, stream, (const __nv_bfloat16*)x, (const __nv_bfloat16*)W, bias, (float*)out, N, K);
  return launch_status("linear_narrow");
}

// ---------------------------------------------------------------------------------------------
// An entry point that allocates nothing (declared in sllm_noalloc.h; see the comment there).
// ---------------------------------------------------------------------------------------------
#include <mutex>

#include "sllm_noalloc.h"

namespace sllm {

// Scratch for the k-split partial sums, part of the library's image: every GPU that loads the
// library holds these 8 MiB until the process exits.
static __device__ __align__(256) float ls_noalloc_scratch[SLLM_NOALLOC_SCRATCH_FLOATS];

constexpr int NOALLOC_MAX_DEVICES = 64;
static float* g_noalloc_ptr[NOALLOC_MAX_DEVICES];      // device address of the array, per device
static std::mutex g_noalloc_mutex;

// out[i] = sum over splits of partial[s][i]
__global__ void sum_partials_kernel(const float* partial, int splits, size_t n, float* __restrict__ out) {
  pdl_wait();
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float v = 0.f;
  for (int s = 0; s < splits; ++s) v += partial[(size_t)s * n + i];
  out[i] = v;
}

}  // namespace sllm

SLLM_EXPORT int sllm_linear_stream_noalloc(const void* x, const void* W, const float* bias, float* out, int M, int N,
                                           int K, int splits, cudaStream_t stream) {
  SLLM_REQUIRE(sllm_linear_stream_supports(M, N, K), "linear_stream_noalloc: sizes M=%d N=%d K=%d (needs M<=64, K%%128==0)", M, N, K);
  SLLM_REQUIRE(splits >= 1, "linear_stream_noalloc: splits=%d", splits);
  const int real = sllm_linear_stream_splits(K, splits);
  if (real == 1)        // nothing to add up: the product goes straight to the caller's buffer
    return sllm_linear_stream(x, W, bias, out, SLLM_F32, nullptr, M, N, K, 1, EPI_STORE, stream);
  const size_t need = (size_t)real * M * N;
  SLLM_REQUIRE(need <= (size_t)SLLM_NOALLOC_SCRATCH_FLOATS,
               "linear_stream_noalloc: %d splits x %d x %d partial sums need %zu floats, the built-in scratch holds %d",
               real, M, N, need, SLLM_NOALLOC_SCRATCH_FLOATS);
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
    set_error("linear_stream_noalloc: cannot tell the current device");
    return SLLM_ERR_LAUNCH;
  }
  float* scratch;
  {
    // The array's name is a host-side handle, not a device address: its address on the
    // current device is asked for once per device and kept.
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_ptr[dev] == nullptr) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, ls_noalloc_scratch);
      if (e != cudaSuccess || p == nullptr) {
        char buf[200];
        snprintf(buf, sizeof buf, "linear_stream_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        set_error(buf);
        return SLLM_ERR_LAUNCH;
      }
      g_noalloc_ptr[dev] = static_cast<float*>(p);
    }
    scratch = g_noalloc_ptr[dev];
  }
  int rc = sllm_linear_stream(x, W, bias, nullptr, SLLM_F32, scratch, M, N, K, real, EPI_STORE, stream);
  if (rc != SLLM_OK) return rc;
  const size_t n = (size_t)M * N;
  launch_kernel(sum_partials_kernel, (unsigned)((n + 255) / 256), 256, 0, stream, (const float*)scratch, real, n, out);
  return launch_status("linear_stream_noalloc");
}
