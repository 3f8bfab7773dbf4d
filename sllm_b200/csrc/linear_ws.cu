// Weight-streaming linear layer for at most 16 tokens (32 for small matrices): y[M, N] = x[M, K] W[N, K]^T.
//
// linear_stream.cu gives 128 weight rows to a CTA and, when N is small, splits K over the grid,
// leaving partial sums for the consumer.  Here a CTA owns 16 output rows at a time over the whole of K and
// its 8 warps split K among themselves: warp w takes the 32-wide k blocks w, w+8, w+16, ...
// (so the CTA reads 512 contiguous bytes of each row at a time), four blocks in flight per warp,
// weights and activations both loaded straight into MMA fragments (same k permutation as in
// linear_stream.cu), no shared memory and no barrier inside the loop.  At the end the warps'
// partial tiles are added through shared memory in warp order (a fixed order), and since the CTA
// holds complete sums the epilogue can finish the layer's job:
//   store      out[M, N] (+ bias), float32 or bfloat16
//              optionally through an activation: max(v, 0)^2, or gelu_tanh(v) times the token's own entry of a table
//   residual   residual[M, N] += y (+ bias): the float32 stream is updated in place, so the next
//              norm has nothing to add
//   gated      act(gate) * up of a gate|up matrix whose rows alternate in blocks of 8: local row r < 8 is a pair's gate row,
//              r + 8 its up row, act SiLU or the tanh form of GELU
//   rotary     for the fused q|k|v matrix of an attention layer: bias, rotary encoding and the write
//              of the new keys and values into their cache pages, so that the decode step needs no
//              kernel between this product and the attention.  A CTA then takes the 8 rows j..j+7
//              of a head and the 8 rows hd/2 apart: the two rows of a rotation pair are the two
//              rows (g, g+8) of one MMA accumulator, and meet in one thread of the epilogue
//              (ref/qwen3_5.py:355-370; cache content ref/incremental.py:135-139).
// About N/16 CTAs keep every SM busy without splitting K over the grid, at most two an SM, the rows dealt evenly (N = 3584: 296 CTAs of
// 12 or 13 rows instead of 224 of 16, of which 76 SMs would get two and 72 one; N = 11264: 296 CTAs of 38 rows in three groups).
//
// The reference calls cublasGemmEx for these products and adds the residual in its next
// add_rms kernel (kernels/cuda/kernels.cu:752-767, 791-839; kernels/device_decode.py:312-325).
#include <cooperative_groups.h>
#include <stdio.h>

#include <atomic>

#include "common.cuh"

namespace sllm {

#define WS_EPI_STORE 0
#define WS_EPI_RESID 1
#define WS_EPI_ROPE 2
#define WS_EPI_GATED 3

// what the rotary epilogue needs beside the product: the rows of W are q heads, then k heads, then v
// heads of `hd` rows each; table [max_pos][2][hd/2] holds cos then sin (rotary_dim == hd), or is null
// (no rotation); a token's key and value go to slot_mapping[token] of the paged caches
// [page][kv head][slot in page][hd] (null: not written), its queries to q_out [M, nq * hd].
struct WsRope {
  const int* positions;
  const float* table;
  const int* slot_mapping;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  __nv_bfloat16* q_out;
  int max_pos, nq, nkv, hd, page_size, num_pages;
};

__device__ __forceinline__ int ws_position(const int* p) {        // which another kernel may be writing: from L2, and nothing stays in L1
  int pos;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(pos) : "l"(p));
  return pos;
}

__device__ __forceinline__ uint4 ws_ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ws_ldg(const void* p) {       // activations: small, shared by all CTAs, keep in L1
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void ws_copy4(void* smem, const void* p) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(p) : "memory");
}
__device__ __forceinline__ void ws_mma(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                       unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr int WS_WARPS = 8;
constexpr int WS_SLICES = 4;        // slices of K a cluster shares at most
constexpr int WS_SIDE = 4;          // groups of rows side by side in a CTA of that form
// k blocks a warp keeps in flight per group (two groups): with two token tiles half as many, so that the
// activation fragments fit the registers of two CTAs an SM (four: 174 registers a thread, one CTA an SM)
__host__ __device__ constexpr int ws_depth(int nt) { return nt == 1 ? 4 : (nt == 2 ? 2 : 1); }
constexpr int WS_SSQ_MAX = 608;     // partial sums of squares per token a consumer takes (the producer's CTAs: at most 592 for 8192 columns)
#define WS_GATE_SILU 0
#define WS_GATE_GELU 1
// with four token tiles (17..32 tokens: small matrices only, where a step is bound by its number of kernels) the table
// is kept to what fits static shared memory beside the warps' tiles: streams of up to 3,072 columns
__host__ __device__ constexpr int ws_ssq_max(int nt) { return nt <= 2 ? WS_SSQ_MAX : 192; }

// An RMSNorm taken apart, so that a decode step needs no kernel for it (y = x * rsqrt(mean(x^2) + eps) * gain,
// ref/standard.py:25-31).  The product that completes the residual stream (residual epilogue) also writes
// xg_out = bfloat16(stream * gain) and, per CTA, each token's sum of squares over the CTA's columns of the
// stream (ssq_out[token][cta]); the product that consumes the normed activations reads xg as its input and
// multiplies each token's row of its result by rsqrt(sum of the token's partial sums / width + eps):
// W (x g / rms) = (W (x g)) / rms.  The partial sums are added in a fixed order.  A table of partial sums is
// [tokens][stride] float32 with stride = parts rounded up to a multiple of 4 (rows start on 16 bytes); what
// lies between parts and stride is never written and never added.
struct WsNorm {
  const float* ssq_in = nullptr;     // consumer: [M][(parts_in + 3) & ~3]
  int parts_in = 0;
  float eps_in = 0.f, inv_width_in = 0.f;
  const float* gain = nullptr;       // producer (residual epilogue): the next norm's gain [N]
  __nv_bfloat16* xg_out = nullptr;   // [M, N]
  float* ssq_out = nullptr;          // [M][(CTAs of rows + 3) & ~3]
};

// NT: 8-token tiles (M <= 8 * NT).  OUT: float or __nv_bfloat16 (store epilogue only).  SCALED: the input
// comes with a norm still owed (WsNorm::ssq_in).
// FORM: one group of rows a CTA; several, one after the other; one that the CTAs of a cluster share, each a slice of K (store and
// residual epilogues); or four side by side, two warps each (store and gated).
#define WS_ONE 0
#define WS_WALK 1
#define WS_SLICED 2
#define WS_ROWS 3
template <int NT, int EPI, typename OUT, bool SCALED, int FORM>
__global__ void __launch_bounds__(WS_WARPS * 32, 2)
linear_ws_kernel(const __nv_bfloat16* x, const __nv_bfloat16* __restrict__ W,
                 const float* __restrict__ bias, OUT* __restrict__ out, float* residual,
                 int M, int N, int K, const WsRope rope, const WsNorm norm, const int act, const TokenTable token, const int slices_) {
  constexpr int WS_DEPTH = ws_depth(NT);
  constexpr bool SLICED = FORM == WS_SLICED, ROWS = FORM == WS_ROWS;
  constexpr int KW = ROWS ? WS_WARPS / WS_SIDE : WS_WARPS, RW = WS_WARPS / KW;      // warps of a group of rows, groups side by side
  __shared__ float red[WS_WARPS][16][8 * NT + 1];
  __shared__ float row_scale[8 * NT];
  __shared__ float slice_sum[SLICED ? WS_SLICES : 1][SLICED ? 16 * 8 * NT : 1];
  __shared__ __align__(16) float ssq_s[SCALED ? 8 * NT : 1][SCALED ? ws_ssq_max(NT) : 4];
  // What the thread's own outputs will need beside the product, copied under the stream of weights: a load behind the last sums is a miss in HBM for what no kernel of the step
  // writes (gain, bias, cos and sin: a step's weights push them out of L2), one in L2 for the stream.  (In a graph of such products, us, before / now: residual
  // with the next norm's input 896 x 896, one token 2.74 / 2.36, 3,584 x 3,584, 8 tokens 7.80 / 7.11, 2,048 x 5,632, 32 tokens 10.3 / 9.3; rotary 1,152 x 896, one token 3.43 / 2.81.)
  // (A residual form that itself has a norm owed does without, and two token tiles with a norm owed keep no bias: shared memory.)
  constexpr bool AHEAD = (EPI == WS_EPI_RESID && !SCALED && (FORM == WS_ONE || FORM == WS_SLICED)) || EPI == WS_EPI_ROPE;
  constexpr bool BIAS_AHEAD = !(SCALED && NT == 2);
  constexpr int AHEAD_N = EPI == WS_EPI_ROPE ? 64 * NT : (16 * 8 * NT + WS_WARPS * 32 - 1) / (WS_WARPS * 32) * WS_WARPS * 32;
  __shared__ int token_s[EPI == WS_EPI_ROPE ? 3 : 1][EPI == WS_EPI_ROPE ? 8 * NT : 1];      // rotary: the position its angles were copied for, its position, its slot
  __shared__ float ahead[AHEAD ? (EPI == WS_EPI_ROPE ? (BIAS_AHEAD ? 4 : 2) : 3) : 1][AHEAD ? AHEAD_N : 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  // The CTA's rows [c0, c1), the N rows dealt evenly over the grid (so that a grid of a whole number of CTAs per SM gives
  // every SM the same bytes to stream), taken in groups of at most 16, these too as even as they get.  Gated: the same over pairs
  // of a gate row and its up row, in groups of at most 8.
  constexpr int PER = EPI == WS_EPI_GATED ? 8 : 16;
  const int units = EPI == WS_EPI_GATED ? N / 2 : N;
  const int slices = SLICED ? slices_ : 1;
  const int cta = blockIdx.x / slices, ctas = gridDim.x / slices, slice = blockIdx.x % slices;
  const int c0 = (int)(((long long)cta * units) / ctas), c1 = (int)(((long long)(cta + 1) * units) / ctas);
  const int groups = FORM != WS_WALK ? 1 : (c1 - c0 + PER - 1) / PER;
  const int k_first = SLICED ? K / 32 * slice / slices : 0, k_blocks = SLICED ? K / 32 * (slice + 1) / slices : K / 32;      // the CTA's k blocks
  int n0, n1;                            // the group's units
  const __nv_bfloat16 *w0, *w1;          // the lane's two rows of the group
  auto take = [&](int i) {
    n0 = c0 + (int)(((long long)i * (c1 - c0)) / (ROWS ? RW : groups));
    n1 = c0 + (int)(((long long)(i + 1) * (c1 - c0)) / (ROWS ? RW : groups));
    int r0 = min(n0 + g, n1 - 1), r1 = min(n0 + g + 8, n1 - 1);   // rows past the group's: clamped loads, skipped stores
    if constexpr (EPI == WS_EPI_ROPE) {
      // CTA b of a head's hd/16: rows [8c, 8c+8) of the head and the 8 rows hd/2 further
      const int per_head = rope.hd / 16;
      n0 = ((int)blockIdx.x / per_head) * rope.hd + ((int)blockIdx.x % per_head) * 8;
      n1 = n0 + 16;                                  // (not a range: local row r is n0 + (r & 7) + (r >> 3) * hd/2)
      r0 = n0 + g;
      r1 = n0 + rope.hd / 2 + g;
    }
    if constexpr (EPI == WS_EPI_GATED) {
      r0 = r0 / 8 * 16 + r0 % 8;                     // pair q: gate row 16 (q / 8) + q % 8, up row 8 further
      r1 = r0 + 8;
    }
    w0 = W + (size_t)r0 * K + t4 * 8;
    w1 = W + (size_t)r1 * K + t4 * 8;
  };
  take(ROWS ? warp / KW : 0);
  const __nv_bfloat16* xr[NT];
#pragma unroll
  for (int j = 0; j < NT; ++j) xr[j] = x + (size_t)min(8 * j + g, M - 1) * K + t4 * 8;   // tokens past M: clamped, skipped

  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;

  // Two groups of WS_DEPTH k blocks are in flight per warp: while one is multiplied, the loads of
  // the next (weights and activations) are already under way.  The first weights do not depend
  // on the step's earlier kernels and are fetched before the wait; the activations after it.
  uint4 wa0[WS_DEPTH], wb0[WS_DEPTH], wa1[WS_DEPTH], wb1[WS_DEPTH];
  uint4 x0[WS_DEPTH][NT], x1[WS_DEPTH][NT];
  auto load_w = [&](uint4 (&wa)[WS_DEPTH], uint4 (&wb)[WS_DEPTH], int kb) {
#pragma unroll
    for (int d = 0; d < WS_DEPTH; ++d) {
      const int b = kb + d * KW;
      if (b < k_blocks) {
        wa[d] = ws_ldg_stream(w0 + (size_t)b * 32);
        wb[d] = ws_ldg_stream(w1 + (size_t)b * 32);
      }
    }
  };
  auto load_x = [&](uint4 (&xv)[WS_DEPTH][NT], int kb) {
#pragma unroll
    for (int d = 0; d < WS_DEPTH; ++d) {
      const int b = kb + d * KW;
      if (b < k_blocks) {
#pragma unroll
        for (int j = 0; j < NT; ++j) xv[d][j] = ws_ldg(xr[j] + (size_t)b * 32);
      }
    }
  };
  auto compute = [&](const uint4 (&wa)[WS_DEPTH], const uint4 (&wb)[WS_DEPTH], const uint4 (&xv)[WS_DEPTH][NT], int kb) {
#pragma unroll
    for (int d = 0; d < WS_DEPTH; ++d) {
      if (kb + d * KW < k_blocks) {
        // (a token tile's two products depend on one another: the tiles' first ones, then their second ones)
#pragma unroll
        for (int j = 0; j < NT; ++j) ws_mma(acc[j], wa[d].x, wb[d].x, wa[d].y, wb[d].y, xv[d][j].x, xv[d][j].y);
#pragma unroll
        for (int j = 0; j < NT; ++j) ws_mma(acc[j], wa[d].z, wb[d].z, wa[d].w, wb[d].w, xv[d][j].z, xv[d][j].w);
      }
    }
  };
  constexpr int GROUP = WS_DEPTH * KW;        // k blocks the CTA covers per group
  const int k_mine = k_first + warp % KW;
  int kb = k_mine;
  // Rotary: a token's position is taken twice.  Before the wait it may still be on its way from an earlier kernel, so it only says which angles to copy; behind the wait it is the token's, and the
  // epilogue looks the angles up again where the two differ.  (Behind the wait alone the product waits for two misses one behind the other: 1,152 x 896, one token 2.45 -> 3.06 us.  In shared
  // memory, because registers are weights in flight: 4,608 x 3,584 7.5 -> 8.5 us with two more.)
  const int ahead_tok = tid / 8, ahead_i = tid % 8;
  const bool ahead_mine = EPI == WS_EPI_ROPE && tid < AHEAD_N && ahead_tok < M;
  int ahead_pos = 0;
  if constexpr (EPI == WS_EPI_ROPE) {         // (one load a token: its eight threads copy the same angles)
    if (ahead_mine && ahead_i == 0 && rope.table != nullptr) ahead_pos = token_s[0][ahead_tok] = min(max(ws_position(rope.positions + ahead_tok), 0), rope.max_pos - 1);
    ahead_pos = __shfl_sync(0xffffffffu, ahead_pos, lane & 24);
  }
  load_w(wa0, wb0, kb);
  if constexpr (EPI == WS_EPI_ROPE) {
    if (ahead_mine && rope.table != nullptr) {
      const float* cs = rope.table + (size_t)ahead_pos * rope.hd + n0 % rope.hd + ahead_i;        // cos[half] then sin[half]
      ws_copy4(&ahead[0][tid], cs);
      ws_copy4(&ahead[1][tid], cs + rope.hd / 2);
    }
    if (ahead_mine && BIAS_AHEAD && bias) {
      ws_copy4(&ahead[BIAS_AHEAD ? 2 : 0][tid], bias + n0 + ahead_i);
      ws_copy4(&ahead[BIAS_AHEAD ? 3 : 0][tid], bias + n0 + rope.hd / 2 + ahead_i);
    }
  }
  auto resid_at = [&](auto&& use) {           // the thread's outputs of the CTA's only group
    for (int idx = tid; idx < 16 * 8 * NT; idx += WS_WARPS * 32) {
      const int tok = idx / 16, n = n0 + idx % 16;
      if (tok < M && n < n1 && slice == 0) use(idx, tok, n);
    }
  };
  if constexpr (EPI == WS_EPI_RESID && AHEAD) {
    resid_at([&](int idx, int, int n) {
      if (norm.gain != nullptr) ws_copy4(&ahead[0][idx], norm.gain + n);
      if (bias) ws_copy4(&ahead[1][idx], bias + n);
    });
  }
  if constexpr (SLICED) cooperative_groups::this_cluster().sync();      // nobody writes to a CTA that has not begun
  pdl_wait();
  if constexpr (EPI == WS_EPI_ROPE) {
    if (ahead_mine && ahead_i == 0 && rope.table != nullptr) ws_copy4(&token_s[1][ahead_tok], rope.positions + ahead_tok);
    if (ahead_mine && ahead_i == 0 && rope.slot_mapping != nullptr) ws_copy4(&token_s[2][ahead_tok], rope.slot_mapping + ahead_tok);
  }
  load_x(x0, kb);
  if constexpr (EPI == WS_EPI_RESID && AHEAD) resid_at([&](int idx, int tok, int n) { ws_copy4(&ahead[2][idx], residual + (size_t)tok * N + n); });
  if constexpr (AHEAD) asm volatile("cp.async.commit_group;\n" ::);
  // a norm still owed on the input: the tokens' partial sums of squares are copied to shared memory under
  // the stream and added after the loop
  if constexpr (SCALED) {
    const int stride = (norm.parts_in + 3) & ~3, chunks = stride >> 2;
    for (int c = tid; c < M * chunks; c += WS_WARPS * 32) {
      const int tok = c / chunks, piece = c % chunks;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(&ssq_s[tok][piece * 4]);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(norm.ssq_in + (size_t)tok * stride + piece * 4));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  }
  constexpr int OUTS = (16 * 8 * NT * RW + WS_WARPS * 32 - 1) / (WS_WARPS * 32);
  float squares[OUTS];                   // residual epilogue: of the thread's places, over the groups
#pragma unroll
  for (int o = 0; o < OUTS; ++o) squares[o] = 0.f;
  for (int group = 0; group < groups; ++group) {
    const int m0 = n0, m1 = n1;          // (the next group's rows are taken while this one's last blocks are multiplied)
    if constexpr (FORM != WS_ONE) {     // (also the better code for the slices: 2,048 x 11,264 10.8 us against 14.5)
      for (kb = k_mine;; kb += 2 * GROUP) {
        load_w(wa1, wb1, kb + GROUP);
        load_x(x1, kb + GROUP);
        compute(wa0, wb0, x0, kb);
        const bool more = kb + 2 * GROUP < k_blocks;
        if (more || group + 1 < groups) {
          if (!more) take(group + 1);
          load_w(wa0, wb0, more ? kb + 2 * GROUP : k_mine);
          load_x(x0, more ? kb + 2 * GROUP : k_mine);
        }
        compute(wa1, wb1, x1, kb + GROUP);
        if (!more) break;
      }
    } else {
      for (; kb < k_blocks; kb += 2 * GROUP) {
        load_w(wa1, wb1, kb + GROUP);
        load_x(x1, kb + GROUP);
        compute(wa0, wb0, x0, kb);
        load_w(wa0, wb0, kb + 2 * GROUP);
        load_x(x0, kb + 2 * GROUP);
        compute(wa1, wb1, x1, kb + GROUP);
      }
    }
    if (group + 1 == groups) pdl_launch_dependents();

    // ---- add the warps' tiles in warp order; acc[j][c]: c0,c1 = (row g, tokens 8j+2t, +1); c2,c3 = (row g+8, ...) ----
    if (group > 0) __syncthreads();      // the group before has been read
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        red[warp][g + ((c & 2) ? 8 : 0)][8 * j + 2 * t4 + (c & 1)] = acc[j][c];
        acc[j][c] = 0.f;
      }
    if constexpr (SCALED || AHEAD) {
      if (group == 0) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    if constexpr (SCALED) {
      if (group == 0) {
        // warp w adds the partial sums of tokens w, w + 8: lane l takes l, l + 32, ..., then the lanes are added
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int tok = warp + 8 * j;
          float sum = 0.f;
          if (tok < M)
            for (int p = lane; p < norm.parts_in; p += 32) sum += ssq_s[tok][p];
          sum = warp_sum(sum);
          if (lane == 0) row_scale[tok] = rsqrtf(sum * norm.inv_width_in + norm.eps_in);
        }
        __syncthreads();
      }
    }
    if constexpr (EPI == WS_EPI_ROPE) {
      const int half = rope.hd / 2;
      const int head = m0 / rope.hd, j0 = m0 % rope.hd;            // j0 = 8c: the pair's lower dimension starts here
      const int i = ahead_i, tok = ahead_tok;                        // consecutive threads -> consecutive dimensions of one token; at most one output a thread
      if (ahead_mine) {
        float lo = 0.f, hi = 0.f;
#pragma unroll
        for (int w = 0; w < WS_WARPS; ++w) { lo += red[w][i][tok]; hi += red[w][i + 8][tok]; }
        if constexpr (SCALED) {
          lo *= row_scale[tok];
          hi *= row_scale[tok];
        }
        if (bias) {
          lo += BIAS_AHEAD ? ahead[BIAS_AHEAD ? 2 : 0][tid] : bias[m0 + i];
          hi += BIAS_AHEAD ? ahead[BIAS_AHEAD ? 3 : 0][tid] : bias[m0 + half + i];
        }
        __nv_bfloat16* dst;
        if (head < rope.nq) {
          dst = rope.q_out + ((size_t)tok * rope.nq + head) * rope.hd;
        } else {
          const int slot = rope.slot_mapping != nullptr ? token_s[2][tok] : -1;
          if (slot < 0 || slot / rope.page_size >= rope.num_pages) return;     // not written (padding row, borrowed cache)
          const bool is_k = head < rope.nq + rope.nkv;
          const int kvh = is_k ? head - rope.nq : head - rope.nq - rope.nkv;
          dst = (is_k ? rope.k_cache : rope.v_cache) +
                (((size_t)(slot / rope.page_size) * rope.nkv + kvh) * rope.page_size + slot % rope.page_size) * rope.hd;
        }
        if (rope.table != nullptr && head < rope.nq + rope.nkv) {
          float c = ahead[0][tid], sn = ahead[1][tid];
          const int pos = min(max(token_s[1][tok], 0), rope.max_pos - 1);
          if (pos != token_s[0][tok]) {
            c = rope.table[(size_t)pos * rope.hd + j0 + i];
            sn = rope.table[(size_t)pos * rope.hd + half + j0 + i];
          }
          const float a = lo * c - hi * sn, b = hi * c + lo * sn;
          lo = a;
          hi = b;
        }
        dst[j0 + i] = __float2bfloat16_rn(lo);
        dst[j0 + half + i] = __float2bfloat16_rn(hi);
      }
      return;
    }
    if constexpr (EPI == WS_EPI_GATED) {
      for (int idx = tid; idx < 8 * 8 * NT * RW; idx += WS_WARPS * 32) {
        const int i = idx % 8, tok = idx / 8 % (8 * NT), rg = idx / (64 * NT);
        const int q = (ROWS ? c0 + rg * (c1 - c0) / RW : m0) + i;
        if (tok >= M || q >= (ROWS ? c0 + (rg + 1) * (c1 - c0) / RW : m1)) continue;
        float gate = 0.f, up = 0.f;
#pragma unroll
        for (int w = 0; w < KW; ++w) { gate += red[rg * KW + w][i][tok]; up += red[rg * KW + w][i + 8][tok]; }
        if constexpr (SCALED) {
          gate *= row_scale[tok];
          up *= row_scale[tok];
        }
        if (bias) {
          gate += bias[q / 8 * 16 + q % 8];
          up += bias[q / 8 * 16 + q % 8 + 8];
        }
        out[(size_t)tok * units + q] = from_f32<OUT>((act == WS_GATE_GELU ? gelu_tanh_f32(gate) : gate * sigmoid_f32(gate)) * up);
      }
      continue;
    }
    if constexpr (SLICED) {              // the slices' sums in the first CTA, added there in the slices' order
      cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
      for (int idx = tid; idx < 16 * 8 * NT; idx += WS_WARPS * 32) {
        const int row = idx % 16, tok = idx / 16;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < WS_WARPS; ++w) v += red[w][row][tok];
        cl.map_shared_rank(&slice_sum[0][0], 0)[slice * (16 * 8 * NT) + idx] = v;
      }
      cl.sync();
      if (slice != 0) return;
    }
#pragma unroll
    for (int o = 0; o < OUTS; ++o) {
      const int idx = tid + o * WS_WARPS * 32;
      if (idx >= 16 * 8 * NT * RW) break;                 // (whole warps: 16 * 8 * NT is a multiple of 32)
      const int row = idx % 16, tok = idx / 16 % (8 * NT), rg = idx / (128 * NT);       // consecutive threads -> consecutive rows of one token
      const int n = (ROWS ? c0 + rg * (c1 - c0) / RW : m0) + row;
      if (tok >= M || n >= (ROWS ? c0 + (rg + 1) * (c1 - c0) / RW : m1)) continue;
      float v = 0.f;
      if constexpr (SLICED) {
        for (int w = 0; w < slices; ++w) v += slice_sum[w][idx];
      } else {
#pragma unroll
        for (int w = 0; w < KW; ++w) v += red[rg * KW + w][row][tok];
      }
      if constexpr (SCALED) v *= row_scale[tok];
      if (bias) v += EPI == WS_EPI_RESID && AHEAD ? ahead[AHEAD ? 1 : 0][AHEAD ? idx : 0] : bias[n];
      if constexpr (EPI == WS_EPI_RESID) {
        const float r = (AHEAD ? ahead[AHEAD ? 2 : 0][AHEAD ? idx : 0] : residual[(size_t)tok * N + n]) + v;
        residual[(size_t)tok * N + n] = r;
        if (norm.xg_out != nullptr) {
          norm.xg_out[(size_t)tok * N + n] = __float2bfloat16_rn(r * (AHEAD ? ahead[0][AHEAD ? idx : 0] : norm.gain[n]));
          squares[o] = fmaf(r, r, squares[o]);
        }
      } else {
        if (act == SLLM_ACT_RELU2) v = relu2_f32(v);
        else if (act == SLLM_ACT_GELU) v = gelu_f32(v);
        else if (act == SLLM_ACT_TOKEN) v = gelu_tanh_f32(v) * __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(token.table)[token_row(token, tok) + n]);
        out[(size_t)tok * N + n] = from_f32<OUT>(v);
      }
    }
  }
  if constexpr (EPI == WS_EPI_RESID) {
    if (norm.ssq_out != nullptr) {
#pragma unroll
      for (int o = 0; o < OUTS; ++o) {                    // the 16 rows of a token lie in 16 consecutive lanes
        const int idx = tid + o * WS_WARPS * 32;
        if (idx >= 16 * 8 * NT) break;
        float sq = squares[o];
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, w);
        if (idx % 16 == 0 && idx / 16 < M) norm.ssq_out[(size_t)(idx / 16) * ((ctas + 3) & ~3) + cta] = sq;
      }
    }
  }
}

// CTAs (of rows) of 16 units, or more of fewer where those would fill the SMs unevenly (two CTAs share an SM): between one
// and two CTAs an SM the next multiple of the SM count (N = 3584: 296 CTAs of 12 or 13 rows for 224 of 16).  Beyond two an SM and up to 8,192
// rows a group a CTA, in full groups (N = 5120, 8 tokens, K = 5120: 13.5 us with 320 CTAs, 14.5 with 592, 14.4 with 296 of two groups of 8 or 9 rows)
// unless the rows are long (K = 27648: 50.4 us with 592 against 61.4).  More rows: two CTAs an SM that walk theirs in groups, the next
// group's first blocks in flight under this one's last and its sums, where a CTA a group paid a ramp and a tail each.
// (8 tokens, us, this / the 128-row form of linear_stream.cu; floor at 6.65 TB/s: 11,264 x 2,048 10.9 / 17.8 / 6.9, 16,512 x 4,096 24.7 / 36.3 / 20.3,
// 22,016 x 4,096 31.3 / 39.8 / 27.1, 152,064 x 3,584 168 / 188 / 164.)  A short K leaves a group too little to stream under its sums (20,000 x 1,024: 12.9 walked, 11.9 a CTA a group).
constexpr int WS_ONE_GROUP_ROWS = 8192, WS_WALK_MIN_K = 1280;
static int ws_ctas(int units, int per, int K, bool rope) {
  const int num_sms = sllm::num_sms();
  const int ctas = (units + per - 1) / per;
  if (rope || ctas <= num_sms) return ctas;
  if (ctas < 2 * num_sms) return 2 * num_sms <= units ? 2 * num_sms : ctas;
  if (ctas * 16 > WS_ONE_GROUP_ROWS) return K >= WS_WALK_MIN_K ? 2 * num_sms : ctas;
  const int even = K > 8192 ? (ctas + 2 * num_sms - 1) / (2 * num_sms) * (2 * num_sms) : ctas;
  return even <= units ? even : ctas;
}
// Slices of K by the CTAs of a cluster: where the rows give less than one CTA an SM, as many (1, 2, 4) as two an SM hold, none shorter than 16 k blocks, and
// only of a K that is worth the pass over the cluster's sums.
// (us, in slices / in one. 8 tokens, residual epilogue: 896 x 4,864 4.5 / 6.1; 2,048 x 2,048 4.2 / 4.6; 2,048 x 1,536 3.8 / 4.2; 1,024 x 1,024 2.9 / 2.8. 8 tokens, store: 512 x
// 2,560 3.1 / 3.9; 256 x 2,048 2.7 / 2.5; 1,024 x 1,024 2.8 / 2.2. 16 tokens: 512 x 2,048 2.9 / 3.3; 2,048 x 1,536 4.3 / 3.6.)
static int ws_slices(int ctas, int K, int M, bool residual) {
  if (K < (M > 8 ? 2048 : residual ? 1536 : 2080)) return 1;
  int s = 1;
  while (s < WS_SLICES && ctas * s * 2 <= 2 * sllm::num_sms() && K / 32 / (s * 2) >= 16) s *= 2;
  return s;
}

// Whether a CTA takes four groups of rows side by side where it would walk them: with two warps a group a short K leaves each warp a stream of
// its own in place of one round of loads between two sums.  Where its CTAs fit the SMs at once or end in a wave that is nearly full; 9..16 tokens, whose
// activations leave a warp half the weights in flight, only a short K at once.  (Store, us, side by side / walk / linear_stream.cu, 8 tokens: 9,728 x 896 6.1 / 7.7
// / 8.0, 17,920 x 1,536 10.3 / 12.9 / 14.8, 11,264 x 2,048 10.4 / 10.7 / 17.8, 37,888 x 3,584 44.0 / 46.2 / 44.8, 151,936 x 1,536 74 / 87 / 81; beyond the line
// 22,528 x 2,048 20.4 / 18.3, 22,016 x 4,096 38.5 / 31.5.  16 tokens: 9,728 x 896 7.2 / 7.6 / 8.2, 17,920 x 1,536 12.1 / 15.5 / 15.6; 11,264 x 2,048 13.6 / 12.6.)
static bool ws_side_by_side(int M, int N, int K) {
  const int places = 2 * sllm::num_sms(), ctas = (N + 16 * WS_SIDE - 1) / (16 * WS_SIDE);
  if (M > 8) return K < 2048 && ctas <= places;
  return ctas <= places || ctas * 100 >= (ctas + places - 1) / places * places * 84;
}

// The kernel, told once a device what shared memory it wants beside L1: what two CTAs need, at least WS_CARVEOUT per cent.  The loads in flight lie in L1, and an SM keeps the split that the kernel
// before had as long as the next one's shared memory fits: behind the decode attention, which takes all of it, this kernel ran with 28 KB of L1 (at 7B sizes gate|up 65 us in place of 45,
// down 67 in place of 25, as soon as no small kernel stood between them).  (8 requests at 7B sizes, 8 of 240 keys at a width of 2,048, 16 of 300, one of 700 at 4,096, ms: no preference 195, 20.0, 29.4, 17.2;
// 0 per cent beyond what fits 131.6, 19.8, 29.4, 16.8; 30 131.6, 19.4, 28.6, 16.6; 60 138.9, 21.4, 28.9, 18.4.)
constexpr int WS_CARVEOUT = 30, WS_SM_SHARED = 228 * 1024;
template <int NT, int EPI, typename OUT, bool SCALED, int FORM>
static auto ws_kernel() {
  auto kernel = linear_ws_kernel<NT, EPI, OUT, SCALED, FORM>;
  static std::atomic<unsigned long long> told{0};                       // a bit a device
  int dev = 0;
  cudaFuncAttributes at;
  if (cudaGetDevice(&dev) == cudaSuccess && dev < 64 && !(told.fetch_or(1ull << dev) >> dev & 1) && cudaFuncGetAttributes(&at, kernel) == cudaSuccess) {
    const int fit = (int)(2 * (at.sharedSizeBytes + 1024) * 100 / WS_SM_SHARED) + 1;
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, fit > WS_CARVEOUT ? fit : WS_CARVEOUT);      // (a preference; nothing depends on it but time)
  }
  return kernel;
}

template <int NT, int EPI, typename OUT>
static int launch_ws(const __nv_bfloat16* x, const __nv_bfloat16* W, const float* bias, void* out, float* residual,
                     int M, int N, int K, cudaStream_t stream, const WsRope& rope = WsRope{}, const WsNorm& norm = WsNorm{},
                     int act = SLLM_ACT_NONE, const TokenTable& token = TokenTable{}) {
  const int ctas = EPI == WS_EPI_GATED ? ws_ctas(N / 2, 8, K, false) : ws_ctas(N, 16, K, EPI == WS_EPI_ROPE);
  // (rows beyond a group a CTA: only the forms that are asked for them)
  const bool walk = EPI != WS_EPI_ROPE && (long long)ctas * (EPI == WS_EPI_GATED ? 8 : 16) < (EPI == WS_EPI_GATED ? N / 2 : N);
  if constexpr (EPI == WS_EPI_GATED || EPI == WS_EPI_STORE) {
    if (N > WS_ONE_GROUP_ROWS && ws_side_by_side(M, N, K)) {
      const int n = (N + 16 * WS_SIDE - 1) / (16 * WS_SIDE);
      if (norm.ssq_in != nullptr)
        launch_kernel(ws_kernel<NT, EPI, OUT, true, WS_ROWS>(), n, WS_WARPS * 32, 0, stream, x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, 1);
      else
        launch_kernel(ws_kernel<NT, EPI, OUT, false, WS_ROWS>(), n, WS_WARPS * 32, 0, stream, x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, 1);
      return launch_status("linear_ws");
    }
  }
  if (norm.ssq_in != nullptr) {
    if constexpr (EPI != WS_EPI_ROPE) {
      if (walk) {
        launch_kernel(ws_kernel<NT, EPI, OUT, true, WS_WALK>(), ctas, WS_WARPS * 32, 0, stream, x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, 1);
        return launch_status("linear_ws");
      }
    }
    launch_kernel(ws_kernel<NT, EPI, OUT, true, WS_ONE>(), ctas, WS_WARPS * 32, 0, stream, x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, 1);
    return launch_status("linear_ws");
  }
  if constexpr (EPI != WS_EPI_ROPE) {
    if (walk) {
      launch_kernel(ws_kernel<NT, EPI, OUT, false, WS_WALK>(), ctas, WS_WARPS * 32, 0, stream, x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, 1);
      return launch_status("linear_ws");
    }
  }
  if constexpr (EPI <= WS_EPI_RESID) {
    const int slices = ws_slices(ctas, K, M, EPI == WS_EPI_RESID);
    if (slices > 1) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(ctas * slices);
      cfg.blockDim = dim3(WS_WARPS * 32);
      cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = slices;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = pdl_enabled() ? 2 : 1;
      cudaLaunchKernelEx(&cfg, ws_kernel<NT, EPI, OUT, false, WS_SLICED>(), x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, slices);
      return launch_status("linear_ws");
    }
  }
  launch_kernel(ws_kernel<NT, EPI, OUT, false, WS_ONE>(), ctas, WS_WARPS * 32, 0, stream, x, W, bias, (OUT*)out, residual, M, N, K, rope, norm, act, token, 1);
  return launch_status("linear_ws");
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_linear_ws_supports(int M, int N, int K) {
  return M >= 1 && M <= 32 && N >= 16 && K >= 32 && K % 32 == 0;
}

// slices of K that the CTAs of a cluster share at more than 8 tokens (no norm owed on the input)
SLLM_EXPORT int sllm_linear_ws_slices(int N, int K) { return ws_slices(ws_ctas(N, 16, K, false), K, 32, false); }
// whether a product of many rows takes the form with groups side by side
SLLM_EXPORT int sllm_linear_ws_side_by_side(int M, int N, int K) { return ws_side_by_side(M, N, K); }

// CTAs a launch for N output columns over a reduction of K uses: the rows of the table of partial sums of squares
// that the residual epilogue writes when it is asked for the next norm's input (see WsNorm).
SLLM_EXPORT int sllm_linear_ws_parts(int N, int K) { return ws_ctas(N, 16, K, false); }

static bool ws_norm_in(WsNorm& n, const float* ssq_in, int parts_in, float eps_in, int width_in, int M) {
  if (ssq_in == nullptr) return true;
  if (parts_in < 1 || parts_in > ws_ssq_max(M <= 16 ? 2 : 4) || width_in < 1 || ((uintptr_t)ssq_in & 15) != 0) return false;
  n.ssq_in = ssq_in; n.parts_in = parts_in; n.eps_in = eps_in; n.inv_width_in = 1.0f / (float)width_in;
  return true;
}

// residual != null: residual[M, N] (float32) += x W^T (+ bias) and `out` is ignored;
// else out[M, N] = x W^T (+ bias) in out_dtype.
// ssq_in != null: x is bfloat16(stream * gain) of a norm still owed and ssq_in [M][parts_in rounded up to 4] holds partial sums of
// squares of the stream's rows (width_in wide): each row of the product is multiplied by rsqrt(sum / width_in + eps_in).
// gain != null (residual epilogue only): also write xg_out [M, N] = bfloat16(residual * gain) and
// ssq_out [M][sllm_linear_ws_parts(N, K) rounded up to 4], the next norm's input in the same form.
// act: what the plain result passes before its store (SLLM_ACT_*; SLLM_ACT_TOKEN with the bfloat16 table of the tokens).
SLLM_EXPORT int sllm_linear_ws(const void* x, const void* W, const float* bias, void* out, int out_dtype, float* residual,
                               int M, int N, int K, const float* ssq_in, int parts_in, float eps_in, int width_in,
                               const float* gain, void* xg_out, float* ssq_out, int act, const void* token_table, const int* token_ids,
                               int token_off, int token_ld, int token_rows, cudaStream_t stream) {
  SLLM_REQUIRE(act == SLLM_ACT_NONE || ((act == SLLM_ACT_RELU2 || act == SLLM_ACT_GELU || act == SLLM_ACT_TOKEN) && residual == nullptr),
               "linear_ws: activation %d (0 none, 1 relu squared, 2 gelu times the tokens' table), not with a residual", act);
  SLLM_REQUIRE(act != SLLM_ACT_TOKEN || (token_table && token_ids && token_rows > 0 && token_off >= 0 && token_off + N <= token_ld),
               "linear_ws: the tokens' table has rows of %d, columns %d..%d are wanted", token_ld, token_off, token_off + N);
  TokenTable tt;
  tt.table = token_table; tt.ids = token_ids; tt.off = token_off; tt.ld = token_ld; tt.V = token_rows;
  SLLM_REQUIRE(sllm_linear_ws_supports(M, N, K), "linear_ws: sizes M=%d N=%d K=%d (needs M<=32, K%%32==0)", M, N, K);
  SLLM_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)W & 15) == 0, "linear_ws: operands must be 16-byte aligned");
  SLLM_REQUIRE(residual != nullptr || out != nullptr, "linear_ws: no destination");
  WsNorm nm;
  SLLM_REQUIRE(ws_norm_in(nm, ssq_in, parts_in, eps_in, width_in, M), "linear_ws: a table of %d partial sums (at most %d) over width %d",
               parts_in, ws_ssq_max(M <= 16 ? 2 : 4), width_in);
  if (gain != nullptr) {
    SLLM_REQUIRE(residual != nullptr && xg_out != nullptr && ssq_out != nullptr, "linear_ws: the next norm's input needs the residual epilogue and both destinations");
    nm.gain = gain; nm.xg_out = (__nv_bfloat16*)xg_out; nm.ssq_out = ssq_out;
  }
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)W;
#define GO(NT_)                                                                                                        \
  if (residual) return launch_ws<NT_, WS_EPI_RESID, float>(xb, wb, bias, nullptr, residual, M, N, K, stream, WsRope{}, nm);          \
  if (out_dtype == SLLM_BF16) return launch_ws<NT_, WS_EPI_STORE, __nv_bfloat16>(xb, wb, bias, out, nullptr, M, N, K, stream, WsRope{}, nm, act, tt); \
  return launch_ws<NT_, WS_EPI_STORE, float>(xb, wb, bias, out, nullptr, M, N, K, stream, WsRope{}, nm, act, tt);
  if (M <= 8) { GO(1) }
  if (M <= 16) { GO(2) }
  GO(4)
#undef GO
}

// out[M, N/2] = act(gate) * up (bfloat16) of the gate|up matrix W [N, K] whose rows (and biases) alternate in blocks of 8; gelu: the tanh form of GELU
// in place of SiLU.  ssq_in: as for sllm_linear_ws.
SLLM_EXPORT int sllm_linear_ws_gated(const void* x, const void* W, const float* bias, void* out, int gelu, int M, int N, int K,
                                     const float* ssq_in, int parts_in, float eps_in, int width_in, cudaStream_t stream) {
  SLLM_REQUIRE(sllm_linear_ws_supports(M, N, K) && M <= 16 && N % 16 == 0, "linear_ws_gated: sizes M=%d N=%d K=%d (needs M<=16, N%%16==0, K%%32==0)", M, N, K);
  SLLM_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)W & 15) == 0 && out != nullptr, "linear_ws_gated: operands must be 16-byte aligned");
  WsNorm nm;
  SLLM_REQUIRE(ws_norm_in(nm, ssq_in, parts_in, eps_in, width_in, M), "linear_ws_gated: a table of %d partial sums (at most %d) over width %d",
               parts_in, ws_ssq_max(M <= 16 ? 2 : 4), width_in);
  const __nv_bfloat16 *xb = (const __nv_bfloat16*)x, *wb = (const __nv_bfloat16*)W;
  const int act = gelu ? WS_GATE_GELU : WS_GATE_SILU;
  if (M <= 8) return launch_ws<1, WS_EPI_GATED, __nv_bfloat16>(xb, wb, bias, out, nullptr, M, N, K, stream, WsRope{}, nm, act);
  return launch_ws<2, WS_EPI_GATED, __nv_bfloat16>(xb, wb, bias, out, nullptr, M, N, K, stream, WsRope{}, nm, act);
}

SLLM_EXPORT int sllm_linear_ws_rope_supports(int M, int N, int K, int nq, int nkv, int hd, int rot) {
  return sllm_linear_ws_supports(M, N, K) && nq > 0 && nkv > 0 && hd >= 16 && hd % 16 == 0 && N == (nq + 2 * nkv) * hd &&
         (rot == 0 || rot == hd);
}

// The fused q|k|v product of an attention layer with its bias, rotary encoding and cache write:
// x [M, K] and W [(nq + 2 nkv) * hd, K] bfloat16; table null or rot == 0: no rotation, else rot == hd and
// table [max_pos][2][hd/2] float32; slot_mapping null: keys and values are not written.  ssq_in: as for sllm_linear_ws.
// W and bias are read before the wait on the stream's earlier kernels, positions and slot_mapping behind it.
SLLM_EXPORT int sllm_linear_ws_rope(const void* x, const void* W, const float* bias, int M, int N, int K, const int* positions,
                                    const float* table, int rot, int max_pos, int nq, int nkv, int hd, const int* slot_mapping,
                                    int page_size, int num_pages, void* k_cache, void* v_cache, void* q_out,
                                    const float* ssq_in, int parts_in, float eps_in, int width_in, cudaStream_t stream) {
  SLLM_REQUIRE(sllm_linear_ws_rope_supports(M, N, K, nq, nkv, hd, rot),
               "linear_ws_rope: sizes M=%d N=%d K=%d nq=%d nkv=%d hd=%d rot=%d", M, N, K, nq, nkv, hd, rot);
  SLLM_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)W & 15) == 0, "linear_ws_rope: operands must be 16-byte aligned");
  SLLM_REQUIRE(q_out != nullptr && (rot == 0 || (table != nullptr && positions != nullptr && max_pos > 0)),
               "linear_ws_rope: destination or rotary table missing");
  SLLM_REQUIRE(slot_mapping == nullptr || (k_cache && v_cache && page_size > 0 && num_pages > 0), "linear_ws_rope: cache arguments missing");
  WsNorm nm;
  SLLM_REQUIRE(ws_norm_in(nm, ssq_in, parts_in, eps_in, width_in, M), "linear_ws_rope: a table of %d partial sums (at most %d) over width %d",
               parts_in, ws_ssq_max(M <= 16 ? 2 : 4), width_in);
  WsRope r;
  r.positions = positions; r.table = rot > 0 ? table : nullptr; r.slot_mapping = slot_mapping;
  r.k_cache = (__nv_bfloat16*)k_cache; r.v_cache = (__nv_bfloat16*)v_cache; r.q_out = (__nv_bfloat16*)q_out;
  r.max_pos = max_pos; r.nq = nq; r.nkv = nkv; r.hd = hd; r.page_size = page_size; r.num_pages = num_pages;
  const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
  const __nv_bfloat16* wb = (const __nv_bfloat16*)W;
  if (M <= 8) return launch_ws<1, WS_EPI_ROPE, __nv_bfloat16>(xb, wb, bias, nullptr, nullptr, M, N, K, stream, r, nm);
  if (M <= 16) return launch_ws<2, WS_EPI_ROPE, __nv_bfloat16>(xb, wb, bias, nullptr, nullptr, M, N, K, stream, r, nm);
  return launch_ws<4, WS_EPI_ROPE, __nv_bfloat16>(xb, wb, bias, nullptr, nullptr, M, N, K, stream, r, nm);
}
