// A mixture of experts over prompt portions with the tokens sorted by expert, so that each expert multiplies its own tokens alone (the dense form, every
// expert over every token with zeros for those not chosen, does experts / top times that work):
//
//   moe_assign   from the router's (index) lists [T, top]: every (token, choice) gets a row of a buffer in which an expert's rows are neighbours and
//                start on a multiple of 256 (the rows of a tile of gemm_pair.cu): its place, the expert of every row tile (-1: nobody's), and the token
//                of every row;
//   moe_gather   the tokens' normed rows to those places;
//   moe_combine  out[t] (+)= sum over the choices of weight * the row at its place, in the choices' order, plus one more row per token (the shared
//                expert's), weighted where it has a gate.
//
// Rows that pad an expert's are never written and never read: a row of a product depends on no other row.
#include "common.cuh"

namespace sllm {

constexpr int MG_TILE = 256, MG_MAX_EXPERTS = 256, MG_THREADS = 1024, MG_AHEAD = 4 /* choices whose loads are in flight */;

// one block; the order of an expert's rows is whatever the counters give (no result depends on it)
__global__ void __launch_bounds__(MG_THREADS)
moe_assign_kernel(const int* idx, int n, int top, int E, int tiles, int* __restrict__ place, int* __restrict__ tile_expert, int* __restrict__ row_token) {
  __shared__ int count[MG_MAX_EXPERTS], start[MG_MAX_EXPERTS + 1];
  const int tid = threadIdx.x;
  pdl_wait();
  for (int e = tid; e < E; e += MG_THREADS) count[e] = 0;
  for (int r = tid; r < tiles * MG_TILE; r += MG_THREADS) row_token[r] = -1;
  __syncthreads();
  for (int i0 = 0; i0 < n; i0 += MG_AHEAD * MG_THREADS) {       // (whole warps: the lanes of one expert count together)
    int chosen[MG_AHEAD];
#pragma unroll
    for (int u = 0; u < MG_AHEAD; ++u) chosen[u] = i0 + u * MG_THREADS + tid < n ? idx[i0 + u * MG_THREADS + tid] : -1;
#pragma unroll
    for (int u = 0; u < MG_AHEAD; ++u) {
      const int i = i0 + u * MG_THREADS + tid, e = chosen[u];
      const unsigned peers = __match_any_sync(0xffffffffu, e);
      const int leader = __ffs(peers) - 1, lane = tid & 31;
      int base = 0;
      if (e >= 0 && lane == leader) base = atomicAdd(&count[e], __popc(peers));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (i < n) place[i] = base + __popc(peers & ((1u << lane) - 1));
    }
  }
  __syncthreads();
  if (tid == 0) {
    int at = 0;
    for (int e = 0; e < E; ++e) {
      start[e] = at;
      at += (count[e] + MG_TILE - 1) / MG_TILE;
    }
    start[E] = at;
  }
  __syncthreads();
  for (int t = tid; t < tiles; t += MG_THREADS) {
    int e = -1;
    if (t < start[E])
      for (e = 0; t >= start[e + 1]; ++e) {}
    tile_expert[t] = e;
  }
  for (int i0 = tid; i0 < n; i0 += MG_AHEAD * MG_THREADS) {        // (a thread's own entries)
    int e[MG_AHEAD], at[MG_AHEAD];
#pragma unroll
    for (int u = 0; u < MG_AHEAD; ++u) {
      const int i = i0 + u * MG_THREADS;
      e[u] = i < n ? idx[i] : 0;
      at[u] = i < n ? place[i] : 0;
    }
#pragma unroll
    for (int u = 0; u < MG_AHEAD; ++u) {
      const int i = i0 + u * MG_THREADS, r = start[e[u]] * MG_TILE + at[u];
      if (i >= n) break;
      place[i] = r;
      row_token[r] = i / top;
    }
  }
}

// a warp per row, 16 bytes a lane
__global__ void __launch_bounds__(256)
moe_gather_kernel(const uint4* x, const int* row_token, uint4* __restrict__ out, int rows, int pieces) {
  pdl_wait();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const int t = row_token[row];
  if (t < 0) return;
  for (int c0 = lane; c0 < pieces; c0 += 256) {
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (c0 + 32 * k < pieces) v[k] = x[(size_t)t * pieces + c0 + 32 * k];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (c0 + 32 * k < pieces) out[(size_t)row * pieces + c0 + 32 * k] = v[k];
  }
}

// a block per token, four columns a thread
__global__ void __launch_bounds__(256)
moe_combine_kernel(const float* y, const int* place, const float* wts, int top, const float* shared,
                   const float* shared_w, int ld_w, float* out, int add, int W) {
  pdl_wait();
  const int t = blockIdx.x;
  const float sw = shared_w != nullptr ? shared_w[(size_t)t * ld_w] : 1.0f;
  for (int c = threadIdx.x * 4; c < W; c += 1024) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < top; ++j) {
      const float w = wts[(size_t)t * top + j];
      if (w == 0.f) continue;                        // not chosen after all
      const float4 r = *reinterpret_cast<const float4*>(y + (size_t)place[(size_t)t * top + j] * W + c);
      v.x = fmaf(w, r.x, v.x); v.y = fmaf(w, r.y, v.y); v.z = fmaf(w, r.z, v.z); v.w = fmaf(w, r.w, v.w);
    }
    if (shared != nullptr) {
      const float4 r = *reinterpret_cast<const float4*>(shared + (size_t)t * W + c);
      v.x = fmaf(sw, r.x, v.x); v.y = fmaf(sw, r.y, v.y); v.z = fmaf(sw, r.z, v.z); v.w = fmaf(sw, r.w, v.w);
    }
    float4* o = reinterpret_cast<float4*>(out + (size_t)t * W + c);
    if (add) {
      const float4 r = *o;
      v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w;
    }
    *o = v;
  }
}

}  // namespace sllm

using namespace sllm;

// idx [T, top] (experts, 0 .. E - 1): place [T, top], tile_expert [tiles], row_token [tiles * 256]; tiles: at least the sum over experts of their tokens'
// tiles (T * top / 256 + E are always enough)
SLLM_EXPORT int sllm_moe_assign(const int* idx, int T, int top, int E, int tiles, int* place, int* tile_expert, int* row_token, cudaStream_t stream) {
  SLLM_REQUIRE(T >= 0 && top >= 1 && E >= 1 && E <= MG_MAX_EXPERTS && (long long)T * top <= (1 << 30), "moe_assign: bad sizes T=%d top=%d E=%d (at most %d experts)", T, top, E, MG_MAX_EXPERTS);
  SLLM_REQUIRE(tiles >= T * top / MG_TILE + E, "moe_assign: %d row tiles for %d x %d choices among %d experts", tiles, T, top, E);
  if (T == 0) return SLLM_OK;
  launch_kernel(moe_assign_kernel, 1, MG_THREADS, 0, stream, idx, T * top, top, E, tiles, place, tile_expert, row_token);
  return launch_status("moe_assign");
}

// out[r] = x[row_token[r]] for rows with a token; rows of `row_bytes` bytes, a multiple of 16
SLLM_EXPORT int sllm_moe_gather(const void* x, const int* row_token, void* out, int rows, int row_bytes, cudaStream_t stream) {
  SLLM_REQUIRE(rows >= 0 && row_bytes > 0 && row_bytes % 16 == 0 && (((uintptr_t)x | (uintptr_t)out) & 15) == 0, "moe_gather: rows of %d bytes (whole 16-byte pieces)", row_bytes);
  if (rows == 0) return SLLM_OK;
  launch_kernel(moe_gather_kernel, (rows + 7) / 8, 256, 0, stream, (const uint4*)x, row_token, (uint4*)out, rows, row_bytes / 16);
  return launch_status("moe_gather");
}

// out[T, W] (+= if add) sum_j wts[t, j] y[place[t, j]] + shared_w[t * ld_w] shared[t] (shared may be null, shared_w too: 1)
SLLM_EXPORT int sllm_moe_combine(const float* y, const int* place, const float* wts, int T, int top, const float* shared, const float* shared_w, int ld_w,
                                 float* out, int add, int W, cudaStream_t stream) {
  SLLM_REQUIRE(T >= 0 && top >= 1 && W > 0 && W % 4 == 0 && (((uintptr_t)y | (uintptr_t)shared | (uintptr_t)out) & 15) == 0, "moe_combine: bad sizes T=%d top=%d W=%d", T, top, W);
  if (T == 0) return SLLM_OK;
  launch_kernel(moe_combine_kernel, T, 256, 0, stream, y, place, wts, top, shared, shared_w, ld_w, out, add, W);
  return launch_status("moe_combine");
}
