// Attention over the paged cache on the CUDA cores, all arithmetic in float32:
// the kernel of the float32 path, and the one that takes head sizes and dtypes the
// tensor-core kernel refuses.  One block per (token, query head): prompt portions and
// single decoded tokens are the same work, so a position's result cannot depend on
// how the batch was cut.
//
//   s_j = (q . k_j) * scale for keys j <= pos (and j > pos - window; and, with `chunk`, j in pos's own block of
//   `chunk` positions counted from 0), softmax with the
//   maximum subtracted, o = sum p_j v_j   (ref/qwen3_5.py:373-390; one row:
//   ref/incremental.py:75-87; kernels/cuda/kernels.cu:957-1025 for one CTA per head).
//   Query head h reads kv head h / (nq / nkv) (ref/standard.py:65-68).
//   With `sink` (one number per query head) the softmax's denominator also holds exp(sink_h).
//   With `softcap` > 0 a score becomes softcap tanh(score / softcap) before the softmax; with `gate` (logits, one per token
//   and query head) the head's output is multiplied by the gate's sigmoid.  With `rel` [nkv, rel_n, nq / nkv] the score then takes in
//   a bias by the distance from key to query (distances beyond the table: its last row) and the query head.
//
// Two ways through the keys.
//   A key a lane (heads of up to 128 channels, from `simt_short` keys on): keys go by aligned blocks of 32 positions, block b to warp (b - first block) mod
//   the block's warps.  In the scores a lane walks its own key's row (16 bytes a load where rows allow it) against the query in shared memory, so the 32
//   dot products of a block run side by side and none needs a sum over lanes; one online-softmax update a block; in the
//   weighted sum a lane is a channel and the block's 32 value rows are independent loads.  What bounds it is the latency of those loads: with
//   a key a step and a warp (every key's page, row and sum over lanes in one chain) a decode step of 3 requests at 190 keys took
//   51 us, now 11; one token at 4,000 keys 1,020, now 70; a portion of 537 tokens 504, now 189 (14 heads of 64, 2 kv heads, float32).
//   Four keys a warp (wider heads, and few keys): aligned groups of four positions, a lane four channels at a time, four sums over lanes side by side, one
//   online-softmax update.  A lane's own row is no longer a few lines of cache where heads are wide, and few keys leave most
//   warps without a block of 32.
// The warps' partial results are merged in warp order.  The order of every sum depends on the position alone.
#include <math.h>
#include <stdio.h>

#include <type_traits>

#include "common.cuh"

namespace sllm {

constexpr int ATT_WARPS = 8;
constexpr int ATT_MAX_HD = 256;        // (instances of 64 and 128 channels too: the accumulators are registers)
// keys below which four a warp are taken at once (128 keys of a window, 1,500 tokens, us, four a warp / a key a lane: 64 bfloat16 channels 206 / 153, 128 205 / 209, 128 float32 200 / 275)
__host__ __device__ constexpr int simt_short(int max_hd) { return max_hd <= 64 ? 96 : 160; }
constexpr int ATT_WIDE_HD = 640;       // a second instance for wider heads (a cached latent beside a rotated key part)

// d consecutive channels of a row against the query in shared memory; VEC: 16 bytes a load (rows of whole 16-byte pieces)
template <typename T, bool VEC>
__device__ __forceinline__ float simt_dot(const T* row, const float* qs, int d) {
  float dot[4] = {0.f, 0.f, 0.f, 0.f};               // four chains
  if (VEC) {
    constexpr int P = 16 / sizeof(T);
#pragma unroll 16
    for (int i = 0; i < d; i += P) {
      const uint4 raw = *reinterpret_cast<const uint4*>(row + i);
      const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int e = 0; e < P; ++e) dot[e % 4] = fmaf(qs[i + e], to_f32(v[e]), dot[e % 4]);
    }
  } else {
    for (int i = 0; i < d; i += 4)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (i + e < d) dot[e] = fmaf(qs[i + e], to_f32(row[i + e]), dot[e]);
  }
  return (dot[0] + dot[1]) + (dot[2] + dot[3]);
}

// four consecutive channels from d on, zeros beyond hd
template <typename T, bool VEC>
__device__ __forceinline__ float4 simt_load4(const T* row, int d, int hd) {
  if (VEC) {                               // (hd is a multiple of 4 then)
    if (d >= hd) return make_float4(0.f, 0.f, 0.f, 0.f);
    if constexpr (sizeof(T) == 4) {
      return *reinterpret_cast<const float4*>(row + d);
    } else {
      const uint2 raw = *reinterpret_cast<const uint2*>(row + d);
      const T* v = reinterpret_cast<const T*>(&raw);
      return make_float4(to_f32(v[0]), to_f32(v[1]), to_f32(v[2]), to_f32(v[3]));
    }
  }
  return make_float4(d < hd ? to_f32(row[d]) : 0.f, d + 1 < hd ? to_f32(row[d + 1]) : 0.f, d + 2 < hd ? to_f32(row[d + 2]) : 0.f,
                     d + 3 < hd ? to_f32(row[d + 3]) : 0.f);
}

// The keys lo .. pos of one query head, four a warp: the warp's maximum m, its sum l (known to all lanes) and its weighted sum of values in acc_s.
template <typename TC, int MAX_HD, bool VEC>
__device__ __forceinline__ void simt_groups(const TC* k_cache, const TC* v_cache, const int* bt, const float* qs,
                                            float* acc_s, int lo, int pos, int kvh, int nkv, int G, int g, int hd, int page_size, float scale,
                                            float softcap, const float* __restrict__ rel, int rel_n, float& m, float& l) {
  constexpr int NC = (MAX_HD + 127) / 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float4 acc[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int j0 = lo / 4 * 4 + warp * 4; j0 <= pos; j0 += ATT_WARPS * 4) {
    const int j = j0 + (lane & 3);
    const int page = j >= lo && j <= pos ? bt[j / page_size] : -1;         // a page that was given back is never dereferenced
    const unsigned counts = __ballot_sync(0xffffffffu, page >= 0) & 15u;   // one answer for all lanes
    if (counts == 0) continue;
    const long long mine = page < 0 ? 0 : (((long long)page * nkv + kvh) * page_size + (j % page_size)) * hd;
    size_t row[4];
    float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 4; ++u) row[u] = (size_t)__shfl_sync(0xffffffffu, mine, u);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int d = 4 * (lane + 32 * i);
      if (d >= hd) break;
      const float4 q4 = *reinterpret_cast<const float4*>(qs + d);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (counts >> u & 1) {
          const float4 k4 = simt_load4<TC, VEC>(k_cache + row[u], d, hd);
          dot[u] = fmaf(q4.w, k4.w, fmaf(q4.z, k4.z, fmaf(q4.y, k4.y, fmaf(q4.x, k4.x, dot[u]))));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < 4; ++u) dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], o);
    float s[4], m_new = m;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s[u] = softcap > 0.f ? softcap * tanhf(dot[u] * scale / softcap) : dot[u] * scale;
      if (rel != nullptr && counts >> u & 1) s[u] += rel[((size_t)kvh * rel_n + min(pos - j0 - u, rel_n - 1)) * G + g];
      if (counts >> u & 1) m_new = fmaxf(m_new, s[u]);
    }
    const float corr = expf(m - m_new);              // exp(-inf) = 0 on the first group
    m = m_new;
    l *= corr;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s[u] = counts >> u & 1 ? expf(s[u] - m_new) : 0.f;
      l += s[u];
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      const int d = 4 * (lane + 32 * i);
      if (d >= hd) break;
      acc[i].x *= corr; acc[i].y *= corr; acc[i].z *= corr; acc[i].w *= corr;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (counts >> u & 1) {
          const float4 v4 = simt_load4<TC, VEC>(v_cache + row[u], d, hd);
          acc[i].x = fmaf(s[u], v4.x, acc[i].x);
          acc[i].y = fmaf(s[u], v4.y, acc[i].y);
          acc[i].z = fmaf(s[u], v4.z, acc[i].z);
          acc[i].w = fmaf(s[u], v4.w, acc[i].w);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    const int d = 4 * (lane + 32 * i);
    if (d < hd) *reinterpret_cast<float4*>(acc_s + d) = acc[i];            // (MAX_HD is a multiple of 4)
  }
}

template <typename TQ, typename TC, int ATT_MAX_HD, bool VEC>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_simt_kernel(const TQ* q, const TC* k_cache, const TC* v_cache,
                      const int* block_tables, int max_pages, const int* positions,
                      const int* seq_of_token, int nq, int nkv, int hd, int page_size, float scale,
                      int window, int chunk, const float* __restrict__ sink, float softcap, const float* gate, int gate_ld,
                      const float* __restrict__ rel, int rel_n, TQ* __restrict__ out) {
  __shared__ __align__(16) float qs[ATT_MAX_HD];
  __shared__ __align__(16) float acc_s[ATT_WARPS][ATT_MAX_HD];
  __shared__ float m_s[ATT_WARPS], l_s[ATT_WARPS];
  constexpr bool NARROW = ATT_MAX_HD <= 128;
  __shared__ float p_s[NARROW ? ATT_WARPS : 1][32];
  __shared__ size_t row_s[NARROW ? ATT_WARPS : 1][32];
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y;
  const int G = nq / nkv, kvh = h / G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int pos = positions[t];
  const int* bt = block_tables + (size_t)seq_of_token[t] * max_pages;
  int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  if (chunk > 0) lo = max(lo, pos / chunk * chunk);

  for (int d = threadIdx.x; d < ATT_MAX_HD; d += blockDim.x) qs[d] = d < hd ? to_f32(q[((size_t)t * nq + h) * hd + d]) : 0.f;
  __syncthreads();

  float m = -INFINITY, l = 0.f;
  if (!NARROW || pos - lo < simt_short(ATT_MAX_HD)) {
    simt_groups<TC, ATT_MAX_HD, VEC>(k_cache, v_cache, bt, qs, acc_s[warp], lo, pos, kvh, nkv, G, h % G, hd, page_size, scale, softcap, rel, rel_n, m, l);
  } else if constexpr (NARROW) {
    float acc[ATT_MAX_HD / 32];
#pragma unroll
    for (int i = 0; i < ATT_MAX_HD / 32; ++i) acc[i] = 0.f;
    // l: this lane's keys alone; added up over the lanes at the end
    for (int j0 = lo / 32 * 32 + warp * 32; j0 <= pos; j0 += ATT_WARPS * 32) {
      const int j = j0 + lane;
      const int page = j >= lo && j <= pos ? bt[j / page_size] : -1;         // a page that was given back is never dereferenced
      const size_t row = page < 0 ? 0 : (((size_t)page * nkv + kvh) * page_size + (j % page_size)) * hd;
      float s = -INFINITY;
      if (page >= 0) {
        const float dot = simt_dot<TC, VEC>(k_cache + row, qs, hd);
        s = softcap > 0.f ? softcap * tanhf(dot * scale / softcap) : dot * scale;
        if (rel != nullptr) s += rel[((size_t)kvh * rel_n + min(pos - j, rel_n - 1)) * G + h % G];
      }
      const unsigned counts = __ballot_sync(0xffffffffu, page >= 0);
      if (counts == 0) continue;
      const float m_new = fmaxf(m, warp_max(s));
      const float corr = expf(m - m_new);              // exp(-inf) = 0 on the first block
      const float p = page < 0 ? 0.f : expf(s - m_new);
      l = l * corr + p;
      m = m_new;
      p_s[warp][lane] = p;
      row_s[warp][lane] = row;                         // (a key that does not count: row 0 of the pages, times zero is not taken)
      __syncwarp();
#pragma unroll
      for (int i = 0; i < ATT_MAX_HD / 32; ++i) acc[i] *= corr;
      // eight value rows are loaded before the first is added, in the last block's keys too (its rows one behind the other were up to 31 misses in a chain: a decode step of 3
      // requests at 190 keys 10.9 us, so 5.8; a portion of 537 tokens 87, so 79; 14 heads of 64, 2 kv heads, float32); rows that do not count are not read
      auto rows = [&](auto whole) {
        constexpr bool ALL = decltype(whole)::value;
#pragma unroll
        for (int u0 = 0; u0 < 32; u0 += 8) {
          if (!ALL && (counts >> u0 & 255u) == 0) continue;
          float v[8][ATT_MAX_HD / 32];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const TC* vr = v_cache + row_s[warp][u0 + k];
#pragma unroll
            for (int i = 0; i < ATT_MAX_HD / 32; ++i) v[k][i] = (ALL || (counts >> (u0 + k) & 1u)) && lane + 32 * i < hd ? to_f32(vr[lane + 32 * i]) : 0.f;
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (!ALL && !(counts >> (u0 + k) & 1u)) continue;
            const float pu = p_s[warp][u0 + k];
#pragma unroll
            for (int i = 0; i < ATT_MAX_HD / 32; ++i) acc[i] = fmaf(pu, v[k][i], acc[i]);
          }
        }
      };
      if (counts == 0xffffffffu) rows(std::true_type{});
      else rows(std::false_type{});
      __syncwarp();
    }
    l = warp_sum(l);
#pragma unroll
    for (int i = 0; i < ATT_MAX_HD / 32; ++i) {
      const int d = lane + 32 * i;
      if (d < hd) acc_s[warp][d] = acc[i];
    }
  }
  if (lane == 0) { m_s[warp] = m; l_s[warp] = l; }
  __syncthreads();
  float mm = -INFINITY;
#pragma unroll
  for (int w = 0; w < ATT_WARPS; ++w) mm = fmaxf(mm, m_s[w]);
  float ll = 0.f;
  float f[ATT_WARPS];
#pragma unroll
  for (int w = 0; w < ATT_WARPS; ++w) {
    f[w] = l_s[w] > 0.f ? expf(m_s[w] - mm) : 0.f;
    ll += l_s[w] * f[w];
  }
  if (sink != nullptr) ll += expf(sink[h] - mm);       // a term of the denominator without key or value, not scaled
  float inv = ll > 0.f ? 1.0f / ll : 0.f;
  if (gate != nullptr) inv *= sigmoid_f32(gate[(size_t)t * gate_ld + h]);
  for (int d = threadIdx.x; d < hd; d += blockDim.x) {
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) o += acc_s[w][d] * f[w];
    out[((size_t)t * nq + h) * hd + d] = from_f32<TQ>(o * inv);
  }
}

template <typename T>
static int simt_launch(const T* q, const T* k_cache, const T* v_cache, const int* block_tables, int max_pages, const int* positions,
                       const int* seq_of_token, int num_tokens, int nq, int nkv, int hd, int page_size, float scale, int window, int chunk,
                       const float* sink, float softcap, const float* gate, int gate_ld, const float* rel, int rel_n, T* out, cudaStream_t stream) {
  const bool vec = hd * (int)sizeof(T) % 16 == 0 && ((reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) == 0;
  auto kernel = hd <= 64 ? (vec ? attention_simt_kernel<T, T, 64, true> : attention_simt_kernel<T, T, 64, false>)
              : hd <= 128 ? (vec ? attention_simt_kernel<T, T, 128, true> : attention_simt_kernel<T, T, 128, false>)
              : hd <= ATT_MAX_HD ? (vec ? attention_simt_kernel<T, T, ATT_MAX_HD, true> : attention_simt_kernel<T, T, ATT_MAX_HD, false>)
                                 : (vec ? attention_simt_kernel<T, T, ATT_WIDE_HD, true> : attention_simt_kernel<T, T, ATT_WIDE_HD, false>);
  launch_kernel(kernel, dim3(num_tokens, nq), ATT_WARPS * 32, 0, stream, q, k_cache, v_cache, block_tables, max_pages, positions, seq_of_token, nq,
                nkv, hd, page_size, scale, window, chunk, sink, softcap, gate, gate_ld, rel, rel_n, out);
  return launch_status("attention_simt");
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_attention_simt(const void* q, const void* k_cache, const void* v_cache, int dtype,
                                    const int* block_tables, int max_pages, const int* positions,
                                    const int* seq_of_token, int T, int nq, int nkv, int hd, int page_size,
                                    float scale, int window, int chunk, const float* sink, float softcap, const float* gate, int gate_ld,
                                    const float* rel, int rel_n, void* out, cudaStream_t stream) {
  SLLM_REQUIRE(T >= 0 && nq > 0 && nkv > 0 && nq % nkv == 0, "attention: bad head counts nq=%d nkv=%d", nq, nkv);
  SLLM_REQUIRE(hd > 0 && hd <= ATT_WIDE_HD, "attention: head_dim=%d is outside 1..%d", hd, ATT_WIDE_HD);
  SLLM_REQUIRE(page_size > 0 && max_pages > 0, "attention: bad page_size=%d max_pages=%d", page_size, max_pages);
  SLLM_REQUIRE(nq <= 65535, "attention: %d query heads exceed one launch", nq);
  SLLM_REQUIRE(rel == nullptr || rel_n >= 1, "attention: a bias by distance needs its table");
  if (T == 0) return SLLM_OK;
  SLLM_REQUIRE(dtype == SLLM_F32 || dtype == SLLM_BF16, "attention: unknown dtype %d", dtype);
  if (dtype == SLLM_F32)
    return simt_launch((const float*)q, (const float*)k_cache, (const float*)v_cache, block_tables, max_pages, positions, seq_of_token, T, nq, nkv,
                       hd, page_size, scale, window, chunk, sink, softcap, gate, gate_ld, rel, rel_n, (float*)out, stream);
  return simt_launch((const __nv_bfloat16*)q, (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache, block_tables, max_pages, positions,
                     seq_of_token, T, nq, nkv, hd, page_size, scale, window, chunk, sink, softcap, gate, gate_ld, rel, rel_n, (__nv_bfloat16*)out,
                     stream);
}
