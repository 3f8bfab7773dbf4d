// Linear attention with a decay per key channel (or one fixed decay per head) over prompt portions, a chunk of 64 tokens at a time:
//
//   S_t = diag(d_t) S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t
//
// in the three forms that delta_rule.cu walks token by token (its modes 2, 3, 4; the walk keeps single tokens and short
// portions).  A walk is one chain of dependent sums per token, on an eighth of the SMs' warp slots for one prompt; a chunk's part of
// the recurrence is small matrix products that run side by side over chunks and heads.  With F_t the product of d over the
// chunk's tokens up to and including t (per channel), n tokens, and the state S the chunk meets:
//
//   o_t = (q_t F_t)^T S + sum_(s <= t) A_ts v_s,   A_ts = sum_i q_ti k_si prod_(s < r <= t) d_ri
//   S'  = diag(F_n) S + sum_s (k_s prod_(s < r <= n) d_r) v_s^T
//
//   1. gated_state  per (chunk, head): what the chunk adds to a state, and F_n, to scratch;
//   2. gated_scan   per (request, head, element): from the request's state slot through its chunks in order; scratch then holds
//                   the state each chunk meets, the slot the portion's last state;
//   3. gated_out    per (chunk, head): the two terms of o.
//
// No decay is ever divided by and no logarithm is summed: every factor is a running product of decays, at most one, so a decay may be as
// small as zero.  Inside a run of 16 tokens A is walked, a lane a key: its product over the decays grows with the query's place.  Between
// runs the key is carried to its run's end and the query from its run's start, and what lies between is multiplied into the query
// as it turns to earlier runs (a warp's 16 queries are the warp's own).  All arithmetic is float32 on the CUDA cores; the products
// are laid out as in retention.cu: a warp owns 16 tokens and all columns.
#include <math.h>

#include "chunked.cuh"

namespace sllm {

constexpr int GC_GATED = 2, GC_FIXED = 3, GC_FORGET = 4;       // delta_rule.cu's modes

struct GatedChunkParams {
  const float* proj;           // [T, ld]
  int ld, off_q, off_k, off_v; // GC_FORGET: the gate's logits at off_k
  const float* z;              // GC_GATED: [T, H*dk] decay logits
  const float* a;              // GC_FIXED: [H] decays; GC_FORGET: [H*dk] lower bounds
  const float* bias;           // GC_FORGET: [H*dk]
  float q_scale, inv_tau;
  float* state;                // [slots, H, dk, dv]
  const int* state_slots;      // [S]
  const int* chunk_t0;         // [chunks] first token (row of proj)
  const int* chunk_n;          // [chunks] tokens, 1 .. 64
  const int* run_seq;          // [runs] a request ...
  const int* run_first;        // [runs] ... its first chunk ...
  const int* run_count;        // [runs] ... and how many it has
  float* scratch;              // [chunks, H, dk, dv]
  float* keeps;                // [chunks, H, dk]: F_n
  float* out;                  // [T, H*dv]
  int H, dk, dv;
  int vec_v;                   // values lie in whole 16-byte pieces
};

// the key and the decay of one channel from what the product holds there (and the decay logit), as the walk's loader makes them
template <int MODE>
__device__ __forceinline__ void gc_key(float x, float z, float a, float bias, float inv_tau, float& k, float& d) {
  if (MODE == GC_FORGET) {
    d = a + (1.0f - a) * sigmoid_f32(x + bias);
    k = 1.0f - d;
  } else if (MODE == GC_FIXED) {
    k = x * sigmoid_f32(x);
    d = a;
  } else {
    k = x;
    d = expf((fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * inv_tau);
  }
}

// grid (chunks, H), 2 DK threads
template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(2 * DK) gated_state_kernel(const GatedChunkParams p) {
  extern __shared__ __align__(16) float gc_sm[];
  float* ks = gc_sm;                   // [RC][DK]
  float* vs = ks + RC * DK;            // [RC][DV]
  float* tail = vs + RC * DV;          // [DK] the second half's product
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int t0 = p.chunk_t0[chunk], n = p.chunk_n[chunk];
  load_block<RC, DV, DV>(vs, p.proj + (size_t)t0 * p.ld + p.off_v + h * p.dv, p.ld, n, p.dv, p.vec_v != 0);
  if (MODE == GC_FIXED) {              // the values pass silu too
    asm volatile("cp.async.wait_group 0;\n" ::);
    for (int e = threadIdx.x; e < RC * DV; e += 2 * DK) {
      // (a thread's own copies in the vector form: four neighbours each)
      if (!p.vec_v) vs[e] *= sigmoid_f32(vs[e]);
    }
    if (p.vec_v)
      for (int e = threadIdx.x; e < RC * (DV / 4); e += 2 * DK)
#pragma unroll
        for (int c = 0; c < 4; ++c) vs[4 * e + c] *= sigmoid_f32(vs[4 * e + c]);
  }
  // a thread a channel and half of the tokens, from the last to the first: the key times the decays behind it
  const int i = threadIdx.x % DK, half = threadIdx.x / DK;
  const bool in = i < p.dk;
  const float a = !in ? 0.f : MODE == GC_FIXED ? p.a[h] : MODE == GC_FORGET ? p.a[h * p.dk + i] : 0.f;
  const float bias = MODE == GC_FORGET && in ? p.bias[h * p.dk + i] : 0.f;
  const float* kp = p.proj + (size_t)t0 * p.ld + p.off_k + h * p.dk + i;
  const float* zp = MODE == GC_GATED ? p.z + (size_t)t0 * p.H * p.dk + h * p.dk + i : nullptr;
  float behind = 1.f;
#pragma unroll
  for (int b = RC / 2 - 8; b >= 0; b -= 8) {
    float x[8], z[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int t = half * (RC / 2) + b + q;
      const bool ok = in && t < n;
      x[q] = ok ? load_now(kp + (size_t)t * p.ld) : 0.f;
      z[q] = MODE == GC_GATED && ok ? load_now(zp + (size_t)t * p.H * p.dk) : 0.f;
    }
#pragma unroll
    for (int q = 7; q >= 0; --q) {
      const int t = half * (RC / 2) + b + q;
      float k, d;
      gc_key<MODE>(x[q], z[q], a, bias, p.inv_tau, k, d);
      const bool ok = in && t < n;
      ks[t * DK + i] = ok ? k * behind : 0.f;
      if (ok) behind *= d;
    }
  }
  if (half) tail[i] = behind;
  __syncthreads();
  if (!half) {
    const float f = tail[i];
#pragma unroll 8
    for (int t = 0; t < RC / 2; ++t) ks[t * DK + i] *= f;
    if (in) p.keeps[((size_t)chunk * p.H + h) * p.dk + i] = behind * f;
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  constexpr int TN = DV / 16;
  const int row = 16 * (threadIdx.x >> 5) + 8 * ((threadIdx.x >> 4) & 1), col = 4 * (threadIdx.x & 15);
  float acc[8][TN];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < TN; ++c) acc[r][c] = 0.f;
#pragma unroll 2
  for (int s = 0; s < n; ++s) {
    const float4 a0 = *reinterpret_cast<const float4*>(ks + s * DK + row), a1 = *reinterpret_cast<const float4*>(ks + s * DK + row + 4);
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
    for (int g = 0; g < TN / 4; ++g) {
      const float4 b = *reinterpret_cast<const float4*>(vs + s * DV + col + 64 * g);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        acc[r][4 * g] = fmaf(av[r], b.x, acc[r][4 * g]);
        acc[r][4 * g + 1] = fmaf(av[r], b.y, acc[r][4 * g + 1]);
        acc[r][4 * g + 2] = fmaf(av[r], b.z, acc[r][4 * g + 2]);
        acc[r][4 * g + 3] = fmaf(av[r], b.w, acc[r][4 * g + 3]);
      }
    }
  }
  pdl_launch_dependents();
  float* out = p.scratch + ((size_t)chunk * p.H + h) * p.dk * p.dv;
  const bool vec = p.dv % 4 == 0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int j0 = row + r;
    if (j0 >= p.dk) break;
#pragma unroll
    for (int g = 0; g < TN / 4; ++g) {
      const int j = col + 64 * g;
      if (vec && j < p.dv) {
        *reinterpret_cast<float4*>(out + (size_t)j0 * p.dv + j) = make_float4(acc[r][4 * g], acc[r][4 * g + 1], acc[r][4 * g + 2], acc[r][4 * g + 3]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (j + c < p.dv) out[(size_t)j0 * p.dv + j + c] = acc[r][4 * g + c];
      }
    }
  }
}

// grid (ceil(dk dv / 256), H, runs): an element of a state a thread, through the request's chunks in order
__global__ void __launch_bounds__(RC_SCAN_THREADS) gated_scan_kernel(const GatedChunkParams p) {
  pdl_wait();
  const int h = blockIdx.y, run = blockIdx.z, size = p.dk * p.dv;
  const int e = blockIdx.x * RC_SCAN_THREADS + threadIdx.x;
  const int first = p.run_first[run], count = p.run_count[run];
  if (e < size) {
    float* slot = p.state + ((size_t)p.state_slots[p.run_seq[run]] * p.H + h) * size + e;
    float* sc = p.scratch + ((size_t)first * p.H + h) * size + e;
    const float* keep = p.keeps + ((size_t)first * p.H + h) * p.dk + e / p.dv;
    const size_t step = (size_t)p.H * size, kstep = (size_t)p.H * p.dk;
    float S = *slot;
    constexpr int AHEAD = 8;
    for (int c0 = 0; c0 < count; c0 += AHEAD) {
      float add[AHEAD], f[AHEAD];
#pragma unroll
      for (int q = 0; q < AHEAD; ++q)
        if (c0 + q < count) { add[q] = sc[(size_t)(c0 + q) * step]; f[q] = keep[(size_t)(c0 + q) * kstep]; }
#pragma unroll
      for (int q = 0; q < AHEAD; ++q)
        if (c0 + q < count) {
          sc[(size_t)(c0 + q) * step] = S;
          S = fmaf(f[q], S, add[q]);
        }
    }
    *slot = S;
  }
  pdl_launch_dependents();
}

template <int DK, int DV> struct GatedOutSmem {
  static constexpr int LQ = DK + 4, LKV = (DK > DV ? DK : DV) + 4;      // row strides: a multiple of 4 that walks the banks
  static constexpr int Q = RC * LQ;                                      // queries; then, row by row, the warps' scores
  static constexpr int KV = RC * LKV;                                    // keys, then values
  static constexpr int S = RC * DK > 2 * RC_SLICE * DV ? RC * DK : 2 * RC_SLICE * DV;   // decays, then two slices of the state
  static constexpr int BYTES = (Q + KV + S + 4 * DK) * 4;
};

// grid (chunks, H)
template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(RC_OUT_THREADS) gated_out_kernel(const GatedChunkParams p) {
  using L = GatedOutSmem<DK, DV>;
  extern __shared__ __align__(16) float gc_sm[];
  float* qs = gc_sm;
  float* kv = qs + L::Q;
  float* ss = kv + L::KV;              // first the decays [RC][DK]
  float* tot = ss + L::S;              // [4][DK] product of the decays of each run of 16
  constexpr int TN = DV / 16, SLICES = DK / RC_SLICE, CPL = DK / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = 16 * warp + 8 * (lane >> 4), l16 = lane & 15;
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int t0 = p.chunk_t0[chunk], n = p.chunk_n[chunk];
  const float* S = p.scratch + ((size_t)chunk * p.H + h) * p.dk * p.dv;
  const bool vec_s = p.dv % 4 == 0;
  auto load_slice = [&](int sl) {
    load_block<RC_SLICE, DV, DV>(ss + (sl & 1) * RC_SLICE * DV, S + (size_t)(sl * RC_SLICE < p.dk ? sl * RC_SLICE : 0) * p.dv, p.dv,
                                 p.dk - sl * RC_SLICE, p.dv, vec_s);
  };
  // the warp's 16 tokens: queries, keys, decays (a lane: every 32nd channel)
  {
    float a[CPL], bias[CPL];
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
      const int i = lane + 32 * m;
      const bool in = i < p.dk;
      a[m] = !in ? 0.f : MODE == GC_FIXED ? p.a[h] : MODE == GC_FORGET ? p.a[h * p.dk + i] : 0.f;
      bias[m] = MODE == GC_FORGET && in ? p.bias[h * p.dk + i] : 0.f;
    }
#pragma unroll 1
    for (int b = 0; b < 16; b += 4) {
      float q[4][CPL], x[4][CPL], z[4][CPL];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int m = 0; m < CPL; ++m) {
          const int t = 16 * warp + b + r, i = lane + 32 * m;
          const bool ok = t < n && i < p.dk;
          const float* src = p.proj + (size_t)(t0 + t) * p.ld + h * p.dk + i;
          q[r][m] = ok ? load_now(src + p.off_q) : 0.f;
          x[r][m] = ok ? load_now(src + p.off_k) : 0.f;
          z[r][m] = MODE == GC_GATED && ok ? load_now(p.z + (size_t)(t0 + t) * p.H * p.dk + h * p.dk + i) : 0.f;
        }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int m = 0; m < CPL; ++m) {
          const int t = 16 * warp + b + r, i = lane + 32 * m;
          const bool ok = t < n && i < p.dk;
          float k, d;
          gc_key<MODE>(x[r][m], z[r][m], a[m], bias[m], p.inv_tau, k, d);
          qs[t * L::LQ + i] = MODE == GC_GATED ? q[r][m] * p.q_scale : q[r][m] * sigmoid_f32(q[r][m]);
          kv[t * L::LKV + i] = ok ? k : 0.f;
          ss[t * DK + i] = ok ? d : 1.f;
        }
    }
  }
  __syncwarp();
  // scores inside the run: a lane a key (l16) and half of the channels; the key's product over the decays grows with the query's place
  float near[16];
#pragma unroll
  for (int t = 0; t < 16; ++t) near[t] = 0.f;
  {
    const float* qr = qs + 16 * warp * L::LQ + (lane >> 4) * (DK / 2);
    const float* kr = kv + (16 * warp + l16) * L::LKV + (lane >> 4) * (DK / 2);
    const float* dr = ss + 16 * warp * DK + (lane >> 4) * (DK / 2);
#pragma unroll 1
    for (int i = 0; i < DK / 2; i += 4) {
      const float4 k = *reinterpret_cast<const float4*>(kr + i);
      float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int t = 0; t < 16; ++t) {
        const float4 q = *reinterpret_cast<const float4*>(qr + t * L::LQ + i), d = *reinterpret_cast<const float4*>(dr + t * DK + i);
        const bool own = t == l16;
        g.x = own ? k.x : g.x * d.x;
        g.y = own ? k.y : g.y * d.y;
        g.z = own ? k.z : g.z * d.z;
        g.w = own ? k.w : g.w * d.w;
        near[t] = fmaf(q.w, g.w, fmaf(q.z, g.z, fmaf(q.y, g.y, fmaf(q.x, g.x, near[t]))));
      }
    }
#pragma unroll
    for (int t = 0; t < 16; ++t) near[t] += __shfl_xor_sync(0xffffffffu, near[t], 16);
  }
  __syncwarp();
  // queries from the run's start, keys to its end
#pragma unroll
  for (int m = 0; m < CPL; ++m) {
    const int i = lane + 32 * m;
    float d[16], f = 1.f;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      d[t] = ss[(16 * warp + t) * DK + i];
      f *= d[t];
      qs[(16 * warp + t) * L::LQ + i] *= f;
    }
    tot[warp * DK + i] = f;
    f = 1.f;
#pragma unroll
    for (int t = 15; t >= 0; --t) {
      kv[(16 * warp + t) * L::LKV + i] *= f;
      f *= d[t];
    }
  }
  __syncthreads();                     // the decays are read: their place takes the state
  load_slice(0);
  load_slice(1);                       // (SLICES >= 2)
  // scores of the lane's 8 tokens against keys l16 of the earlier runs, the latest first; the decays of a run passed go into the queries
  float far[8][3];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) far[r][c] = 0.f;
#pragma unroll
  for (int c = 2; c >= 0; --c) {
    if (c >= warp) continue;           // (whole warps)
#pragma unroll 1
    for (int k = 0; k < DK; k += 4) {
      const float4 b = *reinterpret_cast<const float4*>(kv + (l16 + 16 * c) * L::LKV + k);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float4 a = *reinterpret_cast<const float4*>(qs + (row + r) * L::LQ + k);
        far[r][c] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, far[r][c]))));
      }
    }
    __syncwarp();
#pragma unroll
    for (int m = 0; m < CPL; ++m) {
      const int i = lane + 32 * m;
      const float f = tot[c * DK + i];
#pragma unroll
      for (int t = 0; t < 16; ++t) qs[(16 * warp + t) * L::LQ + i] *= f;
    }
    __syncwarp();
  }
  __syncthreads();                     // the keys are read: their place takes the values
  load_block<RC, DV, L::LKV>(kv, p.proj + (size_t)t0 * p.ld + p.off_v + h * p.dv, p.ld, n, p.dv, p.vec_v != 0);
  float acc[8][TN];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < TN; ++c) acc[r][c] = 0.f;
  // groups in flight by age: slice 0, slice 1, the values, slice 2, slice 3
#pragma unroll
  for (int sl = 0; sl < SLICES; ++sl) {
    if (sl == 0) asm volatile("cp.async.wait_group 2;\n" ::);
    else if (sl == 1) asm volatile("cp.async.wait_group %0;\n" ::"n"(SLICES > 2 ? 2 : 1));
    else if (sl == 2) asm volatile("cp.async.wait_group 1;\n" ::);
    else asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    rows_times_block<L::LQ, DV, TN>(acc, qs + row * L::LQ + sl * RC_SLICE, ss + (sl & 1) * RC_SLICE * DV, RC_SLICE);
    if (sl + 2 < SLICES) {
      __syncthreads();
      load_slice(sl + 2);
    }
  }
  // the warp's scores take the place of its queries (no other warp reads those)
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 3; ++c)
    if (c < warp) {
#pragma unroll
      for (int r = 0; r < 8; ++r) qs[(row + r) * L::LQ + l16 + 16 * c] = far[r][c];
    }
  if (lane < 16) {
#pragma unroll
    for (int t = 0; t < 16; ++t) qs[(16 * warp + t) * L::LQ + 16 * warp + l16] = l16 <= t ? near[t] : 0.f;
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  if (MODE == GC_FIXED) {              // the values pass silu too, by the threads that copied them
    if (p.vec_v) {
      for (int e = threadIdx.x; e < RC * (DV / 4); e += RC_OUT_THREADS) {
        float* v = kv + e / (DV / 4) * L::LKV + e % (DV / 4) * 4;
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] *= sigmoid_f32(v[c]);
      }
    } else {
      for (int e = threadIdx.x; e < RC * DV; e += RC_OUT_THREADS) kv[e / DV * L::LKV + e % DV] *= sigmoid_f32(kv[e / DV * L::LKV + e % DV]);
    }
  }
  __syncthreads();                     // the values have landed
  rows_times_block<L::LQ, L::LKV, TN>(acc, qs + row * L::LQ, kv, 16 * warp);
  rows_times_run<L::LQ, L::LKV, TN>(acc, qs + row * L::LQ + 16 * warp, kv + 16 * warp * L::LKV, 8 * (lane >> 4));
  pdl_launch_dependents();
  const bool vec_o = p.dv % 4 == 0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int t = row + r;
    if (t >= n) continue;
    float* o = p.out + (size_t)(t0 + t) * p.H * p.dv + h * p.dv + 4 * l16;
#pragma unroll
    for (int q = 0; q < TN / 4; ++q) {
      if (4 * l16 + 64 * q >= p.dv) continue;
      if (vec_o) {
        const float v[4] = {acc[r][4 * q], acc[r][4 * q + 1], acc[r][4 * q + 2], acc[r][4 * q + 3]};
        rc_store4(o + 64 * q, v);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (4 * l16 + 64 * q + c < p.dv) o[64 * q + c] = acc[r][4 * q + c];
      }
    }
  }
}

template <int DK, int DV, int MODE>
static int launch_gated(const GatedChunkParams& p, int chunks, int runs, cudaStream_t stream) {
  static SharedLimit state_limit, out_limit;      // (per instantiation)
  constexpr size_t smem_state = (size_t)(RC * DK + RC * DV + DK) * 4, smem_out = GatedOutSmem<DK, DV>::BYTES;
  int rc = rc_smem(gated_state_kernel<DK, DV, MODE>, smem_state, state_limit);
  if (rc == SLLM_OK) rc = rc_smem(gated_out_kernel<DK, DV, MODE>, smem_out, out_limit);
  if (rc != SLLM_OK) return rc;
  const dim3 grid((unsigned)chunks, (unsigned)p.H);
  launch_kernel(gated_state_kernel<DK, DV, MODE>, grid, 2 * DK, smem_state, stream, p);
  launch_kernel(gated_scan_kernel, dim3((unsigned)((p.dk * p.dv + RC_SCAN_THREADS - 1) / RC_SCAN_THREADS), (unsigned)p.H, (unsigned)runs), RC_SCAN_THREADS, 0, stream, p);
  launch_kernel(gated_out_kernel<DK, DV, MODE>, grid, RC_OUT_THREADS, smem_out, stream, p);
  return launch_status("gated_chunked");
}

template <int MODE>
static int dispatch_gated(const GatedChunkParams& p, int chunks, int runs, cudaStream_t stream) {
  if (p.dk <= 64 && p.dv <= 64) return launch_gated<64, 64, MODE>(p, chunks, runs, stream);
  if (p.dk <= 64) return launch_gated<64, 128, MODE>(p, chunks, runs, stream);
  if (p.dv <= 64) return launch_gated<128, 64, MODE>(p, chunks, runs, stream);
  return launch_gated<128, 128, MODE>(p, chunks, runs, stream);
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_gated_chunked_supports(int dk, int dv) { return dk >= 1 && dk <= 128 && dv >= 1 && dv <= 128; }

// mode 2 (gated), 3 (a fixed decay per head), 4 (a forget gate that also writes): see the head of the file and delta_rule.cu.  `chunks` pieces of at
// most 64 tokens (chunk_t0: rows, chunk_n) that belong to `runs` requests (run_seq: rows of state_slots; run_first, run_count: their
// chunks, consecutive, all but a request's last 64 tokens long).  scratch: float32 [chunks, H, dk, dv]; keeps: float32 [chunks, H, dk].  Rows of
// other requests are neither read nor written.
SLLM_EXPORT int sllm_gated_chunked(int mode, const float* proj, int ld, int off_q, int off_k, int off_v, const float* z, const float* a,
                                   const float* bias, float q_scale, float inv_tau, float* state, const int* state_slots, const int* chunk_t0,
                                   const int* chunk_n, int chunks, const int* run_seq, const int* run_first, const int* run_count, int runs,
                                   float* scratch, float* keeps, float* out, int H, int dk, int dv, cudaStream_t stream) {
  SLLM_REQUIRE(chunks >= 0 && runs >= 0 && runs <= 65535 && H > 0 && H <= 65535, "gated_chunked: bad sizes chunks=%d runs=%d H=%d", chunks, runs, H);
  SLLM_REQUIRE(sllm_gated_chunked_supports(dk, dv), "gated_chunked: heads of %d x %d are outside 1..128", dk, dv);
  SLLM_REQUIRE(off_q >= 0 && off_k >= 0 && off_v >= 0 && off_q + H * dk <= ld && off_k + H * dk <= ld && off_v + H * dv <= ld,
               "gated_chunked: columns outside the product's %d", ld);
  SLLM_REQUIRE((mode == GC_GATED && z) || (mode == GC_FIXED && a) || (mode == GC_FORGET && a && bias), "gated_chunked: mode %d without what it reads", mode);
  SLLM_REQUIRE(scratch != nullptr && keeps != nullptr && (((uintptr_t)scratch | (uintptr_t)out) & 15) == 0,
               "gated_chunked: scratch and output must be 16-byte aligned");
  if (chunks == 0 || runs == 0) return SLLM_OK;
  GatedChunkParams p;
  p.proj = proj; p.ld = ld; p.off_q = off_q; p.off_k = off_k; p.off_v = off_v; p.z = z; p.a = a; p.bias = bias; p.q_scale = q_scale; p.inv_tau = inv_tau;
  p.state = state; p.state_slots = state_slots; p.chunk_t0 = chunk_t0; p.chunk_n = chunk_n; p.run_seq = run_seq; p.run_first = run_first;
  p.run_count = run_count; p.scratch = scratch; p.keeps = keeps; p.out = out; p.H = H; p.dk = dk; p.dv = dv;
  p.vec_v = ((uintptr_t)proj & 15) == 0 && ld % 4 == 0 && off_v % 4 == 0 && dv % 4 == 0;
  if (mode == GC_GATED) return dispatch_gated<GC_GATED>(p, chunks, runs, stream);
  if (mode == GC_FIXED) return dispatch_gated<GC_FIXED>(p, chunks, runs, stream);
  return dispatch_gated<GC_FORGET>(p, chunks, runs, stream);
}
