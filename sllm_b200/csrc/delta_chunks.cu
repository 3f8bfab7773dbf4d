// The delta rules over prompt portions, a chunk of 64 tokens at a time (delta_rule.cu walks them token by token and keeps single tokens and
// short portions).  Both are
//
//   S_t = diag(d_t) S_(t-1) - w_t (p_t^T S_(t-1)) + k_t v_t^T,   o_t = S_t^T q_t
//
// whose removal makes every token's write depend on the tokens before it.  Inside a chunk that is a triangular system: with X the 64 rows that
// are written along w (gated: along k), the state S the chunk meets, F_t the product of the decays up to and including t,
//
//   X = Xv - Xk S,   O = Q S + A X (+ O0),   S' = diag(F_n) S + Kn^T X (+ N)
//
// where Xv and Xk solve (I + L) [Xv | Xk] = [right sides] and everything but S comes from the chunk alone:
//   gated (delta_rule.cu's mode 1; one decay g and one rate b per head, unit keys k, unit scaled queries q):
//     L_ts = b_t R_ts (k_t . k_s), s < t;  right sides b_t v_t and b_t F_t k_t;  A_ts = R_ts (q_t . k_s), s <= t;  Q = F_t q_t;
//     Kn = R_nt k_t;  R_ts the product of the decays behind s up to t (products, never a quotient: a decay may be zero)
//   general (mode 0; decays per channel, never below exp(-exp(-1/2)) = 0.545, so that 1 / F_t stays below 1e17 in a chunk):
//     p = u F_(t-1), q = r F_t, k' = k / F_t, w' = a u / F_t:  L_ts = p_t . w'_s;  right sides -sum_(s<t) (p_t . k'_s) v_s and p_t;
//     A_ts = q_t . w'_s;  O0 = sum_(s<=t) (q_t . k'_s) v_s;  Kn = F_n w';  N = sum_s (F_n k'_s) v_s^T
//
//   1. prep   per (chunk, head): the products and the triangular system, a thread a column of the right sides, 16 rows of it in registers at
//             a time (all 64 unrolled were 40 to 160 KB of instructions, read from L2 by every CTA: 400 of 553 us), to scratch;
//   2. scan   per (request, head, 16 value channels): S through the request's chunks in order, X and the state each chunk meets to
//             scratch, the last state to the slot.  The only serial part: two products of 64 x dk x 16 a chunk;
//   3. out    per (chunk, head): O.
//
// A walk is a chain of dependent sums per token (about 0.4 us a token at 128 x 128); here the chain is one step per 64 tokens.  All arithmetic is
// float32 on the CUDA cores.
#include <math.h>

#include "chunked.cuh"

namespace sllm {

constexpr int DC_GENERAL = 0, DC_GATED = 1;                    // delta_rule.cu's modes
constexpr int DC_THREADS = 256, DC_PITCH = RC + 4, DC_COLS = 16;

struct DeltaChunkParams {
  const float* proj;           // [T, ld]
  int ld, off_q, off_k, off_v, off_a;
  const float* decay;          // general: [T, H*dk] decay logits
  const float* a_bias;         // general: [H*dk]
  const float* gates;          // gated: [T, ldg], rate logits at off_b + h, decay logits at off_dt + h
  int ldg, off_b, off_dt, hdiv;
  const float* a_log;          // gated: [H]
  const float* dt_bias;        // gated: [H]
  float q_scale;
  float* state;                // [slots, H, dk, dv]
  const int* state_slots;      // [S]
  const int* chunk_t0;         // [chunks] first token (row of proj)
  const int* chunk_n;          // [chunks] tokens, 1 .. 64
  const int* run_seq;          // [runs] a request ...
  const int* run_first;        // [runs] ... its first chunk ...
  const int* run_count;        // [runs] ... and how many it has
  // scratch, per (chunk, head), DK and DV the padded sizes
  float* xv;                   // [RC][DV] Xv, then X
  float* xk;                   // [DK][RC] Xk, its columns as rows
  float* kn;                   // [RC][DK]
  float* q;                    // [RC][DK]
  float* a;                    // [RC][RC]
  float* keep;                 // [DK] F_n
  float* s;                    // [DK][DV] N, then the state the chunk meets
  float* out;                  // [T, H*dv]; general: O0 until the last kernel
  int H, dk, dv;
  int vec_v;
};

// x[t] += f m[t], t < 16, from shared memory
__device__ __forceinline__ void dc_add16(float (&x)[16], const float* __restrict__ m, float f) {
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    const float4 l = *reinterpret_cast<const float4*>(m + 4 * g);
    x[4 * g] = fmaf(l.x, f, x[4 * g]);
    x[4 * g + 1] = fmaf(l.y, f, x[4 * g + 1]);
    x[4 * g + 2] = fmaf(l.z, f, x[4 * g + 2]);
    x[4 * g + 3] = fmaf(l.w, f, x[4 * g + 3]);
  }
}
// the rows 16 run .. of a lower triangular product: x[t] += sum over s < 16 run of m[s][t] v_s, and over the run's own s before t (or up to t);
// row s of `m` holds column s of the triangle
template <bool UP_TO>
__device__ __forceinline__ void dc_lower16(float (&x)[16], const float* __restrict__ m, const float* __restrict__ v, int ldv, int run) {
#pragma unroll 2
  for (int s = 0; s < 16 * run; ++s) dc_add16(x, m + s * DC_PITCH + 16 * run, v[s * ldv]);
#pragma unroll 1
  for (int s = 0; s < 16; ++s) {
    const float f = v[(16 * run + s) * ldv];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float4 l = *reinterpret_cast<const float4*>(m + (16 * run + s) * DC_PITCH + 16 * run + 4 * g);
      const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int t = 4 * g + c;
        if (UP_TO ? t >= s : t > s) x[t] = fmaf(lv[c], f, x[t]);
      }
    }
  }
}
// the rows 16 run .. of (I + L) x = right side, in place; `col`: the column's rows before, done
__device__ __forceinline__ void dc_solve16(float (&x)[16], const float* __restrict__ lt, const float* __restrict__ col, int ld, int run) {
#pragma unroll 2
  for (int s = 0; s < 16 * run; ++s) dc_add16(x, lt + s * DC_PITCH + 16 * run, -col[s * ld]);
#pragma unroll
  for (int s = 0; s < 15; ++s) {
    const float f = -x[s];
#pragma unroll
    for (int g = (s + 1) / 4; g < 4; ++g) {
      const float4 l = *reinterpret_cast<const float4*>(lt + (16 * run + s) * DC_PITCH + 16 * run + 4 * g);
      const float lv[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (4 * g + c > s) x[4 * g + c] = fmaf(lv[c], f, x[4 * g + c]);
    }
  }
}

// c[i][j] (+)= a row ty + 16 i of A times row tx + 16 j of B, j <= i, over DK channels (rows LD apart)
template <int DK, int LD>
__device__ __forceinline__ void dc_products(float (&c0)[4][4], float (&c1)[4][4], const float* __restrict__ A0, const float* __restrict__ A1,
                                            const float* __restrict__ B, int ty, int tx) {
#pragma unroll 1
  for (int k = 0; k < DK; k += 4) {
    float4 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(B + (tx + 16 * j) * LD + k);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(A0 + (ty + 16 * i) * LD + k), y = *reinterpret_cast<const float4*>(A1 + (ty + 16 * i) * LD + k);
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        c0[i][j] = fmaf(x.w, b[j].w, fmaf(x.z, b[j].z, fmaf(x.y, b[j].y, fmaf(x.x, b[j].x, c0[i][j]))));
        c1[i][j] = fmaf(y.w, b[j].w, fmaf(y.z, b[j].z, fmaf(y.y, b[j].y, fmaf(y.x, b[j].x, c1[i][j]))));
      }
    }
  }
}

template <int DK, int DV> struct GatedPrepSmem {
  static constexpr int LD = DK + 4, LV = (DK > DV ? DK : DV) + 4;
  static constexpr int BYTES = (RC * LD + RC * LV + RC * DC_PITCH + 4 * RC + 8) * 4;
};

// grid (chunks, H); DK + DV <= 256 columns of right sides, a thread each
template <int DK, int DV>
__global__ void __launch_bounds__(DC_THREADS, 2) gated_delta_prep_kernel(const DeltaChunkParams p) {
  using L = GatedPrepSmem<DK, DV>;
  constexpr int LD = L::LD, LV = L::LV;
  extern __shared__ __align__(16) float dc_sm[];
  float* ks = dc_sm;                   // [RC][LD] unit keys, then the columns of Xk
  float* qs = ks + RC * LD;            // [RC][LD] unit queries, scaled; then [RC][LV] the columns of Xv
  float* lt = qs + RC * LV;            // [RC][DC_PITCH] column s of L in row s
  float* beta = lt + RC * DC_PITCH;    // [RC]
  float* g = beta + RC;                // [RC]
  float* head = g + RC;                // [RC] product of the decays from the start of t's run of 16 up to t
  float* tail = head + RC;             // [RC] ... behind t to the end of its run
  float* tot = tail + RC;              // [4] of a run
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y, kh = h / p.hdiv;
  const int t0 = p.chunk_t0[chunk], n = p.chunk_n[chunk];
  const size_t at = (size_t)chunk * p.H + h;
  if (tid < RC) {
    float b = 0.f, d = 1.f;
    if (tid < n) {
      const float* gr = p.gates + (size_t)(t0 + tid) * p.ldg;
      b = sigmoid_f32(gr[p.off_b + h]);
      const float x = gr[p.off_dt + h] + p.dt_bias[h];
      d = expf(-expf(p.a_log[h]) * (fmaxf(x, 0.f) + log1pf(expf(-fabsf(x)))));
    }
    beta[tid] = b;
    g[tid] = d;
  }
  constexpr int CPL = DK / 32;
#pragma unroll 1
  for (int r = 0; r < RC / 8; r += 4) {              // a warp's eight tokens, four of them in flight
    float k[4][CPL], q[4][CPL];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int m = 0; m < CPL; ++m) {
        const int t = 8 * warp + r + u, i = lane + 32 * m;
        const bool ok = t < n && i < p.dk;
        const float* src = p.proj + (size_t)(t0 + t) * p.ld + kh * p.dk + i;
        k[u][m] = ok ? load_now(src + p.off_k) : 0.f;
        q[u][m] = ok ? load_now(src + p.off_q) : 0.f;
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float sk = 0.f, sq = 0.f;
#pragma unroll
      for (int m = 0; m < CPL; ++m) { sk = fmaf(k[u][m], k[u][m], sk); sq = fmaf(q[u][m], q[u][m], sq); }
      sk = 1.0f / sqrtf(warp_sum(sk) + 1e-6f);
      sq = p.q_scale / sqrtf(warp_sum(sq) + 1e-6f);
#pragma unroll
      for (int m = 0; m < CPL; ++m) {
        ks[(8 * warp + r + u) * LD + lane + 32 * m] = k[u][m] * sk;
        qs[(8 * warp + r + u) * LD + lane + 32 * m] = q[u][m] * sq;
      }
    }
  }
  __syncthreads();
  if (tid < RC) {                                    // (what a run needs of its decays; read after the products' barrier)
    const int run = tid & ~15;
    float a = 1.f, b = 1.f;
    for (int t = run; t < run + 16; ++t) {
      if (t <= tid) a *= g[t]; else b *= g[t];
    }
    head[tid] = a;
    tail[tid] = b;
    if ((tid & 15) == 15) tot[tid >> 4] = a;
  }
  const int ty = tid / 16, tx = tid % 16;
  float kk[4][4], qk[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) kk[i][j] = qk[i][j] = 0.f;
  dc_products<DK, LD>(kk, qk, ks, qs, ks, ty, tx);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = ty + 16 * i;
    float between = 1.f;                             // the whole runs between
#pragma unroll
    for (int j = i; j >= 0; --j) {
      const int s = tx + 16 * j;
      float r = 0.f;
      if (j == i) {
        if (tx <= ty) {
          r = 1.f;
          for (int u = s + 1; u <= t; ++u) r *= g[u];
        }
      } else {
        r = head[t] * between * tail[s];
        between *= tot[j];
      }
      lt[s * DC_PITCH + t] = s < t ? beta[t] * r * kk[i][j] : 0.f;
      p.a[at * RC * RC + t * RC + s] = s <= t ? r * qk[i][j] : 0.f;
    }
  }
  // what the scan and the last kernel read: keys carried to the chunk's end, queries from its start
  for (int e = tid; e < RC * DK / 4; e += DC_THREADS) {
    const int t = e / (DK / 4), i = e % (DK / 4) * 4, run = t >> 4;
    float f = head[t], b = tail[t];
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      if (o < run) f *= tot[o];
      if (o > run) b *= tot[o];
    }
    const float4 k = *reinterpret_cast<const float4*>(ks + t * LD + i), q = *reinterpret_cast<const float4*>(qs + t * LD + i);
    *reinterpret_cast<float4*>(p.kn + (at * RC + t) * DK + i) = make_float4(k.x * b, k.y * b, k.z * b, k.w * b);
    *reinterpret_cast<float4*>(p.q + (at * RC + t) * DK + i) = make_float4(q.x * f, q.y * f, q.z * f, q.w * f);
  }
  if (tid < DK) p.keep[at * DK + tid] = tot[0] * tot[1] * tot[2] * tot[3];
  __syncthreads();                     // the queries are read: their place takes the values
  if (tid < DV) {
    const float* v = p.proj + (size_t)t0 * p.ld + p.off_v + h * p.dv + tid;
#pragma unroll 16
    for (int t = 0; t < RC; ++t) qs[t * LV + tid] = t < n && tid < p.dv ? beta[t] * load_now(v + (size_t)t * p.ld) : 0.f;
  } else if (tid < DV + DK) {
    float f = 1.f;
    for (int run = 0; run < 4; ++run) {
#pragma unroll
      for (int t = 16 * run; t < 16 * run + 16; ++t) ks[t * LD + tid - DV] *= beta[t] * (head[t] * f);
      f *= tot[run];
    }
  }
  if (tid < DV + DK) {                 // (a thread's own column: nothing to wait for)
    float* col = tid < DV ? qs + tid : ks + tid - DV;
    const int ld = tid < DV ? LV : LD;
#pragma unroll 1
    for (int run = 0; run < 4; ++run) {
      float x[16];
#pragma unroll
      for (int t = 0; t < 16; ++t) x[t] = col[(16 * run + t) * ld];
      dc_solve16(x, lt, col, ld, run);
#pragma unroll
      for (int t = 0; t < 16; ++t) col[(16 * run + t) * ld] = x[t];
      if (tid < DV) {
#pragma unroll
        for (int t = 0; t < 16; ++t) p.xv[(at * RC + 16 * run + t) * DV + tid] = x[t];
      } else {
#pragma unroll
        for (int t = 0; t < 16; t += 4)
          *reinterpret_cast<float4*>(p.xk + (at * DK + tid - DV) * RC + 16 * run + t) = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
      }
    }
  }
  pdl_launch_dependents();
}

constexpr int GENERAL_PREP_BYTES = (5 * RC * DC_PITCH + RC * 64 + RC + 4 * 64 + 64) * 4;

// grid (chunks, H), heads of up to 64 x 64
__global__ void __launch_bounds__(DC_THREADS, 2) general_delta_prep_kernel(const DeltaChunkParams p) {
  constexpr int D = 64, LD = DC_PITCH;
  extern __shared__ __align__(16) float dc_sm[];
  float* pu = dc_sm;                   // [RC][LD] u F_(t-1), then the columns of Xk
  float* qr = pu + RC * LD;            // [RC][LD] r F_t; then column s of (q . k') in row s
  float* kt = qr + RC * LD;            // [RC][LD] k / F_t; then the columns of -Xv
  float* wt = kt + RC * LD;            // [RC][LD] a u / F_t; then column s of (p . k') in row s
  float* lt = wt + RC * LD;            // [RC][LD] column s of L in row s
  float* vs = lt + RC * LD;            // [RC][D]
  float* kinv = vs + RC * D;           // [RC]
  float* tot = kinv + RC;              // [4][D] product of the decays of a run of 16
  float* last = tot + 4 * D;           // [D] F_n
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int t0 = p.chunk_t0[chunk], n = p.chunk_n[chunk];
  const size_t at = (size_t)chunk * p.H + h;
  load_block<RC, D, D>(vs, p.proj + (size_t)t0 * p.ld + p.off_v + h * p.dv, p.ld, n, p.dv, p.vec_v != 0);
  // the keys' lengths: a warp's eight tokens
  {
    float k[8][2];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int t = 8 * warp + u, i = lane + 32 * m;
        k[u][m] = t < n && i < p.dk ? load_now(p.proj + (size_t)(t0 + t) * p.ld + p.off_k + h * p.dk + i) : 0.f;
      }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float ss = warp_sum(fmaf(k[u][0], k[u][0], k[u][1] * k[u][1]));
      if (lane == 0) kinv[8 * warp + u] = 1.0f / sqrtf(ss + 1e-6f);
    }
  }
  // a thread a channel and 16 tokens: the decays, their running product, and the four vectors
  const int i = tid % D, run = tid / D;
  const bool in = i < p.dk;
  {
    float d[16], r[16], k[16], a[16];
    const float* row = p.proj + (size_t)t0 * p.ld + h * p.dk + i;
    const float bias = in ? p.a_bias[h * p.dk + i] : 0.f, c = -expf(-0.5f);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int t = 16 * run + u;
      const bool ok = in && t < n;
      d[u] = ok ? load_now(p.decay + (size_t)(t0 + t) * p.H * p.dk + h * p.dk + i) : 0.f;
      r[u] = ok ? load_now(row + (size_t)t * p.ld + p.off_q) : 0.f;
      k[u] = ok ? load_now(row + (size_t)t * p.ld + p.off_k) : 0.f;
      a[u] = ok ? load_now(row + (size_t)t * p.ld + p.off_a) : 0.f;
    }
    float f = 1.f;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      d[u] = in && 16 * run + u < n ? expf(c * sigmoid_f32(d[u])) : 1.f;
      f *= d[u];
    }
    tot[run * D + i] = f;
    __syncthreads();
    f = 1.f;
    float all = 1.f;
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      if (o < run) f *= tot[o * D + i];
      all *= tot[o * D + i];
    }
    if (run == 0) {
      last[i] = all;
      p.keep[at * D + i] = all;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int t = 16 * run + u;
      const float unit = k[u] * kinv[t];
      pu[t * LD + i] = unit * f;
      f *= d[u];
      const float inv = 1.0f / f, w = in && t < n ? sigmoid_f32(a[u] + bias) * unit * inv : 0.f;
      qr[t * LD + i] = r[u] * f;
      kt[t * LD + i] = k[u] * inv;
      wt[t * LD + i] = w;
      p.q[(at * RC + t) * D + i] = r[u] * f;
      p.kn[(at * RC + t) * D + i] = w * all;
    }
  }
  __syncthreads();
  const int ty = tid / 16, tx = tid % 16;
  float bk[4][4], ak[4][4], bw[4][4], aw[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) bk[a][b] = ak[a][b] = bw[a][b] = aw[a][b] = 0.f;
  dc_products<D, LD>(bk, ak, pu, qr, kt, ty, tx);
  dc_products<D, LD>(bw, aw, pu, qr, wt, ty, tx);
  __syncthreads();                     // the queries and the removals are read: the scores take their places
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int t = ty + 16 * a, s = tx + 16 * b;
      if (b <= a) {
        wt[s * LD + t] = s < t ? bk[a][b] : 0.f;
        qr[s * LD + t] = s <= t ? ak[a][b] : 0.f;
        lt[s * LD + t] = s < t ? bw[a][b] : 0.f;
        p.a[at * RC * RC + t * RC + s] = s <= t ? aw[a][b] : 0.f;
      }
    }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  const int col = tid % 64, part = tid / 64;
  float x[16];
  {                                    // N: 16 rows a thread
#pragma unroll
    for (int t = 0; t < 16; ++t) x[t] = 0.f;
#pragma unroll 2
    for (int t = 0; t < n; ++t) dc_add16(x, kt + t * LD + 16 * part, vs[t * D + col]);
#pragma unroll
    for (int k = 0; k < 16; ++k) p.s[(at * D + 16 * part + k) * D + col] = x[k] * last[16 * part + k];
  }
  __syncthreads();                     // the keys are read: their place takes the solution
  if (part < 2) {                      // the written rows without the state, and their dependence on it
    float* mine = part == 0 ? kt + col : pu + col;
#pragma unroll 1
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int t = 0; t < 16; ++t) x[t] = part == 0 ? 0.f : mine[(16 * r + t) * LD];
      if (part == 0) dc_lower16<false>(x, wt, vs + col, D, r);
      dc_solve16(x, lt, mine, LD, r);
#pragma unroll
      for (int t = 0; t < 16; ++t) mine[(16 * r + t) * LD] = x[t];
      if (part == 0) {
#pragma unroll
        for (int t = 0; t < 16; ++t) p.xv[(at * RC + 16 * r + t) * D + col] = -x[t];
      } else {
#pragma unroll
        for (int t = 0; t < 16; t += 4)
          *reinterpret_cast<float4*>(p.xk + (at * D + col) * RC + 16 * r + t) = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
      }
    }
  } else {                             // O0: runs 0 and 3, or 1 and 2
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int r = part == 2 ? 3 * half : 1 + half;
#pragma unroll
      for (int t = 0; t < 16; ++t) x[t] = 0.f;
      dc_lower16<true>(x, qr, vs + col, D, r);
#pragma unroll
      for (int t = 0; t < 16; ++t)
        if (16 * r + t < n && col < p.dv) p.out[(size_t)(t0 + 16 * r + t) * p.H * p.dv + h * p.dv + col] = x[t];
    }
  }
  pdl_launch_dependents();
}

template <int DK> struct DeltaScanSmem {
  static constexpr int XK = DK * RC, KN = RC * DK, WARPS = DC_THREADS / 32;
  static constexpr int BYTES = (2 * XK + 2 * KN + DK * DC_COLS + WARPS * RC * DC_COLS + RC * DC_COLS) * 4;
};

// grid (DV / 16, H, runs).  Warp w owns rows w DK/8 .. of the state: their part of Xk S, and their update.
template <int DK, int MODE>
__global__ void __launch_bounds__(DC_THREADS) delta_scan_kernel(const DeltaChunkParams p, int DV) {
  using L = DeltaScanSmem<DK>;
  constexpr int KW = DK / L::WARPS, KQ = KW / 4;     // rows a warp, groups of four of them
  constexpr int CL = 32 / KQ, CN = DC_COLS / CL;     // lanes over the columns, columns a lane
  extern __shared__ __align__(16) float dc_sm[];
  float* xk = dc_sm;                   // [2][DK][RC]
  float* kn = xk + 2 * L::XK;          // [2][RC][DK]
  float* ss = kn + 2 * L::KN;          // [DK][DC_COLS] the state
  float* part = ss + DK * DC_COLS;     // [WARPS][RC][DC_COLS]
  float* xs = part + L::WARPS * RC * DC_COLS;      // [RC][DC_COLS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  const int c0 = blockIdx.x * DC_COLS, h = blockIdx.y, run = blockIdx.z;
  const int first = p.run_first[run], count = p.run_count[run];
  float* S = p.state + ((size_t)p.state_slots[p.run_seq[run]] * p.H + h) * p.dk * p.dv;
  auto fetch = [&](int c) {
    const size_t at = (size_t)(first + c) * p.H + h;
    const float *a = p.xk + at * L::XK, *b = p.kn + at * L::KN;
    float *da = xk + (c & 1) * L::XK, *db = kn + (c & 1) * L::KN;
#pragma unroll 4
    for (int e = tid * 4; e < L::XK; e += DC_THREADS * 4) {
      rc_cp16(da + e, a + e, true);
      rc_cp16(db + e, b + e, true);
    }
    rc_commit();
  };
  // the lane's rows and columns of the state
  const int k0 = warp * KW + lane / CL * 4, cl = lane % CL * CN;
  float s[4][CN];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < CN; ++c) s[r][c] = k0 + r < p.dk && c0 + cl + c < p.dv ? S[(size_t)(k0 + r) * p.dv + c0 + cl + c] : 0.f;
  // what a chunk brings beside the two blocks: general, one chunk ahead in registers (N comes from far: 242 -> 126 us at 2,048 tokens of 32 heads); gated,
  // when it is met (115 us against 132 ahead, 16 heads of 128 x 128)
  constexpr bool AHEAD = MODE == DC_GENERAL;
  float keep[4], add[4][CN], next_keep[4], next_add[4][CN];
  float4 xv, next_xv;
  auto bring = [&](int c, float (&k)[4], float (&n)[4][CN], float4& x) {
    const size_t at = (size_t)(first + c) * p.H + h;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      k[r] = load_now_l2(p.keep + at * DK + k0 + r);
#pragma unroll
      for (int q = 0; q < CN; ++q) n[r][q] = MODE == DC_GENERAL ? load_now_l2(p.s + (at * DK + k0 + r) * DV + c0 + cl + q) : 0.f;
    }
    x = load_now_l2(reinterpret_cast<const float4*>(p.xv + (at * RC + tid / 4) * DV + c0 + tid % 4 * 4));
  };
  fetch(0);
  if (AHEAD) bring(0, keep, add, xv);
  const int tg = lane / 4 * 4, cg = lane % 4 * 4;    // phase 1: the lane's tokens tg .. and 32 + tg .., its columns
  for (int c = 0; c < count; ++c) {
    const size_t at = (size_t)(first + c) * p.H + h;
    if (AHEAD && c + 1 < count) {
      fetch(c + 1);
      bring(c + 1, next_keep, next_add, next_xv);
    }
    if (!AHEAD) bring(c, keep, add, xv);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < CN; ++q) {
        p.s[(at * DK + k0 + r) * DV + c0 + cl + q] = s[r][q];        // (N of this chunk has been read)
        ss[(k0 + r) * DC_COLS + cl + q] = s[r][q];
      }
    if (c + 1 < count) {
      if (!AHEAD) fetch(c + 1);
      asm volatile("cp.async.wait_group 1;\n" ::);
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::);
    }
    __syncthreads();
    float acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[r][q] = 0.f;
    const float* a = xk + (c & 1) * L::XK + warp * KW * RC + tg;
#pragma unroll 4
    for (int k = 0; k < KW; ++k) {
      const float4 lo = *reinterpret_cast<const float4*>(a + k * RC), hi = *reinterpret_cast<const float4*>(a + k * RC + 32);
      const float4 b = *reinterpret_cast<const float4*>(ss + (warp * KW + k) * DC_COLS + cg);
      const float av[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        acc[r][0] = fmaf(av[r], b.x, acc[r][0]);
        acc[r][1] = fmaf(av[r], b.y, acc[r][1]);
        acc[r][2] = fmaf(av[r], b.z, acc[r][2]);
        acc[r][3] = fmaf(av[r], b.w, acc[r][3]);
      }
    }
    float* mine = part + warp * RC * DC_COLS + cg;
#pragma unroll
    for (int r = 0; r < 8; ++r) rc_store4(mine + (tg + r % 4 + r / 4 * 32) * DC_COLS, acc[r]);
    __syncthreads();
    {
      float x[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int w = 0; w < L::WARPS; ++w) {
        const float4 y = *reinterpret_cast<const float4*>(part + w * RC * DC_COLS + tid * 4);
        x[0] -= y.x; x[1] -= y.y; x[2] -= y.z; x[3] -= y.w;
      }
      rc_store4(xs + tid * 4, x);
      rc_store4(p.xv + (at * RC + tid / 4) * DV + c0 + tid % 4 * 4, x);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < CN; ++q) s[r][q] = fmaf(keep[r], s[r][q], add[r][q]);
    const float* kp = kn + (c & 1) * L::KN + k0;
#pragma unroll 8
    for (int t = 0; t < RC; ++t) {
      const float4 k = *reinterpret_cast<const float4*>(kp + t * DK);
      float x[CN];
#pragma unroll
      for (int q = 0; q < CN; ++q) x[q] = xs[t * DC_COLS + cl + q];
#pragma unroll
      for (int q = 0; q < CN; ++q) {
        s[0][q] = fmaf(k.x, x[q], s[0][q]);
        s[1][q] = fmaf(k.y, x[q], s[1][q]);
        s[2][q] = fmaf(k.z, x[q], s[2][q]);
        s[3][q] = fmaf(k.w, x[q], s[3][q]);
      }
    }
    if (AHEAD) {
      xv = next_xv;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        keep[r] = next_keep[r];
#pragma unroll
        for (int q = 0; q < CN; ++q) add[r][q] = next_add[r][q];
      }
    }
    __syncthreads();                   // the buffers of this chunk are read
  }
  pdl_launch_dependents();
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < CN; ++c)
      if (k0 + r < p.dk && c0 + cl + c < p.dv) S[(size_t)(k0 + r) * p.dv + c0 + cl + c] = s[r][c];
}

template <int DK, int DV> struct DeltaOutSmem {
  static constexpr int LQ = (DK > RC ? DK : RC) + 4;
  static constexpr int BYTES = (RC * LQ + RC * (DV + 4) + 2 * RC_SLICE * DV) * 4;
};

// grid (chunks, H)
template <int DK, int DV, int MODE>
__global__ void __launch_bounds__(RC_OUT_THREADS) delta_chunk_out_kernel(const DeltaChunkParams p) {
  using L = DeltaOutSmem<DK, DV>;
  constexpr int TN = DV / 16, SLICES = DK / RC_SLICE, LX = DV + 4;
  extern __shared__ __align__(16) float dc_sm[];
  float* qs = dc_sm;                   // [RC][LQ] queries, then the scores
  float* xs = qs + RC * L::LQ;         // [RC][LX]
  float* ss = xs + RC * LX;            // two slices of the state
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = 16 * warp + 8 * (lane >> 4), l16 = lane & 15;
  pdl_wait();
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int t0 = p.chunk_t0[chunk], n = p.chunk_n[chunk];
  const size_t at = (size_t)chunk * p.H + h;
  auto load_slice = [&](int sl) {
    load_block<RC_SLICE, DV, DV>(ss + (sl & 1) * RC_SLICE * DV, p.s + (at * DK + sl * RC_SLICE) * DV, DV, RC_SLICE, DV, true);
  };
  load_block<RC, DK, L::LQ>(qs, p.q + at * RC * DK, DK, RC, DK, true);
  load_slice(0);
  load_slice(1);                       // (SLICES >= 2)
  load_block<RC, DV, LX>(xs, p.xv + at * RC * DV, DV, RC, DV, true);
  float acc[8][TN];
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int c = 0; c < TN; ++c) acc[r][c] = 0.f;
  // groups in flight by age: queries, slice 0, slice 1, X, slice 2, slice 3
#pragma unroll
  for (int sl = 0; sl < SLICES; ++sl) {
    if (sl == 0) asm volatile("cp.async.wait_group 2;\n" ::);
    else if (sl == 1) asm volatile("cp.async.wait_group %0;\n" ::"n"(SLICES > 2 ? 2 : 1));
    else if (sl == 2) asm volatile("cp.async.wait_group 1;\n" ::);
    else asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    rows_times_block<L::LQ, DV, TN>(acc, qs + row * L::LQ + sl * RC_SLICE, ss + (sl & 1) * RC_SLICE * DV, RC_SLICE);
    __syncthreads();
    if (sl + 2 < SLICES) load_slice(sl + 2);
  }
  load_block<RC, RC, L::LQ>(qs, p.a + at * RC * RC, RC, RC, RC, true);
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  rows_times_block<L::LQ, LX, TN>(acc, qs + row * L::LQ, xs, 16 * warp);
  rows_times_run<L::LQ, LX, TN>(acc, qs + row * L::LQ + 16 * warp, xs + 16 * warp * LX, 8 * (lane >> 4));
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
      float v[4] = {acc[r][4 * q], acc[r][4 * q + 1], acc[r][4 * q + 2], acc[r][4 * q + 3]};
      if (vec_o) {
        if (MODE == DC_GENERAL) {
          const float4 b = *reinterpret_cast<const float4*>(o + 64 * q);
          v[0] += b.x; v[1] += b.y; v[2] += b.z; v[3] += b.w;
        }
        rc_store4(o + 64 * q, v);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (4 * l16 + 64 * q + c < p.dv) o[64 * q + c] = v[c] + (MODE == DC_GENERAL ? o[64 * q + c] : 0.f);
      }
    }
  }
}

template <int DK, int DV, int MODE>
static int launch_delta_chunks(const DeltaChunkParams& p, int chunks, int runs, cudaStream_t stream) {
  static SharedLimit prep_limit, scan_limit, out_limit;      // (per instantiation)
  const size_t smem_prep = MODE == DC_GATED ? GatedPrepSmem<DK, DV>::BYTES : GENERAL_PREP_BYTES;
  constexpr size_t smem_scan = DeltaScanSmem<DK>::BYTES, smem_out = DeltaOutSmem<DK, DV>::BYTES;
  void (*prep)(const DeltaChunkParams);
  if constexpr (MODE == DC_GATED) prep = gated_delta_prep_kernel<DK, DV>;
  else prep = general_delta_prep_kernel;
  int rc = rc_smem(prep, smem_prep, prep_limit);
  if (rc == SLLM_OK) rc = rc_smem(delta_scan_kernel<DK, MODE>, smem_scan, scan_limit);
  if (rc == SLLM_OK) rc = rc_smem(delta_chunk_out_kernel<DK, DV, MODE>, smem_out, out_limit);
  if (rc != SLLM_OK) return rc;
  const dim3 grid((unsigned)chunks, (unsigned)p.H);
  launch_kernel(prep, grid, DC_THREADS, smem_prep, stream, p);
  launch_kernel(delta_scan_kernel<DK, MODE>, dim3(DV / DC_COLS, (unsigned)p.H, (unsigned)runs), DC_THREADS, smem_scan, stream, p, DV);
  launch_kernel(delta_chunk_out_kernel<DK, DV, MODE>, grid, RC_OUT_THREADS, smem_out, stream, p);
  return launch_status("delta_chunked");
}

}  // namespace sllm

using namespace sllm;

static int padded64(int d) { return d <= 64 ? 64 : 128; }

SLLM_EXPORT int sllm_delta_chunked_supports(int mode, int dk, int dv) {
  const int most = mode == DC_GATED ? 128 : mode == DC_GENERAL ? 64 : 0;
  return dk >= 1 && dk <= most && dv >= 1 && dv <= most;
}

// floats of scratch per chunk and head
SLLM_EXPORT int sllm_delta_chunked_scratch(int dk, int dv) {
  const int K = padded64(dk), V = padded64(dv);
  return RC * V + 3 * RC * K + RC * RC + K + K * V;
}

// mode 0 (general: r | k | v | removal logits at off_q, off_k, off_v, off_a of `proj`, `decay` logits and `a_bias`) or 1 (gated: q | k | v, `gates`,
// `a_log`, `dt_bias`, q_scale): see the head of the file and delta_rule.cu.  `chunks` pieces of at most 64 tokens (chunk_t0: rows, chunk_n) that
// belong to `runs` requests (run_seq: rows of state_slots; run_first, run_count: their chunks, consecutive, all but a request's last 64
// tokens long).  scratch: chunks * H * sllm_delta_chunked_scratch floats.  Rows of other requests are neither read nor written.
SLLM_EXPORT int sllm_delta_chunked(int mode, const float* proj, int ld, int off_q, int off_k, int off_v, int off_a, const float* decay,
                                   const float* a_bias, const float* gates, int ldg, int off_b, int off_dt, const float* a_log,
                                   const float* dt_bias, float q_scale, float* state, const int* state_slots, const int* chunk_t0,
                                   const int* chunk_n, int chunks, const int* run_seq, const int* run_first, const int* run_count, int runs,
                                   float* scratch, float* out, int H, int key_heads, int dk, int dv, cudaStream_t stream) {
  SLLM_REQUIRE(chunks >= 0 && runs >= 0 && runs <= 65535 && H > 0 && H <= 65535 && key_heads > 0 && H % key_heads == 0,
               "delta_chunked: bad sizes chunks=%d runs=%d H=%d key heads=%d", chunks, runs, H, key_heads);
  SLLM_REQUIRE(sllm_delta_chunked_supports(mode, dk, dv), "delta_chunked: mode %d does not take heads of %d x %d", mode, dk, dv);
  SLLM_REQUIRE(off_q >= 0 && off_k >= 0 && off_v >= 0 && off_a >= 0 && off_q + key_heads * dk <= ld && off_k + key_heads * dk <= ld &&
                   off_v + H * dv <= ld && (mode == DC_GATED || off_a + H * dk <= ld), "delta_chunked: columns outside the product's %d", ld);
  SLLM_REQUIRE(mode == DC_GATED ? gates && a_log && dt_bias && off_b >= 0 && off_dt >= 0 && off_b + H <= ldg && off_dt + H <= ldg
                                : decay && a_bias && key_heads == H, "delta_chunked: mode %d without what it reads", mode);
  SLLM_REQUIRE(scratch != nullptr && (((uintptr_t)scratch | (uintptr_t)out) & 15) == 0, "delta_chunked: scratch and output must be 16-byte aligned");
  if (chunks == 0 || runs == 0) return SLLM_OK;
  DeltaChunkParams p;
  p.proj = proj; p.ld = ld; p.off_q = off_q; p.off_k = off_k; p.off_v = off_v; p.off_a = off_a; p.decay = decay; p.a_bias = a_bias;
  p.gates = gates; p.ldg = ldg; p.off_b = off_b; p.off_dt = off_dt; p.hdiv = H / key_heads; p.a_log = a_log; p.dt_bias = dt_bias; p.q_scale = q_scale;
  p.state = state; p.state_slots = state_slots; p.chunk_t0 = chunk_t0; p.chunk_n = chunk_n; p.run_seq = run_seq; p.run_first = run_first;
  p.run_count = run_count; p.out = out; p.H = H; p.dk = dk; p.dv = dv;
  const size_t pieces = (size_t)chunks * H, K = padded64(dk), V = padded64(dv);
  p.xv = scratch;
  p.xk = p.xv + pieces * RC * V;
  p.kn = p.xk + pieces * RC * K;
  p.q = p.kn + pieces * RC * K;
  p.a = p.q + pieces * RC * K;
  p.s = p.a + pieces * RC * RC;
  p.keep = p.s + pieces * K * V;
  p.vec_v = ((uintptr_t)proj & 15) == 0 && ld % 4 == 0 && off_v % 4 == 0 && dv % 4 == 0;
  if (mode == DC_GENERAL) return launch_delta_chunks<64, 64, DC_GENERAL>(p, chunks, runs, stream);
  if (K == 64 && V == 64) return launch_delta_chunks<64, 64, DC_GATED>(p, chunks, runs, stream);
  if (K == 64) return launch_delta_chunks<64, 128, DC_GATED>(p, chunks, runs, stream);
  if (V == 64) return launch_delta_chunks<128, 64, DC_GATED>(p, chunks, runs, stream);
  return launch_delta_chunks<128, 128, DC_GATED>(p, chunks, runs, stream);
}
