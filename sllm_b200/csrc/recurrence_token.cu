// The recurrences of delta_rule.cu (modes 0 to 4) for a step in which every request brings ONE token, and what follows them in a layer.
//
// With one token there is nothing to walk: a state is read once, changed and written once, and what bounds the kernel is that traffic.  A
// CTA takes one (request, head) and holds its state in registers, 16 bytes a load along the value channels and all of a thread's rows in flight
// at once (64 KB a CTA at 128 x 128), while its threads make the token's vectors; the sums over rows (u^T S where the rule removes, then
// S^T r) end in shared memory.  The walk's form keeps every eighth row of a column in a lane, 4 bytes a row and lane where the state is
// cut into 16-column slices: 16 requests x 16 heads of 128 x 128 31 us for 34 MB, now 11.9 (floor 5.1).  The CTA has the head's
// whole output, so its norm, gain and gate, and the rounding to the compute type, are done here too: one kernel less a layer.
#include "common.cuh"

namespace sllm {

constexpr int RT_THREADS = 256;

struct TokenParams {
  const float* proj;           // [S, ld]
  int ld, off_q, off_k, off_v, off_a;
  const float* decay;          // mode 0: [S, H*dk] decay logits; mode 2: [S, H*dk]
  const float* a;              // mode 0: removal bias [H*dk]; mode 1: A_log [H]; mode 3: decays [H]; mode 4: lower bounds [H*dk]
  const float* bias;           // mode 1: dt_bias [H]; mode 4: [H*dk]
  const float* gates;          // mode 1: [S, ldg], rate logits at off_b + h, decay logits at off_dt + h
  int ldg, off_b, off_dt, hdiv;
  float q_scale, inv_tau;
  float* state;                // [slots, H, dk, dv]
  const int* state_slots;      // [S]
  int H, dk, dv;
  // what follows: gain != null or gate >= 0: o / sqrt(mean o^2 + eps) * gain * act(gate logit)
  int norm, gate_act;          // norm 0: o as it is; gate_act 0 sigmoid, 1 silu, 2 none
  const float* gain;           // [H*dv]; null: ones
  const float* gate;           // [S, ld_gate], logits at off_g + h*dv
  int ld_gate, off_g;
  float eps;
  int out_ld, out_off;
};

// sum of v over the threads below `n` (a multiple of 32), known to all; `sums`: n / 32 floats of its own
__device__ __forceinline__ float rt_sum(float v, float* sums, int n) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0 && threadIdx.x < n) sums[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int w = 0; w < n / 32; ++w) t += sums[w];
  return t;
}

template <int DKP, int DVP, int MODE, typename TO>
__global__ void __launch_bounds__(RT_THREADS, 2) recurrence_token_kernel(const TokenParams p, TO* __restrict__ out) {
  constexpr int LV = DVP / 4, RG = RT_THREADS / LV, RPT = DKP / RG;      // lanes over the value channels, rows at a time, rows a thread
  __shared__ __align__(16) float u[DKP], d[DKP], au[DKP], k[DKP], r[DKP], v[DVP], part[RG][DVP], sums[24];
  const int tid = threadIdx.x;
  pdl_wait();
  const int t = blockIdx.x, h = blockIdx.y, dk = p.dk, dv = p.dv;
  const int col = tid % LV * 4, row = tid / LV;
  float* S = p.state + ((size_t)p.state_slots[t] * p.H + h) * dk * dv;
  float4 s[RPT];
#pragma unroll
  for (int n = 0; n < RPT; ++n) {
    const int i = row + n * RG;
    s[n] = i < dk && col < dv ? *reinterpret_cast<const float4*>(S + (size_t)i * dv + col) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // ---- the token's vectors, a thread a channel ----
  const float* x = p.proj + (size_t)t * p.ld;
  const int kh = h / p.hdiv;
  const bool in = tid < dk;
  float kx = in ? x[p.off_k + kh * dk + tid] : 0.f, qx = in ? x[p.off_q + kh * dk + tid] : 0.f;
  float vx = tid < dv ? x[p.off_v + h * dv + tid] : 0.f;
  float g = 1.f, bg = 0.f;             // mode 1: the head's decay, and the rate times it
  if (MODE == 0) {
    const float inv = 1.0f / sqrtf(rt_sum(kx * kx, sums, DKP) + 1e-6f);
    const float z = in ? p.decay[(size_t)t * p.H * dk + h * dk + tid] : 0.f;
    const float a = in ? x[p.off_a + h * dk + tid] + p.a[h * dk + tid] : 0.f;
    if (tid < DKP) {
      u[tid] = kx * inv;
      au[tid] = sigmoid_f32(a) * (kx * inv);
      d[tid] = expf(-expf(-0.5f) * sigmoid_f32(z));
    }
  } else if (MODE == 1) {
    const float* gr = p.gates + (size_t)t * p.ldg;
    const float beta = sigmoid_f32(gr[p.off_b + h]);
    const float dt = gr[p.off_dt + h] + p.bias[h];
    g = expf(-expf(p.a[h]) * (fmaxf(dt, 0.f) + log1pf(expf(-fabsf(dt)))));
    bg = beta * g;
    const float kinv = 1.0f / sqrtf(rt_sum(kx * kx, sums, DKP) + 1e-6f);
    const float qinv = p.q_scale / sqrtf(rt_sum(qx * qx, sums + 8, DKP) + 1e-6f);
    kx *= kinv;
    qx *= qinv;
    vx *= beta;
  } else if (MODE == 2) {
    const float z = in ? p.decay[(size_t)t * p.H * dk + h * dk + tid] : 0.f;
    if (tid < DKP) d[tid] = expf((fminf(z, 0.f) - log1pf(expf(-fabsf(z)))) * p.inv_tau);
    qx *= p.q_scale;
  } else if (MODE == 3) {
    kx *= sigmoid_f32(kx);
    qx *= sigmoid_f32(qx);
    vx *= sigmoid_f32(vx);
    g = p.a[h];
  } else {
    const float lo = in ? p.a[h * dk + tid] : 0.f, b = in ? p.bias[h * dk + tid] : 0.f;
    const float f = lo + (1.0f - lo) * sigmoid_f32(kx + b);
    if (tid < DKP) d[tid] = f;
    kx = in ? 1.0f - f : 0.f;
    qx *= sigmoid_f32(qx);
  }
  if (tid < DKP) {
    k[tid] = kx;
    r[tid] = qx;
  }
  if (tid < DVP) v[tid] = vx;
  __syncthreads();
  // ---- what the rule removes: the sum over the state's rows before the token ----
  float4 vv = *reinterpret_cast<const float4*>(v + col), gone = make_float4(0.f, 0.f, 0.f, 0.f);
  if (MODE == 0 || MODE == 1) {
    const float* w = MODE == 0 ? u : k;
#pragma unroll
    for (int n = 0; n < RPT; ++n) {
      const float f = w[row + n * RG];
      gone.x = fmaf(f, s[n].x, gone.x); gone.y = fmaf(f, s[n].y, gone.y); gone.z = fmaf(f, s[n].z, gone.z); gone.w = fmaf(f, s[n].w, gone.w);
    }
    *reinterpret_cast<float4*>(&part[row][col]) = gone;
    __syncthreads();
    gone = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int n = 0; n < RG; ++n) {
      const float4 o = *reinterpret_cast<const float4*>(&part[n][col]);
      gone.x += o.x; gone.y += o.y; gone.z += o.z; gone.w += o.w;
    }
    __syncthreads();
    if (MODE == 1) {                   // written along the key it removes
      vv.x = fmaf(-bg, gone.x, vv.x); vv.y = fmaf(-bg, gone.y, vv.y); vv.z = fmaf(-bg, gone.z, vv.z); vv.w = fmaf(-bg, gone.w, vv.w);
    }
  }
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int n = 0; n < RPT; ++n) {
    const int i = row + n * RG;
    const float keep = MODE == 1 || MODE == 3 ? g : d[i], ki = k[i], ri = r[i];
    s[n].x *= keep; s[n].y *= keep; s[n].z *= keep; s[n].w *= keep;
    if (MODE == 0) {
      const float a = -au[i];
      s[n].x = fmaf(a, gone.x, s[n].x); s[n].y = fmaf(a, gone.y, s[n].y); s[n].z = fmaf(a, gone.z, s[n].z); s[n].w = fmaf(a, gone.w, s[n].w);
    }
    s[n].x = fmaf(ki, vv.x, s[n].x); s[n].y = fmaf(ki, vv.y, s[n].y); s[n].z = fmaf(ki, vv.z, s[n].z); s[n].w = fmaf(ki, vv.w, s[n].w);
    o.x = fmaf(ri, s[n].x, o.x); o.y = fmaf(ri, s[n].y, o.y); o.z = fmaf(ri, s[n].z, o.z); o.w = fmaf(ri, s[n].w, o.w);
    if (i < dk && col < dv) *reinterpret_cast<float4*>(S + (size_t)i * dv + col) = s[n];
  }
  *reinterpret_cast<float4*>(&part[row][col]) = o;
  pdl_launch_dependents();
  __syncthreads();
  float y = 0.f;
  if (tid < DVP) {
#pragma unroll
    for (int n = 0; n < RG; ++n) y += part[n][tid];
  }
  if (p.norm) {
    const float inv = 1.0f / sqrtf(rt_sum(tid < dv ? y * y : 0.f, sums + 16, DVP) / (float)dv + p.eps);
    if (tid < dv) {
      float z = 1.f;
      if (p.gate_act != 2) {
        z = p.gate[(size_t)t * p.ld_gate + p.off_g + h * dv + tid];
        z = p.gate_act == 1 ? z * sigmoid_f32(z) : sigmoid_f32(z);
      }
      y = y * inv * (p.gain != nullptr ? p.gain[h * dv + tid] : 1.0f) * z;
    }
  }
  if (tid < dv) out[(size_t)t * p.out_ld + p.out_off + h * dv + tid] = from_f32<TO>(y);
}

template <int DKP, int DVP, typename TO>
static void launch_token(int mode, const TokenParams& p, int S, TO* out, cudaStream_t stream) {
  auto kernel = mode == 0 ? recurrence_token_kernel<DKP, DVP, 0, TO> : mode == 1 ? recurrence_token_kernel<DKP, DVP, 1, TO>
              : mode == 2 ? recurrence_token_kernel<DKP, DVP, 2, TO> : mode == 3 ? recurrence_token_kernel<DKP, DVP, 3, TO>
                                                                            : recurrence_token_kernel<DKP, DVP, 4, TO>;
  launch_kernel(kernel, dim3((unsigned)S, (unsigned)p.H), RT_THREADS, 0, stream, p, out);
}

template <typename TO>
static int dispatch_token(int mode, const TokenParams& p, int S, TO* out, cudaStream_t stream) {
  if (p.dk <= 64 && p.dv <= 64) launch_token<64, 64, TO>(mode, p, S, out, stream);
  else if (p.dk <= 64) launch_token<64, 128, TO>(mode, p, S, out, stream);
  else if (p.dv <= 64) launch_token<128, 64, TO>(mode, p, S, out, stream);
  else launch_token<128, 128, TO>(mode, p, S, out, stream);
  return launch_status("recurrence_token");
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_recurrence_token_supports(int dk, int dv) { return dk >= 1 && dk <= 128 && dv >= 4 && dv <= 128 && dv % 4 == 0; }

// S requests of one token each (row s of `proj` and of the output is request s).  mode, proj, offsets, decay, a, bias, gates: see TokenParams.  norm 0: out
// [S, out_ld] receives the heads' outputs at columns out_off ..; else their norm, gain and gate on the way (gate_act 2: no gate).
SLLM_EXPORT int sllm_recurrence_token(int mode, const float* proj, int ld, int off_q, int off_k, int off_v, int off_a, const float* decay,
                                      const float* a, const float* bias, const float* gates, int ldg, int off_b, int off_dt, int key_heads,
                                      float q_scale, float inv_tau, float* state, const int* state_slots, int S, int H, int dk, int dv, int norm,
                                      int gate_act, const float* gain, const float* gate, int ld_gate, int off_g, float eps, void* out,
                                      int out_dtype, int out_ld, int out_off, cudaStream_t stream) {
  SLLM_REQUIRE(S >= 0 && H > 0 && H <= 65535 && key_heads > 0 && H % key_heads == 0, "recurrence_token: bad sizes S=%d H=%d key heads=%d", S, H, key_heads);
  SLLM_REQUIRE(sllm_recurrence_token_supports(dk, dv) && ((uintptr_t)state & 15) == 0, "recurrence_token: heads of %d x %d (at most 128, value channels a multiple of 4) on 16 bytes", dk, dv);
  SLLM_REQUIRE(off_q >= 0 && off_k >= 0 && off_v >= 0 && off_a >= 0 && off_q + key_heads * dk <= ld && off_k + key_heads * dk <= ld &&
                   off_v + H * dv <= ld && (mode != 0 || off_a + H * dk <= ld), "recurrence_token: columns outside the product's %d", ld);
  SLLM_REQUIRE(mode >= 0 && mode <= 4 && (mode == 1 || key_heads == H) && (mode == 2 || a) && ((mode != 0 && mode != 2) || decay) && ((mode != 1 && mode != 4) || bias) &&
                   (mode != 1 || (gates && off_b >= 0 && off_dt >= 0 && off_b + H <= ldg && off_dt + H <= ldg)), "recurrence_token: mode %d without what it reads", mode);
  SLLM_REQUIRE(gate_act >= 0 && gate_act <= 2 && (!norm || gate_act == 2 || (gate && off_g >= 0 && off_g + H * dv <= ld_gate)), "recurrence_token: gate columns outside %d", ld_gate);
  SLLM_REQUIRE(out_off >= 0 && out_off + H * dv <= out_ld, "recurrence_token: the output's columns lie outside its %d", out_ld);
  if (S == 0) return SLLM_OK;
  TokenParams p;
  p.proj = proj; p.ld = ld; p.off_q = off_q; p.off_k = off_k; p.off_v = off_v; p.off_a = off_a; p.decay = decay; p.a = a; p.bias = bias; p.gates = gates;
  p.ldg = ldg; p.off_b = off_b; p.off_dt = off_dt; p.hdiv = H / key_heads; p.q_scale = q_scale; p.inv_tau = inv_tau; p.state = state; p.state_slots = state_slots;
  p.H = H; p.dk = dk; p.dv = dv; p.norm = norm; p.gate_act = gate_act; p.gain = gain; p.gate = gate; p.ld_gate = ld_gate; p.off_g = off_g; p.eps = eps;
  p.out_ld = out_ld; p.out_off = out_off;
  if (out_dtype == SLLM_F32) return dispatch_token<float>(mode, p, S, (float*)out, stream);
  if (out_dtype == SLLM_BF16) return dispatch_token<__nv_bfloat16>(mode, p, S, (__nv_bfloat16*)out, stream);
  SLLM_REQUIRE(false, "recurrence_token: unknown dtype %d", out_dtype);
}
