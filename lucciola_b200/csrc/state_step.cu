// One token a sequence through the linear recurrences (decode steps of the bfloat16 engine), every kind that chunk_recurrence.cu
// lists with its formulas: the state of a head is read, moved on by one token and written back.
//
// Such a step is a stream of the states, 64 KB a head of 128 x 128 read and as much written.  A CTA of 256 threads takes
// 4 * VL value columns of a head: a thread four neighbouring columns of every (256 / VL)-th row, requested all at once as
// 16-byte words and kept in registers, so that with two CTAs an SM 128 KB are under way; sums over the rows go through the
// warp (VL < 32) and then through shared memory, in one order.  Narrower CTAs (VL 16, 8) where the heads alone would leave
// SMs idle.  The kernels that walk several tokens stage the state in shared memory, and their loads follow one another.
//
// Channel decays, 64 requests of 16 heads of 128 x 128 (134 MB in and out): 55 -> 25.6 us, 5.2 TB/s.
#include "common.cuh"

namespace lb {

enum StepKind : int { SS_FIXED = 0, SS_SSM = 1, SS_DELTA = 2, SS_HGRN2 = 3, SS_CHANNELS = 4 };

struct StateStepParams {
  const float* q; const float* k; const float* v; const float* a; const float* b;    // hgrn2: k is the gate's input
  long long q_ld, k_ld, v_ld, a_ld, b_ld;
  const float* A_log; const float* dt_bias; const float* D; const float* bias; const float* lower; const float* decay;
  float* state; float* out; long long out_ld;
  const int* cu_tokens; const int* slots;
  int heads, groups, dim, vdim, unit_norm, act;
  float q_scale, unit_eps;
};

__device__ __forceinline__ float ss_sigmoid(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float ss_silu(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float ss_softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

template <int KIND, int VL, int RPT>
__global__ void __launch_bounds__(256, RPT == 16 ? 2 : RPT == 8 ? 3 : 4) state_step_kernel(StateStepParams p) {
  constexpr bool DELTA = KIND == SS_DELTA || KIND == SS_CHANNELS, ROWS = KIND == SS_HGRN2 || KIND == SS_CHANNELS;
  constexpr int G = 256 / VL;                      // rows side by side
  __shared__ float qs[128], ks[128], gs[128], red[8];
  __shared__ float4 part[8][VL];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, seq = blockIdx.z, grp = h / (p.heads / p.groups);
  const int c4 = tid % VL, rg = tid / VL, col = (blockIdx.x * VL + c4) * 4;
  const bool live = col < p.vdim;                  // vdim is a multiple of four
  pdl_wait();
  const int t = p.cu_tokens[seq];
  float* S = p.state + ((size_t)p.slots[seq] * p.heads + h) * p.dim * p.vdim + col;
  float4 s[RPT];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = i * G + rg;
    s[i] = live && r < p.dim ? *reinterpret_cast<const float4*>(S + (size_t)r * p.vdim) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // q by the first half of the threads, k by the second
  const int d = tid & 127;
  float x = 0.f;
  if (d < p.dim) x = tid < 128 ? p.q[(size_t)t * p.q_ld + (size_t)grp * p.dim + d] : p.k[(size_t)t * p.k_ld + (size_t)grp * p.dim + d];
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (live) {
    const float* vr = p.v + (size_t)t * p.v_ld + (size_t)h * p.vdim + col;
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = vr[e];
  }
  float g = 1.f, w = 1.f;
  if (KIND == SS_FIXED) {
    g = p.decay[h];
    if (p.act) {
      x = ss_silu(x);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = ss_silu(v[e]);
    }
  }
  if (KIND == SS_SSM || KIND == SS_DELTA) {
    const float sp = ss_softplus(p.a[(size_t)t * p.a_ld + h] + p.dt_bias[h]);
    g = expf(-expf(p.A_log[h]) * sp);
    w = sp;
  }
  if (DELTA) w = ss_sigmoid(p.b[(size_t)t * p.b_ld + h]);
  if (KIND == SS_CHANNELS && tid >= 128) {         // as channel_decay_kernel of state_recurrence.cu
    gs[d] = 1.f;
    if (d < p.dim) gs[d] = expf(-expf(p.A_log[h]) * ss_softplus(p.a[(size_t)t * p.a_ld + (size_t)h * p.dim + d] + p.dt_bias[h * p.dim + d]));
  }
  if (KIND == SS_HGRN2) {
    if (tid < 128) x = ss_silu(x);
    else {
      const float low = d < p.dim ? p.lower[h * p.dim + d] : 1.f, bi = d < p.dim ? p.bias[h * p.dim + d] : 0.f;
      gs[d] = low + (1.f - low) * ss_sigmoid(x + bi);
    }
  }
  (tid < 128 ? qs : ks)[d] = x;
  if (DELTA) {
    const float ss = warp_sum(x * x);
    if (lane == 0) red[warp] = ss;
  }
  __syncthreads();
  float fq = 1.f, fk = 1.f;
  if (DELTA && p.unit_norm) {
    fq = p.q_scale / sqrtf((red[0] + red[1]) + (red[2] + red[3]) + p.unit_eps);
    fk = 1.f / sqrtf((red[4] + red[5]) + (red[6] + red[7]) + p.unit_eps);
  }
  if (ROWS && DELTA) {
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const float f = gs[(i * G + rg) & 127];
      s[i].x *= f; s[i].y *= f; s[i].z *= f; s[i].w *= f;
    }
  }
  // the sum of a thread's rows over the CTA: through the warp, then through `part`, in warp order
  auto gather = [&](float4 y) {
#pragma unroll
    for (int m = VL; m < 32; m <<= 1) {
      y.x += __shfl_xor_sync(0xffffffffu, y.x, m); y.y += __shfl_xor_sync(0xffffffffu, y.y, m);
      y.z += __shfl_xor_sync(0xffffffffu, y.z, m); y.w += __shfl_xor_sync(0xffffffffu, y.w, m);
    }
    if (lane < VL) part[warp][lane] = y;
  };
  auto total = [&]() {
    float4 y = part[0][c4];
#pragma unroll
    for (int i = 1; i < 8; ++i) { const float4 z = part[i][c4]; y.x += z.x; y.y += z.y; y.z += z.z; y.w += z.w; }
    return y;
  };
  float u[4];
  if (DELTA) {
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const float k = ks[(i * G + rg) & 127];
      y.x = fmaf(s[i].x, k, y.x); y.y = fmaf(s[i].y, k, y.y); y.z = fmaf(s[i].z, k, y.z); y.w = fmaf(s[i].w, k, y.w);
    }
    gather(y);
    __syncthreads();
    y = total();
    u[0] = w * (v[0] - g * (fk * y.x)); u[1] = w * (v[1] - g * (fk * y.y)); u[2] = w * (v[2] - g * (fk * y.z)); u[3] = w * (v[3] - g * (fk * y.w));
    __syncthreads();                               // `part` is read
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) u[e] = w * v[e];
  }
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int r = i * G + rg;
    if (KIND == SS_HGRN2) {                        // f s + (1 - f) v as v + f (s - v)
      const float f = gs[r & 127];
      s[i].x = fmaf(f, s[i].x - u[0], u[0]); s[i].y = fmaf(f, s[i].y - u[1], u[1]);
      s[i].z = fmaf(f, s[i].z - u[2], u[2]); s[i].w = fmaf(f, s[i].w - u[3], u[3]);
    } else {
      const float k = ks[r & 127] * fk;
      s[i].x = fmaf(g, s[i].x, k * u[0]); s[i].y = fmaf(g, s[i].y, k * u[1]);
      s[i].z = fmaf(g, s[i].z, k * u[2]); s[i].w = fmaf(g, s[i].w, k * u[3]);
    }
    const float q = r < p.dim ? qs[r & 127] : 0.f;
    o.x = fmaf(s[i].x, q, o.x); o.y = fmaf(s[i].y, q, o.y); o.z = fmaf(s[i].z, q, o.z); o.w = fmaf(s[i].w, q, o.w);
    if (live && r < p.dim) *reinterpret_cast<float4*>(S + (size_t)r * p.vdim) = s[i];
  }
  gather(o);
  __syncthreads();
  if (rg == 0 && live) {
    o = total();
    const float Dh = p.D ? p.D[h] : 0.f;
    float* dst = p.out + (size_t)t * p.out_ld + (size_t)h * p.vdim + col;
    dst[0] = fmaf(fq, o.x, Dh * v[0]); dst[1] = fmaf(fq, o.y, Dh * v[1]); dst[2] = fmaf(fq, o.z, Dh * v[2]); dst[3] = fmaf(fq, o.w, Dh * v[3]);
  }
}

template <int KIND, int VL>
static cudaError_t launch_state_step(const StateStepParams& p, int num_seqs, cudaStream_t stream) {
  constexpr int G = 256 / VL, R = 128 / G;         // 16, 8, 4 rows a thread for up to 128
  const dim3 grid((p.vdim + 4 * VL - 1) / (4 * VL), p.heads, num_seqs), block(256);
  if (p.dim <= 64) return launch(state_step_kernel<KIND, VL, R / 2>, grid, block, 0, stream, p);
  return launch(state_step_kernel<KIND, VL, R>, grid, block, 0, stream, p);
}

// The widest CTAs of which there are two an SM.
template <int KIND>
static cudaError_t launch_state_step_kind(const StateStepParams& p, int num_seqs, cudaStream_t stream) {
  const long long heads = (long long)num_seqs * p.heads;
  if (p.vdim > 64 && heads * ((p.vdim + 127) / 128) >= 296) return launch_state_step<KIND, 32>(p, num_seqs, stream);
  if (p.vdim > 32 && heads * ((p.vdim + 63) / 64) >= 296) return launch_state_step<KIND, 16>(p, num_seqs, stream);
  return launch_state_step<KIND, 8>(p, num_seqs, stream);
}

}  // namespace lb

// Every sequence of the step brings one token.  Operands as lb_chunk_recurrence's; channel decays are formed here from `a` as the
// product left it (with 16 heads a CTA has 128 of them to form, and a launch less to wait for).
LB_EXPORT int lb_state_step(int kind, const float* q, long long q_ld, const float* k, long long k_ld, const float* v, long long v_ld,
                            const float* a, long long a_ld, const float* b, long long b_ld, const float* A_log, const float* dt_bias,
                            const float* D, const float* bias, const float* lower, const float* decay, float* state, float* out,
                            long long out_ld, const int* cu_tokens, const int* slots, int num_seqs, int heads, int groups, int dim,
                            int vdim, int unit_norm, float q_scale, float unit_eps, int act, cudaStream_t stream) {
  LB_CHECK_ARG(kind >= 0 && kind <= lb::SS_CHANNELS, "state_step: kind %d", kind);
  LB_CHECK_ARG(q && k && v && state && out && cu_tokens && slots, "state_step: null argument");
  LB_CHECK_ARG(heads > 0 && heads <= 65535 && groups > 0 && heads % groups == 0, "state_step: %d heads are not a multiple of %d groups", heads, groups);
  LB_CHECK_ARG(dim > 0 && dim <= 128 && vdim > 0 && vdim % 4 == 0 && ((uintptr_t)state & 15) == 0, "state_step: a state of %d x %d", dim, vdim);
  LB_CHECK_ARG(num_seqs >= 0 && num_seqs <= 65535, "state_step: %d sequences", num_seqs);
  LB_CHECK_ARG(kind != lb::SS_FIXED || decay, "state_step: no decays");
  const bool delta = kind == lb::SS_DELTA || kind == lb::SS_CHANNELS;
  LB_CHECK_ARG((kind != lb::SS_SSM && !delta) || (a && A_log && dt_bias), "state_step: null argument");
  LB_CHECK_ARG(!delta || b, "state_step: null argument");
  LB_CHECK_ARG(kind != lb::SS_HGRN2 || (bias && lower), "state_step: null argument");
  if (num_seqs == 0) return 0;
  lb::StateStepParams p;
  p.q = q; p.k = k; p.v = v; p.a = a; p.b = b; p.q_ld = q_ld; p.k_ld = k_ld; p.v_ld = v_ld; p.a_ld = a_ld; p.b_ld = b_ld;
  p.A_log = A_log; p.dt_bias = dt_bias; p.D = D; p.bias = bias; p.lower = lower; p.decay = decay;
  p.state = state; p.out = out; p.out_ld = out_ld; p.cu_tokens = cu_tokens; p.slots = slots;
  p.heads = heads; p.groups = groups; p.dim = dim; p.vdim = vdim; p.unit_norm = unit_norm; p.act = act;
  p.q_scale = q_scale; p.unit_eps = unit_eps;
  cudaError_t e;
  switch (kind) {
    case lb::SS_FIXED: e = lb::launch_state_step_kind<lb::SS_FIXED>(p, num_seqs, stream); break;
    case lb::SS_SSM: e = lb::launch_state_step_kind<lb::SS_SSM>(p, num_seqs, stream); break;
    case lb::SS_DELTA: e = lb::launch_state_step_kind<lb::SS_DELTA>(p, num_seqs, stream); break;
    case lb::SS_HGRN2: e = lb::launch_state_step_kind<lb::SS_HGRN2>(p, num_seqs, stream); break;
    default: e = lb::launch_state_step_kind<lb::SS_CHANNELS>(p, num_seqs, stream); break;
  }
  if (e != cudaSuccess) { lb::set_error("state_step: %s", cudaGetErrorString(e)); return 2; }
  LB_CHECK_LAUNCH("state_step");
  return 0;
}
