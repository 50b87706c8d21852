// A short causal convolution over time on each channel of 32-bit rows, with an optional bias and silu:
//
//   out_t = act( b + sum_{j < taps} w[j, :] * x_(t - taps + 1 + j) )        (zeros before the sequence's start)
//
// for the tokens of a step, which are portions of several sequences.  Unlike causal_taps.cu the input is not added
// to the result, and input and output are 32-bit rows that may be column ranges of wider matrices (a product's
// 32-bit output goes in, what a recurrence reads comes out).  What lies before a portion comes from the sequence's
// state: the last taps - 1 inputs, oldest first, [slots + 1, taps - 1, channels] in 32-bit, zero for a new sequence.
// lb_short_conv reads the state; lb_short_conv_state, launched after it, replaces the state by the last taps - 1
// inputs of (state ++ portion).  The weight comes transposed, [taps, channels], oldest tap first.  A token's sum
// visits the taps in one order whatever the portion, so a result does not depend on how a sequence is cut.
#include "common.cuh"

namespace lb {

// x / (1 + e^-x) as the approximate reciprocal and one step on the quotient's remainder (Markstein's), which leaves half an ulp as a division does at a
// third of its instructions; a division only where the reciprocal would be no normal number or the remainder no number.
__device__ __forceinline__ bool silu_plain(float x) { return fabsf(x) < 80.f; }
__device__ __forceinline__ float silu_divided(float x) { return x / (1.f + expf(-x)); }
__device__ __forceinline__ float silu_near(float x) {
  const float d = 1.f + expf(-x);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float y = x * r;
  return fmaf(fmaf(-y, d, x), r, y);
}
__device__ __forceinline__ float silu_exact(float x) { return silu_plain(x) ? silu_near(x) : silu_divided(x); }
__device__ __forceinline__ void silu_exact(float4& a) {
  if (silu_plain(a.x) && silu_plain(a.y) && silu_plain(a.z) && silu_plain(a.w))
    a = make_float4(silu_near(a.x), silu_near(a.y), silu_near(a.z), silu_near(a.w));
  else
    a = make_float4(silu_exact(a.x), silu_exact(a.y), silu_exact(a.z), silu_exact(a.w));
}

__global__ void short_conv_kernel(float* __restrict__ out, long long out_ld, const float* __restrict__ x, long long x_ld,
                                  const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ state,
                                  const int* __restrict__ token_seq, const int* __restrict__ cu_tokens,
                                  const int* __restrict__ slots, int channels, int taps, int act) {
  pdl_trigger();
  pdl_wait(x, state, token_seq, cu_tokens, slots);
  const int t = blockIdx.x;
  const int s = token_seq[t];
  const int idx = t - cu_tokens[s];                       // place of the token in its portion
  const float* st = state + (size_t)slots[s] * (taps - 1) * channels;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
    float acc = 0.f;
    for (int j = 0; j < taps; ++j) {                      // the input taps - 1 - j tokens back
      const int back = taps - 1 - j;
      const float v = idx - back >= 0 ? x[(size_t)(t - back) * x_ld + c] : st[(size_t)(taps - 1 + idx - back) * channels + c];
      acc = fmaf(w[(size_t)j * channels + c], v, acc);
    }
    if (bias) acc += bias[c];
    out[(size_t)t * out_ld + c] = act ? silu_exact(acc) : acc;
  }
}

// The same with four channels a thread (16-byte words), for rows whose sizes and addresses allow it.  Two tokens a CTA
// would read each input once more from L2 instead of twice; the taps' order within a token's sum is the same.
__global__ void short_conv_x4_kernel(float* __restrict__ out, long long out_ld, const float* __restrict__ x, long long x_ld,
                                     const float* __restrict__ w, const float* __restrict__ bias, const float* __restrict__ state,
                                     const int* __restrict__ token_seq, const int* __restrict__ cu_tokens,
                                     const int* __restrict__ slots, int channels, int taps, int act) {
  pdl_trigger();
  pdl_wait(x, state, token_seq, cu_tokens, slots);
  const int t = blockIdx.x;
  const int s = token_seq[t];
  const int idx = t - cu_tokens[s];
  const float* st = state + (size_t)slots[s] * (taps - 1) * channels;
  for (int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4; c < channels; c += gridDim.y * blockDim.x * 4) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < taps; ++j) {
      const int back = taps - 1 - j;
      const float4 v = *reinterpret_cast<const float4*>(idx - back >= 0 ? x + (size_t)(t - back) * x_ld + c
                                                                         : st + (size_t)(taps - 1 + idx - back) * channels + c);
      const float4 f = *reinterpret_cast<const float4*>(w + (size_t)j * channels + c);
      acc.x = fmaf(f.x, v.x, acc.x); acc.y = fmaf(f.y, v.y, acc.y); acc.z = fmaf(f.z, v.z, acc.z); acc.w = fmaf(f.w, v.w, acc.w);
    }
    if (bias) {
      const float4 b = *reinterpret_cast<const float4*>(bias + c);
      acc.x += b.x; acc.y += b.y; acc.z += b.z; acc.w += b.w;
    }
    if (act) silu_exact(acc);
    *reinterpret_cast<float4*>(out + (size_t)t * out_ld + c) = acc;
  }
}

// Four taps, four channels a thread and TT neighbouring tokens: the inputs of the last three tokens slide through registers, so an
// input is read once and three eighths of it once again (four times with a token a thread), and the weights once.  At a portion's
// start the window comes from the state.  2048 tokens of 4096 channels, 67 MB: 29 us with a token a thread, 22 us with eight, 16 us with
// the silu's reciprocal, one look at the portion for all eight and CTAs of 64 threads (of 256: 18.5); what it moves takes 10.
template <int TT>
__global__ void __launch_bounds__(64) short_conv_x4_tokens_kernel(float* __restrict__ out, long long out_ld, const float* __restrict__ x, long long x_ld,
                                                                   const float* __restrict__ w, const float* __restrict__ bias,
                                                                   const float* __restrict__ state, const int* __restrict__ token_seq,
                                                                   const int* __restrict__ cu_tokens, const int* __restrict__ slots, int num_tokens,
                                                                   int channels, int act) {
  pdl_trigger();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4, t0 = blockIdx.x * TT;
  if (c >= channels) { pdl_wait(); return; }
  float4 f[4], b = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = *reinterpret_cast<const float4*>(w + (size_t)j * channels + c);
  if (bias) b = *reinterpret_cast<const float4*>(bias + c);
  pdl_wait(x, state, token_seq, cu_tokens, slots);
  float4 v[TT + 3];                                // v[i]: the input of token t0 + i - 3
#pragma unroll
  for (int i = 0; i < TT; ++i) v[i + 3] = t0 + i < num_tokens ? *reinterpret_cast<const float4*>(x + (size_t)(t0 + i) * x_ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 3; ++i) v[i] = t0 + i >= 3 ? *reinterpret_cast<const float4*>(x + (size_t)(t0 + i - 3) * x_ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  const int last = min(t0 + TT, num_tokens) - 1, seq = token_seq[t0];
  const bool inside = token_seq[last] == seq && t0 - cu_tokens[seq] >= 3;      // one portion's, and none of its first three tokens
#pragma unroll
  for (int i = 0; i < TT; ++i) {
    const int t = t0 + i;
    if (t > last) break;
    float4 h[3] = {v[i], v[i + 1], v[i + 2]};
    if (!inside) {
      const int s = token_seq[t], idx = t - cu_tokens[s];                        // place of the token in its portion
      if (idx < 3) {
        const float* st = state + (size_t)slots[s] * 3 * channels + c;
#pragma unroll
        for (int j = 0; j < 3; ++j)                // tap j: the input 3 - j tokens back
          if (idx < 3 - j) h[j] = *reinterpret_cast<const float4*>(st + (size_t)(idx + j) * channels);
      }
    }
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 y = j < 3 ? h[j] : v[i + 3];
      a.x = fmaf(f[j].x, y.x, a.x); a.y = fmaf(f[j].y, y.y, a.y); a.z = fmaf(f[j].z, y.z, a.z); a.w = fmaf(f[j].w, y.w, a.w);
    }
    if (bias) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
    if (act) silu_exact(a);
    *reinterpret_cast<float4*>(out + (size_t)t * out_ld + c) = a;
  }
}

// Steps of one token a sequence: the token's output and the state's move in one pass over the state.  The CTAs from `round_from`
// on round other columns of the same rows, which the next product wants in bfloat16, so that these need no launch of their own.
__global__ void __launch_bounds__(256) short_conv_step_kernel(float* __restrict__ out, long long out_ld, const float* __restrict__ x, long long x_ld,
                                                              const float* __restrict__ w, const float* __restrict__ bias, float* __restrict__ state,
                                                              const int* __restrict__ slots, int channels, int act, int round_from,
                                                              bf16* __restrict__ rounded, const float* __restrict__ round_x, long long round_ld, int round_n) {
  pdl_trigger();
  const int s = blockIdx.x;
  if ((int)blockIdx.y >= round_from) {
    const int c = ((blockIdx.y - round_from) * blockDim.x + threadIdx.x) * 4;
    pdl_wait(round_x);
    if (c >= round_n) return;
    const float4 y = *reinterpret_cast<const float4*>(round_x + (size_t)s * round_ld + c);
    __nv_bfloat162 lo = __floats2bfloat162_rn(y.x, y.y), hi = __floats2bfloat162_rn(y.z, y.w);
    *reinterpret_cast<uint2*>(rounded + (size_t)s * round_n + c) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    return;
  }
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (c >= channels) { pdl_wait(); return; }
  float4 f[4], v[4], b = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = *reinterpret_cast<const float4*>(w + (size_t)j * channels + c);
  if (bias) b = *reinterpret_cast<const float4*>(bias + c);
  pdl_wait(x, slots);
  float* st = state + (size_t)slots[s] * 3 * channels + c;
  v[3] = *reinterpret_cast<const float4*>(x + (size_t)s * x_ld + c);
#pragma unroll
  for (int j = 0; j < 3; ++j) v[j] = *reinterpret_cast<const float4*>(st + (size_t)j * channels);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a.x = fmaf(f[j].x, v[j].x, a.x); a.y = fmaf(f[j].y, v[j].y, a.y); a.z = fmaf(f[j].z, v[j].z, a.z); a.w = fmaf(f[j].w, v[j].w, a.w);
  }
  if (bias) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
  if (act) silu_exact(a);
  *reinterpret_cast<float4*>(out + (size_t)s * out_ld + c) = a;
#pragma unroll
  for (int j = 0; j < 3; ++j) *reinterpret_cast<float4*>(st + (size_t)j * channels) = v[j + 1];
}

__global__ void short_conv_state_kernel(float* __restrict__ state, const float* __restrict__ x, long long x_ld,
                                        const int* __restrict__ cu_tokens, const int* __restrict__ slots, int channels, int taps) {
  pdl_trigger();
  pdl_wait(x, cu_tokens, slots);
  const int s = blockIdx.x;
  const int first = cu_tokens[s], n = cu_tokens[s + 1] - first;
  float* st = state + (size_t)slots[s] * (taps - 1) * channels;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < channels; c += gridDim.y * blockDim.x) {
    // entry i of the new state is element n - (taps - 1) + i of the portion, or, where that lies before the
    // portion, entry i + n of the old state; i ascends, so an old entry is read before it is overwritten
    for (int i = 0; i < taps - 1; ++i) {
      const int m = n - (taps - 1) + i;
      st[(size_t)i * channels + c] = m >= 0 ? x[(size_t)(first + m) * x_ld + c] : st[(size_t)(i + n) * channels + c];
    }
  }
}

}  // namespace lb

LB_EXPORT int lb_short_conv(float* out, long long out_ld, const float* x, long long x_ld, const float* w, const float* bias,
                            const float* state, const int* token_seq, const int* cu_tokens, const int* slots, int num_tokens,
                            int channels, int taps, int act, cudaStream_t stream) {
  LB_CHECK_ARG(num_tokens >= 0 && channels > 0 && taps >= 1 && taps <= 16, "short_conv: bad sizes T=%d channels=%d taps=%d",
               num_tokens, channels, taps);
  LB_CHECK_ARG(out && x && w && token_seq && cu_tokens && slots && (taps == 1 || state), "short_conv: null argument");
  LB_CHECK_ARG(out != x, "short_conv: the output must not be the input (a token reads the inputs before it)");
  if (num_tokens == 0) return 0;
  auto a16 = [](const void* q) { return (uintptr_t)q % 16 == 0; };
  if (channels % 4 == 0 && out_ld % 4 == 0 && x_ld % 4 == 0 && a16(out) && a16(x) && a16(w) && a16(bias) && a16(state)) {
    const int threads4 = 64;
    const int by = (channels / 4 + threads4 - 1) / threads4;
    if (taps == 4 && by <= 65535 && num_tokens >= 8) {
      // as many tokens a thread as leave every SM a few CTAs; these are small, so that the last ones leave no SM idle for long (2048 tokens
      // of 12288 channels, cold: 71.7 us with 256 threads and a division, 59 with the reciprocal, 51.2 with 64 threads)
      const long long ctas = (long long)num_tokens * by;
      const int tt = ctas >= 8 * 148 * 16 ? 8 : ctas >= 4 * 148 * 8 ? 4 : ctas >= 2 * 148 * 8 ? 2 : 1;
      const dim3 grid((num_tokens + tt - 1) / tt, by), block(threads4);
      if (tt == 8) lb::launch(lb::short_conv_x4_tokens_kernel<8>, grid, block, 0, stream, out, out_ld, x, x_ld, w, bias, state, token_seq, cu_tokens, slots, num_tokens, channels, act);
      else if (tt == 4) lb::launch(lb::short_conv_x4_tokens_kernel<4>, grid, block, 0, stream, out, out_ld, x, x_ld, w, bias, state, token_seq, cu_tokens, slots, num_tokens, channels, act);
      else if (tt == 2) lb::launch(lb::short_conv_x4_tokens_kernel<2>, grid, block, 0, stream, out, out_ld, x, x_ld, w, bias, state, token_seq, cu_tokens, slots, num_tokens, channels, act);
      if (tt > 1) {
        LB_CHECK_LAUNCH("short_conv");
        return 0;
      }
    }
    int by4 = (channels / 4 + threads4 - 1) / threads4;
    if (by4 > 64) by4 = 64;
    lb::launch(lb::short_conv_x4_kernel, dim3(num_tokens, by4), dim3(threads4), 0, stream, out, out_ld, x, x_ld, w, bias, state,
               token_seq, cu_tokens, slots, channels, taps, act);
    LB_CHECK_LAUNCH("short_conv");
    return 0;
  }
  const int threads = channels >= 256 ? 256 : 64;
  int by = (channels + threads - 1) / threads;
  if (by > 64) by = 64;
  lb::launch(lb::short_conv_kernel, dim3(num_tokens, by), dim3(threads), 0, stream, out, out_ld, x, x_ld, w, bias, state, token_seq,
             cu_tokens, slots, channels, taps, act);
  LB_CHECK_LAUNCH("short_conv");
  return 0;
}

// One token a sequence, four taps: the outputs, and the state moved on, in one launch.  Returns 3 (and launches nothing) for
// operands that are not in whole 16-byte words.  `rounded` (may be null): [num_seqs, round_n] bfloat16 receives the columns at round_x.
LB_EXPORT int lb_short_conv_step(float* out, long long out_ld, const float* x, long long x_ld, const float* w, const float* bias,
                                 float* state, const int* slots, int num_seqs, int channels, int act, void* rounded, const float* round_x,
                                 long long round_ld, int round_n, cudaStream_t stream) {
  LB_CHECK_ARG(out && x && w && state && slots && num_seqs >= 0 && channels > 0, "short_conv_step: bad arguments");
  LB_CHECK_ARG(!rounded || (round_x && round_n > 0 && round_ld >= round_n), "short_conv_step: bad columns to round");
  LB_CHECK_ARG(out != x, "short_conv_step: the output must not be the input");
  auto a16 = [](const void* q) { return (uintptr_t)q % 16 == 0; };
  const int threads = 64, by = (channels / 4 + threads - 1) / threads;
  if (rounded && (round_n % 4 || round_ld % 4 || !a16(round_x) || (uintptr_t)rounded % 8)) return 3;
  const int more = rounded ? (round_n / 4 + threads - 1) / threads : 0;
  if (channels % 4 || out_ld % 4 || x_ld % 4 || !a16(out) || !a16(x) || !a16(w) || !a16(bias) || !a16(state) || by + more > 65535) return 3;
  if (num_seqs == 0) return 0;
  lb::launch(lb::short_conv_step_kernel, dim3(num_seqs, by + more), dim3(threads), 0, stream, out, out_ld, x, x_ld, w, bias, state, slots, channels, act,
             by, (lb::bf16*)rounded, round_x, round_ld, round_n);
  LB_CHECK_LAUNCH("short_conv_step");
  return 0;
}

LB_EXPORT int lb_short_conv_state(float* state, const float* x, long long x_ld, const int* cu_tokens, const int* slots,
                                  int num_seqs, int channels, int taps, cudaStream_t stream) {
  LB_CHECK_ARG(num_seqs >= 0 && channels > 0 && taps >= 2 && taps <= 16, "short_conv_state: bad sizes");
  LB_CHECK_ARG(state && x && cu_tokens && slots, "short_conv_state: null argument");
  if (num_seqs == 0) return 0;
  const int threads = channels >= 256 ? 256 : 64;
  int by = (channels + threads - 1) / threads;
  if (by > 64) by = 64;
  lb::launch(lb::short_conv_state_kernel, dim3(num_seqs, by), dim3(threads), 0, stream, state, x, x_ld, cu_tokens, slots, channels, taps);
  LB_CHECK_LAUNCH("short_conv_state");
  return 0;
}
