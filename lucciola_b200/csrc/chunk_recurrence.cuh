// What the kernels of the chunked recurrences share (chunk_recurrence.cu has the formulas): the parameters of a launch, where a chunk
// lies, the numbers of its tokens, and the cutting of 32-bit operands in three.
#pragma once

#include "common.cuh"
#include "warp_mma.cuh"

namespace lb {

constexpr int CR_C = 64;                 // tokens a chunk
constexpr int CR_PT = CR_C + 4;          // floats between rows of 64 places: 16-byte pieces of 8 rows lie in all banks
constexpr int CR_THREADS = 512;
constexpr int CR_SCAN = 256, CR_WALK = 256;
constexpr int CR_SEQS = 64;              // sequences a launch

constexpr unsigned long long CR_WAIT_CYCLES = 4000000000ull;     // a bounded wait's limit

// What a launch of lb_chunk_recurrence_wait_test leaves out, so that a wait runs out: the commits of the states' kernel; the copies or the
// products of the wide walk, of the outputs.
enum CrHold : int { CR_HOLD_STATES = 1, CR_HOLD_WALK_COPIES = 2, CR_HOLD_WALK = 4, CR_HOLD_OUT_COPIES = 8, CR_HOLD_OUT = 16 };

enum CrKind : int { CR_FIXED = 0, CR_SSM = 1, CR_DELTA = 2, CR_HGRN2 = 3, CR_CHANNELS = 4 };

__host__ __device__ constexpr bool cr_delta(int kind) { return kind == CR_DELTA || kind == CR_CHANNELS; }
__host__ __device__ constexpr bool cr_rows(int kind) { return kind == CR_HGRN2 || kind == CR_CHANNELS; }   // a decay for every row

struct ChunkParams {
  const float* q; const float* k; const float* v; const float* a; const float* b;    // hgrn2: k is the gate's input
  long long q_ld, k_ld, v_ld, a_ld, b_ld;
  const float* A_log; const float* dt_bias; const float* D; const float* bias; const float* lower; const float* decay;
  float* state; float* out; long long out_ld;
  const int* cu_tokens; const int* slots;
  int heads, groups, dim, vdim, unit_norm, act;
  float q_scale, unit_eps;
  int vec, vecv;                         // rows of q, k, a and rows of v in whole aligned 16-byte pieces
  int slot0;                             // first chunk of this launch, counted over the sequences below
  int num_seqs;
  unsigned long long wait_cycles;        // after this many clock cycles a wait on a barrier gives up
  int hold;                              // tests of the give-up paths only, CrHold
  int wide;                              // delta rules: the walk of chunk_tcgen05.cu, which wants W and K cut
  float* scratch;                        // per (chunk of this launch, head), the arrays at these offsets
  long long per_head;
  // [KD][v_ld_s] K^T U at 0; or W and K [64][KD] in three parts (wide), or W [64][KD + 4] and K^T [KD][68], then U' [64][v_ld_s]; the
  // state before the chunk and U as the outputs' products take them, of a tile of columns after the other (columns behind the last one
  // are not written); the first token whose U is not finite, of every column; c_63
  int off_w, off_k, off_u, off_s, off_up, off_f, off_g, v_ld_s;
  int seq[CR_SEQS];                      // sequence of the step
  int base[CR_SEQS + 1];                 // its first chunk
};

// 1 / d and x / d for d = 1 + e^-x >= 1: the approximate reciprocal (off by 1 ulp) and one step on the remainder (Newton's, and Markstein's for
// the quotient), which leaves half an ulp;
// a d whose reciprocal is no normal number counts as 2^126.
__device__ __forceinline__ float cr_reciprocal(float& d) {
  float r;
  d = fminf(d, 8.5e37f);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  return r;
}
__device__ __forceinline__ float cr_sigmoid(float x) {
  float d = 1.f + expf(-x);
  const float r = cr_reciprocal(d);
  return x != x ? x : fmaf(fmaf(-d, r, 1.f), r, r);
}
__device__ __forceinline__ float cr_silu(float x) {
  float d = 1.f + expf(-x);
  const float r = cr_reciprocal(d), y = x * r;
  return fmaf(fmaf(-y, d, x), r, y);
}

// 1 / sqrt(x) as r + rest: a token's factor errs for the whole row at once.
__device__ __forceinline__ void cr_unit(float x, float scale, float& r, float& rest) {
  r = 1.f / sqrtf(x);
  const float p = r * r;
  rest = 0.5f * r * fmaf(-x, fmaf(r, r, -p), fmaf(-x, p, 1.f));
  rest = fmaf(scale, rest, fmaf(scale, r, -(scale * r)));
  r *= scale;
}
template <typename F>
__device__ __forceinline__ float4 cr_map(float4 x, F f) { return make_float4(f(x.x), f(x.y), f(x.z), f(x.w)); }
// Two numbers (the places that share a register of an operand) as three bfloat16 each, x = h + m + l: rounded to 8 bits, the rest
// rounded to 8, and what is left, which has no more than 8.
struct Split { uint32_t h, m, l; };
__device__ __forceinline__ Split cr_split(float x, float y) {
  Split s;
  s.h = pack_bf16(x, y);
  x -= __uint_as_float(s.h << 16); y -= __uint_as_float(s.h & 0xffff0000u);
  s.m = pack_bf16(x, y);
  x -= __uint_as_float(s.m << 16); y -= __uint_as_float(s.m & 0xffff0000u);
  s.l = pack_bf16(x, y);
  return s;
}

// Whether a value is finite and stays so when it is split.
__device__ __forceinline__ bool cr_finite(float x) { return fabsf(x) <= 3.38e38f; }

struct ChunkPlace { int seq, first, m; };        // sequence, first token, tokens

__device__ __forceinline__ ChunkPlace cr_place(const ChunkParams& p, int at) {
  const int slot = p.slot0 + at;
  int si = 0;
  while (si + 1 < p.num_seqs && p.base[si + 1] <= slot) ++si;
  ChunkPlace c;
  c.seq = p.seq[si];
  c.first = p.cu_tokens[c.seq] + (slot - p.base[si]) * CR_C;
  c.m = min(CR_C, p.cu_tokens[c.seq + 1] - c.first);
  return c;
}

// Decay and write strength of each token, one number a head (decay 1, strength 0 behind the last token).  In 64 bits: a handful of
// values a token while its rows are on their way, and an error here stays in the state as long as the token does.
template <int KIND>
__device__ __forceinline__ void cr_numbers(const ChunkParams& p, const ChunkPlace& c, int h, float* gs, float* ws, int tid) {
  if (tid >= CR_C) return;
  float g = 1.f, w = 0.f;
  if (tid < c.m) {
    w = 1.f;
    if (KIND == CR_FIXED) g = p.decay[h];
    if (KIND == CR_SSM || KIND == CR_DELTA) {
      const double x = (double)p.a[(size_t)(c.first + tid) * p.a_ld + h] + (double)p.dt_bias[h];
      const double sp = x > 20.0 ? x : log1p(exp(x));
      g = (float)exp(-exp((double)p.A_log[h]) * sp);
      w = (float)sp;
    }
    if (cr_delta(KIND)) w = (float)(1.0 / (1.0 + exp(-(double)p.b[(size_t)(c.first + tid) * p.b_ld + h])));
  }
  gs[tid] = g;
  ws[tid] = w;
}

// A product of decays with what its roundings drop: the error of 63 roundings is the same in every chunk of a head whose decay
// does not change, and adds up over a state that lives for thousands of tokens.
struct Product {
  float h = 1.f, l = 0.f;
  __device__ __forceinline__ void times(float g) {
    const float p = h * g;
    l = fmaf(l, g, fmaf(h, g, -p));
    h = p;
  }
  __device__ __forceinline__ float value() const { return h + l; }
};

// G(j, i) at [i][j] for one decay a token (zeros above the diagonal), and c_i: a thread eight rows of a column, from the product
// of the decays between.
__device__ __forceinline__ void cr_products(const float* gs, float* Ds, float* cs, int tid) {
  static_assert(CR_THREADS == 8 * CR_C, "a thread eight rows of a column");
  const int j = tid % CR_C, i0 = tid / CR_C * 8;
  float g[8];
  Product d, c;
#pragma unroll 8
  for (int i = 0; i < i0; ++i) { const float x = gs[i]; if (i > j) d.times(x); }
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] = gs[i0 + i];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i0 + i > j) d.times(g[i]);
    Ds[(i0 + i) * CR_PT + j] = i0 + i >= j ? d.value() : 0.f;
  }
  if (j == 0) {                                    // one thread a block of eight: c_i
#pragma unroll 8
    for (int i = 0; i < i0; ++i) c.times(gs[i]);
#pragma unroll
    for (int i = 0; i < 8; ++i) { c.times(g[i]); cs[i0 + i] = c.value(); }
  }
}

// Byte of (row, column) in one part of an operand of the tensor cores: 64 columns of bfloat16 a row of 128 bytes, swizzled; `rows` rows,
// then the next 64 columns.
__device__ __forceinline__ uint32_t cr_at(int row, int col, int rows) {
  return (uint32_t)((col >> 6) * rows * 128 + row * 128 + (((col & 63) * 2) ^ ((row & 7) << 4)));
}
__host__ __device__ inline int cr_tile(int vdim) { return vdim <= 64 ? 64 : 128; }       // columns a tile
// Where (row d, column v) of the state, (token t, column v) of U lie in the scratch, first part; the parts of a tile are 128 * cr_tile bytes apart.
__device__ __forceinline__ uint8_t* cr_state_at(const ChunkParams& p, float* mine, int kd, int d, int v) {
  const int vt = cr_tile(p.vdim);
  return reinterpret_cast<uint8_t*>(mine + p.off_s) + ((v / vt) * (kd / 64) + d / 64) * 3 * 128 * vt + cr_at(d % 64, v % vt, 64);
}
__device__ __forceinline__ uint8_t* cr_u_at(const ChunkParams& p, float* mine, int t, int v) {
  const int vt = cr_tile(p.vdim);
  return reinterpret_cast<uint8_t*>(mine + p.off_up) + (v / vt) * 3 * 128 * vt + cr_at(t, v % vt, 64);
}
__device__ __forceinline__ void cr_put(uint8_t* at, int part, const Split& x) {
  *reinterpret_cast<uint32_t*>(at) = x.h;
  *reinterpret_cast<uint32_t*>(at + part) = x.m;
  *reinterpret_cast<uint32_t*>(at + 2 * part) = x.l;
}

// SMs of the current device.
inline cudaError_t cr_sms(int* sms) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  return e != cudaSuccess ? e : cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
}

// chunk_tcgen05.cu: the states before the chunks of the delta rules; K^T U of the other kinds; the outputs.
cudaError_t cr_launch_walk(const ChunkParams& p, int nslots, cudaStream_t stream);       // delta rules, `wide`
cudaError_t cr_launch_states(int kind, const ChunkParams& p, int nslots, cudaStream_t stream);
cudaError_t cr_launch_outputs(int kind, const ChunkParams& p, int nslots, cudaStream_t stream);

}  // namespace lb
