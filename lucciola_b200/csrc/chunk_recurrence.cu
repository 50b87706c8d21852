// The linear recurrences of the decoder designs over long portions, 64 tokens at a time (the bfloat16 engine's steps; single
// tokens, short portions and the 32-bit engine stay in the token-by-token kernels of decay_attention.cu, gated_recurrence.cu
// and state_recurrence.cu).  Per head, with a 32-bit state S [dim, vdim]:
//
//   fixed     S_t = d S_(t-1) + k_t v_t^T                              linear attention with a fixed decay
//   ssm       S_t = g_t S_(t-1) + k_t (w_t v_t)^T   (+ D v_t behind)   selective state space
//   hgrn2     S_t = diag(f_t) S_(t-1) + (1 - f_t) v_t^T
//   delta     S' = g_t S_(t-1);  u_t = w_t (v_t - S'^T k_t);  S_t = S' + k_t u_t^T
//   channels  the same with a decay for every row of the state, S' = diag(g_t) S_(t-1)
//   and always  o_t = S_t^T q_t
//
// With S0 the state before a chunk, G(j, i) the product of the decays of tokens j + 1 .. i and c_i = G(-1, i), one set of
// formulas covers all five:
//
//   U = U' - W S0        o = Q S0 + A U        S = diag(c_63) S0 + K^T U
//   Q_i = c_i q_i     K_j = G(j, 63) k_j     A_ij = sum_d q_id k_jd G(j, i)_d   (j <= i)
//   delta:  (1 + L) [U' | W] = [w v | w c k],  L_ij = w_i sum_d k_id k_jd G(j, i)_d (j < i);   else U' = w v, no W
//
// Three launches.  First, every (chunk, head) by itself: K^T U (chunk_states_kernel), or W, U' and K (chunk_solve_kernel) for
// the delta rules.  Then the states before all chunks, which is the only part that goes from chunk to chunk: a sum with decays
// (chunk_scan_kernel), or two small products a chunk (chunk_walk_kernel).  Last, every (chunk, head) by itself again, the
// outputs (chunk_outputs_kernel).  A walk token by token is a chain of 2048 dependent updates for a prompt of 2048 tokens; here
// the chain has 32 links.
//
// Decays never appear as quotients or as exponentials of sums: every G is a running product of factors in [0, 1].  With a
// decay for every row the chunk is cut into blocks of 16: pairs inside a block are formed one by one (their G is carried along
// in registers), pairs of different blocks as (q_i G(block start, i)) . (k_j G(j, block start)).
//
// Infinities and NaN stay where the walk would have them: a bad value of token t reaches no output before t and no other request
// (the two products in which a row meets later tokens, with zeros, take what is not finite out and mark the rows from it on);
// from t on the walk may leave an infinity where a NaN stands here.
//
// Everything is 32-bit.  The products run on the tensor cores as six bfloat16 products of operands cut in three, which hold all 24
// bits, 16 places at a time, and the sums from one 16 to the next are ordinary additions: those of single chunks, and the walk where its
// CTAs run at once, in chunk_tcgen05.cu; here the triangular solve's and the walk in several rounds (see cr_step).  Decays
// and strengths that are one number a token come out of 64 bits, and their products carry what rounding drops.  Against 64 bits the
// outputs before the norm and the states are 0.1 to 0.97 times as far off as those of the kernels that walk token by token, over the layers' sizes
// and operands (rms; HGRN2's outputs, 0.85 to 0.93, were 0.82 to 0.91 while mma.sync formed them: 7.3e-8 -> 7.6e-8 of the result); with fast
// decays and operands of random sign HGRN2's outputs are up to 1.07 times as far off, states of channel decays up to 1.22.
//
// Measured (B200, all launches, token by token | every product by mma.sync | here): HGRN2, one prompt of 2048 tokens and 16 heads of
// 128 x 128, 403 | 147 | 130 us; the delta rule 865 | 214 | 185; fixed decays, four prompts of 1654 tokens in all, 341 | 137 | 84.  Channel decays, 263
// (275 by mma.sync); where 256 to 288 (chunk, head)s stand in more walks than run at once (32 heads, 512 tokens: 134 | 139 us; nine portions of 128,
// 142 | 147) the outputs' second round of CTAs costs them more than their products gain, 1 to 6 %.
// What bounds the kernels here: mma.sync issues one product every 8 cycles a scheduler on this GPU whatever its type, so the six products
// of 16 places are worth 1.3 times the ordinary 32-bit pipes; the walk is 32 links of two small products each.
#include "chunk_recurrence.cuh"

namespace lb {

__device__ __forceinline__ void cr_mma(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Operands of a product over 16 places, split.  The order of the places within a product is free as long as both sides agree: a
// lane's registers hold places q, q + 4 | q + 8, q + 12 (q = lane % 4), which is what 32-bit loads give it.
struct Left { uint32_t h[4], m[4], l[4]; };
struct Right { uint32_t h[2], m[2], l[2]; };
__device__ __forceinline__ void cr_put(Left& a, int i, float x, float y) { const Split s = cr_split(x, y); a.h[i] = s.h; a.m[i] = s.m; a.l[i] = s.l; }
__device__ __forceinline__ void cr_put(Right& b, int i, float x, float y) { const Split s = cr_split(x, y); b.h[i] = s.h; b.m[i] = s.m; b.l[i] = s.l; }

// The 16 x 16 tile of a row-major 32-bit matrix at `tile` (shared address of its first element, `pitch` floats a row).
__device__ __forceinline__ void cr_left(uint32_t tile, int pitch, int lane, Left& a) {
  const uint32_t at = tile + 4 * ((((lane >> 3) & 1) * 8 + (lane & 7)) * pitch + (lane >> 4) * 4);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    uint32_t r[4];
    ldmatrix_x4(at + 32 * i, r[0], r[1], r[2], r[3]);
    cr_put(a, 2 * i, __uint_as_float(r[0]), __uint_as_float(r[2]));
    cr_put(a, 2 * i + 1, __uint_as_float(r[1]), __uint_as_float(r[3]));
  }
}
// A right operand of 8 columns: from [8 columns][16 places] (ldmatrix), from [16 places][8 columns] (plain loads).
__device__ __forceinline__ void cr_right(uint32_t tile, int pitch, int lane, Right& b) {
  uint32_t r[4];
  ldmatrix_x4(tile + 4 * ((lane & 7) * pitch + (lane >> 3) * 4), r[0], r[1], r[2], r[3]);
  cr_put(b, 0, __uint_as_float(r[0]), __uint_as_float(r[1]));
  cr_put(b, 1, __uint_as_float(r[2]), __uint_as_float(r[3]));
}
__device__ __forceinline__ void cr_right_t(const float* tile, int pitch, int lane, Right& b) {
  const float* x = tile + (lane & 3) * pitch + (lane >> 2);
  cr_put(b, 0, x[0], x[4 * pitch]);
  cr_put(b, 1, x[8 * pitch], x[12 * pitch]);
}

// 16 rows times NT tiles of 8 columns over 16 places: the six products of parts that matter (m * l and l * l are below 2^-25 of a
// term), the smallest first, in accumulators of their own; their sum is then added to `acc` rounded to nearest.  The tensor core
// cuts its sums: a chain through its accumulator over all places leaned towards zero and was 1.2 to 6 times as far from 64 bits
// as the kernels that walk token by token.
template <int NT>
__device__ __forceinline__ void cr_step(float (*acc)[4], const Left& a, const Right* b) {
  float t[NT][4] = {}, hh[NT][4] = {};
#pragma unroll
  for (int n = 0; n < NT; ++n) cr_mma(t[n], a.l, b[n].h[0], b[n].h[1]);
#pragma unroll
  for (int n = 0; n < NT; ++n) cr_mma(t[n], a.h, b[n].l[0], b[n].l[1]);
#pragma unroll
  for (int n = 0; n < NT; ++n) cr_mma(t[n], a.m, b[n].m[0], b[n].m[1]);
#pragma unroll
  for (int n = 0; n < NT; ++n) cr_mma(t[n], a.m, b[n].h[0], b[n].h[1]);
#pragma unroll
  for (int n = 0; n < NT; ++n) cr_mma(t[n], a.h, b[n].m[0], b[n].m[1]);
#pragma unroll
  for (int n = 0; n < NT; ++n) cr_mma(hh[n], a.h, b[n].h[0], b[n].h[1]);
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] += hh[n][e] + t[n][e];
}

// 16 rows of `left` times NT n-tiles of `right` (both row-major along the KS * 16 places summed over); two chains of half the
// length, whose roundings are fewer.
template <int KS, int NT>
__device__ __forceinline__ void cr_scores(uint32_t left, uint32_t right, int pitch, int lane, float (*acc)[4]) {
  float even[NT][4] = {};
#pragma unroll 1
  for (int ks = 0; ks < KS; ks += 2) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      Left a;
      Right b[NT];
      cr_left(left + 64 * (ks + u), pitch, lane, a);
#pragma unroll
      for (int t = 0; t < NT; ++t) cr_right(right + 4 * (8 * t * pitch + 16 * (ks + u)), pitch, lane, b[t]);
      cr_step<NT>(u ? acc : even, a, b);
    }
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[t][e] += even[t][e];
}

// The scores of a chunk on and below its diagonal, in 20 tiles of 16 x 8 shared out over the warps, at most two a warp.
// leave(r, n, tile): 16-row tile r, 8-column tile n.
template <int KS, typename F>
__device__ __forceinline__ void cr_triangle(uint32_t left, uint32_t right, int pitch, int warp, int lane, F leave) {
  auto run = [&](int r, int n0, auto count) {
    constexpr int NT = decltype(count)::value;
    float acc[NT][4] = {};
    cr_scores<KS, NT>(left + 4 * 16 * r * pitch, right + 4 * 8 * n0 * pitch, pitch, lane, acc);
#pragma unroll
    for (int t = 0; t < NT; ++t) leave(r, n0 + t, acc[t]);
  };
  struct One { enum { value = 1 }; };
  struct Two { enum { value = 2 }; };
  if (warp < 8) run(3, warp, One());
  else if (warp < 11) run(2, 2 * (warp - 8), Two());
  else if (warp < 13) run(1, 2 * (warp - 11), Two());
  else if (warp < 15) run(0, warp - 13, One());
}

// 64 rows of COLS floats into shared memory by asynchronous copies, PITCH floats apart; rows from m and columns from cols on
// are zeros.
template <int COLS, int PITCH>
__device__ __forceinline__ void cr_fetch(float* dst, const float* src, long long ld, int m, int cols, bool vec, int tid) {
  if (vec) {
    constexpr int STEP = CR_THREADS / (COLS / 4);  // rows between two of a thread's pieces
    const int t0 = tid / (COLS / 4), c = (tid % (COLS / 4)) * 4;
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + t0 * PITCH + c);
    const float* x = src + (size_t)t0 * ld + c;
    const int rows = c < cols ? m - t0 : 0;
#pragma unroll
    for (int i = 0; i < CR_C / STEP; ++i) {
      const bool real = i * STEP < rows;
      cp_async16(d + 4 * i * STEP * PITCH, real ? x : src, real);
      x += (size_t)STEP * ld;
    }
  } else {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int i = tid; i < CR_C * COLS; i += CR_THREADS) {
      const int t = i / COLS, c = i % COLS;
      const bool real = t < m && c < cols;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * (t * PITCH + c)), "l"(real ? src + (size_t)t * ld + c : src),
                   "r"(real ? 4 : 0) : "memory");
    }
  }
}

// The fetched keys to unit length, in place.
template <int KD, int PITCH>
__device__ __forceinline__ void cr_form(const ChunkParams& p, float* Ks, int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  if (!p.unit_norm) return;
#pragma unroll
  for (int t = warp; t < CR_C; t += CR_THREADS / 32) {                    // rows behind the last token are zeros and stay so
    float sk = 0.f, y[KD / 32];
#pragma unroll
    for (int u = 0; u < KD / 32; ++u) {
      y[u] = Ks[t * PITCH + lane + 32 * u];
      sk += y[u] * y[u];
    }
    sk = warp_sum(sk);
    float f, rest;
    cr_unit(sk + p.unit_eps, 1.f, f, rest);
#pragma unroll
    for (int u = 0; u < KD / 32; ++u) Ks[t * PITCH + lane + 32 * u] = fmaf(y[u], f, y[u] * rest);
  }
}

// The decays of 16 tokens from `b0` on, a warp a token and a lane KD / 32 neighbouring channels: requested, then left in Gb [16][PITCH].
template <int KD>
__device__ __forceinline__ void cr_request_decays(const ChunkParams& p, const ChunkPlace& c, int h, int b0, int tid, float* g) {
  const int t = b0 + tid / 32, d0 = (tid % 32) * (KD / 32);
  const float* src = p.a + (size_t)(c.first + t) * p.a_ld + (size_t)h * p.dim + d0;
#pragma unroll
  for (int e = 0; e < KD / 32; ++e) g[e] = 1.f;
  if (t < c.m && p.vec && KD == 128) {
    if (d0 < p.dim) {
      const float4 x = *reinterpret_cast<const float4*>(src);
      g[0] = x.x; g[1] = x.y; g[KD / 32 - 2] = x.z; g[KD / 32 - 1] = x.w;
    }
  } else if (t < c.m) {
#pragma unroll
    for (int e = 0; e < KD / 32; ++e) if (d0 + e < p.dim) g[e] = src[e];
  }
}
template <int KD, int PITCH>
__device__ __forceinline__ void cr_put_decays(int tid, const float* g, float* Gb) {
#pragma unroll
  for (int e = 0; e < KD / 32; ++e) Gb[tid / 32 * PITCH + tid % 32 * (KD / 32) + e] = g[e];
}

// sum_d x_id k_jd G(j, i)_d for one column j and the rows i of its block of 16 from j + 1 on, a warp: a lane takes KD / 32
// neighbouring channels and carries k_j G(j, i); four rows are added up together, in six shuffles.  store(i, sum).
template <int KD, int PITCH, typename F>
__device__ __forceinline__ void cr_pairs(const float* Xs, const float* Ks, const float* Gb, int b0, int j, int lane, F store) {
  const int end = b0 + 16;
  constexpr int N = KD / 32;
  float kk[N];
  auto load = [&](const float* x, float* to) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(to) = *reinterpret_cast<const float4*>(x + 4 * lane);
    else *reinterpret_cast<float2*>(to) = *reinterpret_cast<const float2*>(x + 2 * lane);
  };
  load(Ks + j * PITCH, kk);
  for (int i0 = j + 1; i0 < end; i0 += 4) {
    float s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u;
      s[u] = 0.f;
      if (i < end) {
        float x[N], g[N];
        load(Xs + i * PITCH, x);
        load(Gb + (i - b0) * PITCH, g);
#pragma unroll
        for (int e = 0; e < N; ++e) { kk[e] *= g[e]; s[u] = fmaf(x[e], kk[e], s[u]); }
      }
    }
    const bool high = lane & 16, upper = lane & 8;
    const float x0 = (high ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, high ? s[0] : s[2], 16);
    const float x1 = (high ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, high ? s[1] : s[3], 16);
    float x = (upper ? x1 : x0) + __shfl_xor_sync(0xffffffffu, upper ? x0 : x1, 8);
    x += __shfl_xor_sync(0xffffffffu, x, 4);
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    const int i = i0 + (high ? 2 : 0) + (upper ? 1 : 0);
    if ((lane & 7) == 0 && i < end) store(i, x);
  }
}

// ---- the states before the chunks: S <- diag(c) S + K^T U, element by element --------------------------------------------------
// A thread four neighbouring columns of one row; eight chunks are requested ahead.
__global__ void __launch_bounds__(CR_SCAN) chunk_scan_kernel(const __grid_constant__ ChunkParams p, int nslots, int kd) {
  pdl_trigger();
  const int h = blockIdx.y, seq = p.seq[blockIdx.z], base = p.base[blockIdx.z];
  const int c_lo = max(0, p.slot0 - base), c_hi = min(p.base[blockIdx.z + 1], p.slot0 + nslots) - base;
  const int idx = blockIdx.x * CR_SCAN + threadIdx.x, per = p.v_ld_s / 4;
  pdl_wait();
  if (c_lo >= c_hi || idx >= kd * per) return;
  const int d = idx / per, e = (idx - d * per) * 4;
  float* S = p.state + ((size_t)p.slots[seq] * p.heads + h) * p.dim * p.vdim + (size_t)d * p.vdim + e;
  const int have = d < p.dim ? min(4, p.vdim - e) : 0;           // columns of the state; the rest of the scratch is zeros
  float s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = i < have ? S[i] : 0.f;
  const size_t stride = (size_t)p.heads * p.per_head;
  float* x = p.scratch + ((size_t)(base + c_lo - p.slot0) * p.heads + h) * p.per_head;
  uint8_t* keep = cr_state_at(p, x, kd, d, e);
  const int part = 128 * cr_tile(p.vdim);
  for (int c = c_lo; c < c_hi; c += 8) {
    float4 ds[8];
    float g[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c + i < c_hi) {
        ds[i] = *reinterpret_cast<const float4*>(x + i * stride + (size_t)d * p.v_ld_s + e);
        g[i] = x[i * stride + p.off_g + d];
      }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (c + i < c_hi) {
        const Split lo = cr_split(s[0], s[1]), hi = cr_split(s[2], s[3]);
        uint8_t* to = keep + i * stride * sizeof(float);
        *reinterpret_cast<uint2*>(to) = make_uint2(lo.h, hi.h);
        *reinterpret_cast<uint2*>(to + part) = make_uint2(lo.m, hi.m);
        *reinterpret_cast<uint2*>(to + 2 * part) = make_uint2(lo.l, hi.l);
        s[0] = fmaf(g[i], s[0], ds[i].x); s[1] = fmaf(g[i], s[1], ds[i].y);
        s[2] = fmaf(g[i], s[2], ds[i].z); s[3] = fmaf(g[i], s[3], ds[i].w);
      }
    x += 8 * stride;
    keep += 8 * stride * sizeof(float);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) if (i < have) S[i] = s[i];
}

// ---- every chunk by itself: W, U' and K of the delta rules ----------------------------------------------------------------------
// (1 + L) X = B goes by blocks of 16 rows, X_I = (1 + L_II)^-1 (B_I - sum_(J < I) L_IJ X_J), on the tensor cores: the four inverses
// are formed first (a thread a column), then a warp owns 16 columns of [U' | W] and needs nobody else's.  A thread a column
// down all 64 rows took 2000 dependent multiply-adds, most of this kernel's time.
constexpr int CR_XV = 128;               // value columns at a time
constexpr int CR_PI = 20;                // floats between rows of an inverse

__host__ __device__ constexpr int cr_solve_floats(int kind, int kd) {
  const int mat = CR_C * (kd + 4);
  const int x = CR_C * (CR_XV + 4);
  return mat + 3 * CR_C + CR_C * CR_PT + 64 * CR_PI + (cr_rows(kind) ? (mat > x ? mat : x) + 32 * (kd + 4) + 5 * kd : CR_C * CR_PT + x);
}

template <int KIND, int KD>
__global__ void __launch_bounds__(CR_THREADS, 2) chunk_solve_kernel(const __grid_constant__ ChunkParams p) {
  constexpr int PK = KD + 4, MAT = CR_C * PK, KS = KD / 16;
  constexpr bool ROWS = cr_rows(KIND);
  extern __shared__ __align__(16) float cr_smem[];
  float* Ks = cr_smem;                             // [64][PK]
  float* gs = Ks + MAT;
  float* ws = gs + CR_C;
  float* cs = ws + CR_C;                           // c_i
  float* Ls = cs + CR_C;                           // [64][PT]
  constexpr int PX = CR_XV + 4;
  float* Ti = Ls + CR_C * CR_PT;                   // [4][16][PI]: inverses of the diagonal blocks
  float* Xv = Ti + 64 * CR_PI;                     // [64][PX]: w v, then U'; with a decay for every row it takes the place of Kr
  float* Ds = Xv + CR_C * PX;                      // one decay a token: G(j, i) at [i][j]
  float* Kr = Xv;                                  // a decay for every row: k_j G(j, start of the block at work)
  float* Gb = Kr + (MAT > CR_C * PX ? MAT : CR_C * PX);    // [2][16][PK]: decays of the block at work and of the next
  float* starts = Gb + 32 * PK;                    // [5][KD]: product of the decays before block I; [4]: over the block at work
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, grp = h / (p.heads / p.groups);
  pdl_wait();
  const ChunkPlace c = cr_place(p, blockIdx.x);
  float* mine = p.scratch + ((size_t)blockIdx.x * p.heads + h) * p.per_head;
  float* oW = mine + p.off_w;
  float* oK = mine + p.off_k;
  float* oU = mine + p.off_u;
  float* oG = mine + p.off_g;
  for (int i = tid; i < p.v_ld_s; i += CR_THREADS) reinterpret_cast<int*>(mine)[p.off_f + i] = CR_C;
  cr_fetch<KD, PK>(Ks, p.k + (size_t)c.first * p.k_ld + (size_t)grp * p.dim, p.k_ld, c.m, p.dim, p.vec, tid);
  const float* vsrc = p.v + (size_t)c.first * p.v_ld + (size_t)h * p.vdim;
  if (!ROWS) cr_fetch<CR_XV, PX>(Xv, vsrc, p.v_ld, c.m, min(CR_XV, p.vdim), p.vecv, tid);
  cp_async_commit();
  float gn[KD / 32];
  if (ROWS) cr_request_decays<KD>(p, c, h, 0, tid, gn);
  cr_numbers<KIND>(p, c, h, gs, ws, tid);
  cp_async_wait<0>();
  __syncthreads();
  cr_form<KD, PK>(p, Ks, tid);
  if (ROWS) cr_put_decays<KD, PK>(tid, gn, Gb);
  if (!ROWS) cr_products(gs, Ds, cs, tid);
  __syncthreads();
  const uint32_t Ka = (uint32_t)__cvta_generic_to_shared(Ks);
  // Keys to the state behind the chunk: cut, as the wide walk's products read them, or a row of the state a row.
  const bool wide = KD == 128 && p.wide;
  auto keys_out = [&](const float* K, const float* scale) {
    if (wide) {
      for (int i = tid; i < CR_C * KD / 4; i += CR_THREADS) {
        const int t = i / (KD / 4), d = i % (KD / 4) * 4;
        const float g = scale ? scale[t] : 1.f;
        const float4 x = *reinterpret_cast<const float4*>(K + t * PK + d);
        const Split a = cr_split(x.x * g, x.y * g), b = cr_split(x.z * g, x.w * g);
        uint8_t* to = reinterpret_cast<uint8_t*>(oK) + cr_at(t, d, CR_C);
        *reinterpret_cast<uint2*>(to) = make_uint2(a.h, b.h);
        *reinterpret_cast<uint2*>(to + CR_C * KD * 2) = make_uint2(a.m, b.m);
        *reinterpret_cast<uint2*>(to + 2 * CR_C * KD * 2) = make_uint2(a.l, b.l);
      }
    } else {
      for (int i = warp; i < 2 * (KD / 4); i += CR_THREADS / 32) {
        const int t = (i & 1) * 32 + lane, d = (i >> 1) * 4;
        const float g = scale ? scale[t] : 1.f;
        const float4 x = *reinterpret_cast<const float4*>(K + t * PK + d);
        oK[d * CR_PT + t] = x.x * g; oK[(d + 1) * CR_PT + t] = x.y * g; oK[(d + 2) * CR_PT + t] = x.z * g; oK[(d + 3) * CR_PT + t] = x.w * g;
      }
    }
  };
  if (!ROWS) {
    cr_triangle<KS>(Ka, Ka, PK, warp, lane, [&](int r, int n, const float* s) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 16 * r + (lane >> 2) + (e >> 1) * 8, j = 8 * n + 2 * (lane & 3) + (e & 1);
        Ls[i * CR_PT + j] = j < i ? s[e] * ws[i] * Ds[i * CR_PT + j] : 0.f;
      }
    });
    keys_out(Ks, Ds + (CR_C - 1) * CR_PT);
    if (tid < KD) oG[tid] = cs[CR_C - 1];
  } else {
    const uint32_t Kra = (uint32_t)__cvta_generic_to_shared(Kr);
    float c_start = 1.f;                           // of this thread's channel: product of the decays before the block
    const int ch = tid % KD;
    for (int I = 0; I < 4; ++I) {
      const int b0 = 16 * I;
      float* Gi = Gb + (I & 1) * 16 * PK;
      if (I < 3) cr_request_decays<KD>(p, c, h, b0 + 16, tid, gn);
      const int jj = b0 + warp;                    // pairs inside the block: a warp a column
      cr_pairs<KD, PK>(Ks, Ks, Gi, b0, jj, lane, [&](int i, float x) { Ls[i * CR_PT + jj] = x * ws[i]; });
      if (lane < 16 && b0 + lane <= jj) Ls[(b0 + lane) * CR_PT + jj] = 0.f;
      __syncthreads();                             // the block's rows as they came are read (and the keys before it moved on)
      if (tid < KD) {                              // times c_i from the block's start, in place; times G(i, block's end)
        float g = 1.f, kb[16], gb[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) { kb[i] = Ks[(b0 + i) * PK + ch]; gb[i] = Gi[i * PK + ch]; }
#pragma unroll
        for (int i = 0; i < 16; ++i) { g *= gb[i]; Ks[(b0 + i) * PK + ch] = kb[i] * g; }
        starts[I * KD + ch] = c_start;
        starts[4 * KD + ch] = g;
        c_start *= g;
        if (I == 3) oG[ch] = c_start;
        g = 1.f;
#pragma unroll
        for (int i = 15; i >= 0; --i) { Kr[(b0 + i) * PK + ch] = kb[i] * g; g *= gb[i]; }
      }
      __syncthreads();
      if (I < 3) cr_put_decays<KD, PK>(tid, gn, Gb + (~I & 1) * 16 * PK);
      if (I > 0) {                                 // the block's rows against all tokens before it
        for (int n = warp; n < 2 * I; n += CR_THREADS / 32) {
          float acc[1][4] = {};
          cr_scores<KS, 1>(Ka + 4 * b0 * PK, Kra + 4 * 8 * n * PK, PK, lane, acc);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = b0 + (lane >> 2) + (e >> 1) * 8;
            Ls[i * CR_PT + 8 * n + 2 * (lane & 3) + (e & 1)] = acc[0][e] * ws[i];
          }
        }
      }
      __syncthreads();
      if (I > 0) {
        const float g = starts[4 * KD + ch];
        for (int j = tid / KD; j < b0; j += CR_THREADS / KD) Kr[j * PK + ch] *= g;     // the keys move on to the block's end
      }
    }
    __syncthreads();
    keys_out(Kr, nullptr);
  }
  __syncthreads();                                 // L is complete, the keys are out
  if (ROWS) {
    cr_fetch<CR_XV, PX>(Xv, vsrc, p.v_ld, c.m, min(CR_XV, p.vdim), p.vecv, tid);
    cp_async_commit();
  }
  if (tid < 64) {                                  // column tid % 16 of the inverse of block tid / 16
    const float* L = Ls + (tid & ~15) * (CR_PT + 1);
    const int col = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float y0 = 0.f, y1 = 0.f;
#pragma unroll
      for (int j = 0; j < i; j += 2) {
        y0 = fmaf(L[i * CR_PT + j], x[j], y0);
        if (j + 1 < i) y1 = fmaf(L[i * CR_PT + j + 1], x[j + 1], y1);
      }
      x[i] = (i == col ? 1.f : 0.f) - (y0 + y1);
      Ti[((tid & ~15) + i) * CR_PI + col] = x[i];
    }
  }
  {                                                // w c k, in place
    constexpr int STEP = CR_THREADS / (KD / 4);
#pragma unroll
    for (int i = 0; i < CR_C / STEP; ++i) {
      const int t = tid / (KD / 4) + i * STEP, d = (tid % (KD / 4)) * 4;
      float4* x = reinterpret_cast<float4*>(Ks + t * PK + d);
      const float w = ws[t];
      const float4 g = ROWS ? *reinterpret_cast<const float4*>(starts + (t / 16) * KD + d) : make_float4(cs[t], cs[t], cs[t], cs[t]);
      *x = make_float4(x->x * g.x * w, x->y * g.y * w, x->z * g.z * w, x->w * g.w * w);
    }
  }
  const uint32_t La = (uint32_t)__cvta_generic_to_shared(Ls), Ta = (uint32_t)__cvta_generic_to_shared(Ti);
  // 16 columns of X [64][pitch] (a warp's own; values still without their w), solved in place and written out
  auto solve = [&](float* X, int pitch, float* dst, int ld, bool values, bool stored0, bool stored1) {
    for (int I = 0; I < 4; ++I) {
      float acc[2][4] = {};
      Left a;
      Right b[2];
#pragma unroll 1
      for (int ks = 0; ks < I; ++ks) {
        cr_left(La + 4 * (16 * I * CR_PT + 16 * ks), CR_PT, lane, a);
#pragma unroll
        for (int t = 0; t < 2; ++t) cr_right_t(X + 16 * ks * pitch + 8 * t, pitch, lane, b[t]);
        cr_step<2>(acc, a, b);
      }
      float* mineX = X + (16 * I + (lane >> 2)) * pitch + 2 * (lane & 3);
      bool finite = true;
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float* x = mineX + (e >> 1) * 8 * pitch + 8 * t + (e & 1);
          const float y = fmaf(values ? ws[16 * I + (lane >> 2) + (e >> 1) * 8] : 1.f, *x, -acc[t][e]);
          *x = y;
          acc[t][e] = 0.f;
          finite &= cr_finite(y);
        }
      if (!__all_sync(0xffffffffu, finite)) {      // rare: a column is bad from its first such row on, and no earlier
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int e1 = 0; e1 < 2; ++e1) {
            float* x = mineX + 8 * t + e1;
            const bool upper = !cr_finite(x[0]), lower = !cr_finite(x[8 * pitch]);
            int from = upper ? lane >> 2 : lower ? (lane >> 2) + 8 : 16;
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) from = min(from, __shfl_xor_sync(0xffffffffu, from, d));
            if (upper) x[0] = 0.f;
            if (lower) x[8 * pitch] = 0.f;
            if ((lane >> 2) >= from) acc[t][e1] = __int_as_float(0x7fffffff);
            if ((lane >> 2) + 8 >= from) acc[t][2 + e1] = __int_as_float(0x7fffffff);
          }
      }
      __syncwarp();
      cr_left(Ta + 4 * 16 * I * CR_PI, CR_PI, lane, a);
#pragma unroll
      for (int t = 0; t < 2; ++t) cr_right_t(X + 16 * I * pitch + 8 * t, pitch, lane, b[t]);
      cr_step<2>(acc, a, b);
      __syncwarp();
      float* out = dst + (16 * I + (lane >> 2)) * ld + 2 * (lane & 3);
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
          const float2 x = make_float2(acc[t][2 * e2], acc[t][2 * e2 + 1]);
          *reinterpret_cast<float2*>(mineX + e2 * 8 * pitch + 8 * t) = x;
          if (wide && !values)
            cr_put(reinterpret_cast<uint8_t*>(oW) + cr_at(16 * I + (lane >> 2) + 8 * e2, (int)(dst - oW) + 8 * t + 2 * (lane & 3), CR_C), CR_C * KD * 2, cr_split(x.x, x.y));
          else if (t ? stored1 : stored0) *reinterpret_cast<float2*>(out + e2 * 8 * ld + 8 * t) = x;
        }
      __syncwarp();
    }
  };
  for (int v0 = 0; v0 < p.v_ld_s; v0 += CR_XV) {
    if (v0 > 0) {
      __syncthreads();
      cr_fetch<CR_XV, PX>(Xv, vsrc + v0, p.v_ld, c.m, min(CR_XV, p.vdim - v0), p.vecv, tid);
      cp_async_commit();
    }
    cp_async_wait<0>();
    __syncthreads();                               // the inverses, w c k and the values are in place
    const int left = p.v_ld_s - v0;                // columns still to come, in whole tiles of eight
    if (warp < 8) {
      if (16 * warp < left) solve(Xv + 16 * warp, PX, oU + v0 + 16 * warp, p.v_ld_s, true, true, 16 * warp + 8 < left);
    } else if (v0 == 0 && 16 * (warp - 8) < KD) {
      solve(Ks + 16 * (warp - 8), PK, oW + 16 * (warp - 8), PK, false, true, true);
    }
  }
}

// ---- the states before the chunks of the delta rules: U = U' - W S, S <- diag(c) S + K^T U --------------------------------------
// A CTA for every (NV value columns, head, sequence).  A chunk is two phases: the product with W (16 rows a pair of warps,
// which share out the places summed over) and the one with K^T (16 rows a warp, whose part of the state stays in registers).
// The right operands lie in shared memory already split, the places of a product in the order of the left operands' registers.  W, K^T and U' of the next chunk are under way during both phases.
__host__ __device__ constexpr int cr_walk_floats(int kd, int nv) {
  return 2 * (CR_C * (kd + 4) + kd * CR_PT) + 3 * nv * ((kd + 8) + (CR_C + 8)) / 2 + CR_C * (nv + 8);
}

template <int KD, int NV>
__global__ void __launch_bounds__(CR_WALK) chunk_walk_kernel(const __grid_constant__ ChunkParams p, int nslots) {
  constexpr int PK = KD + 4, NT = NV / 8, MW = KD / 16, WK = CR_C * PK + KD * CR_PT;       // MW warps hold the state, 16 rows each
  extern __shared__ __align__(16) float cr_smem[];
  float* WK_s = cr_smem;                           // [2]: W [64][PK], K^T [KD][PT]
  constexpr int PS = KD + 8, PU = CR_C + 8;        // values between rows of the split operands: 8 rows' pieces lie in all banks
  bf16* Ss = reinterpret_cast<bf16*>(WK_s + 2 * WK);             // [3][NV][PS] state, a column a row, its three parts
  bf16* Us = Ss + 3 * NV * PS;                     // [3][NV][PU]
  float* Y = reinterpret_cast<float*>(Us + 3 * NV * PU);         // [64][NV + 8] the second half of the places' share of W S
  constexpr int PY = NV + 8;
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, seq = p.seq[blockIdx.z], base = p.base[blockIdx.z];
  const int c_lo = max(0, p.slot0 - base), c_hi = min(p.base[blockIdx.z + 1], p.slot0 + nslots) - base;
  const int col0 = blockIdx.x * NV, row = lane >> 2, cc = 2 * (lane & 3);
  pdl_wait();
  if (c_lo >= c_hi) return;
  float* S = p.state + ((size_t)p.slots[seq] * p.heads + h) * p.dim * p.vdim;
  const size_t stride = (size_t)p.heads * p.per_head;
  float* mine = p.scratch + ((size_t)(base + c_lo - p.slot0) * p.heads + h) * p.per_head;
  const uint32_t wk_a = (uint32_t)__cvta_generic_to_shared(WK_s);
  const uint32_t s_a = (uint32_t)__cvta_generic_to_shared(Ss), u_a = (uint32_t)__cvta_generic_to_shared(Us);
  const int r0 = (warp & 3) * 16 + row;            // a pair's token rows
  auto fetch = [&](int buf, const float* src) {    // W and, right behind it, K^T
    const uint32_t dst = wk_a + buf * WK * 4 + 16 * tid;
    const float* x = src + p.off_w + 4 * tid;
#pragma unroll
    for (int i = 0; i < WK / 4 / CR_WALK; ++i) cp_async16(dst + i * 16 * CR_WALK, x + i * 4 * CR_WALK, true);
    constexpr int left = WK / 4 % CR_WALK, done = WK / 4 - left;
    if (tid < left) cp_async16(dst + done * 16, x + done * 4, true);
    cp_async_commit();
  };
  float u_next[NT][4], g_next[2];
  auto request = [&](const float* src) {
    if (warp < 4) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
          const int cl = col0 + nt * 8 + cc;       // v_ld_s is a multiple of eight
          const float2 x = cl < p.v_ld_s ? *reinterpret_cast<const float2*>(src + p.off_u + (r0 + e2 * 8) * p.v_ld_s + cl) : make_float2(0.f, 0.f);
          u_next[nt][2 * e2] = x.x; u_next[nt][2 * e2 + 1] = x.y;
        }
    }
    if (warp < MW) {
      g_next[0] = src[p.off_g + warp * 16 + row];
      g_next[1] = src[p.off_g + warp * 16 + row + 8];
    }
  };
  fetch(0, mine);
  request(mine);

  float s[NT][4];                                  // warps 0 .. MW - 1: the state at (16 warp + row + 8 (e / 2), 8 nt + cc + e % 2)
  // rows (places) r and r + 8 of the columns 8 nt + cc, + 1 of x, split: place q of eight lies at 2 q, place q + 4 behind it
  const int part = 128 * cr_tile(p.vdim);
  int s_off[NT], u_off[NT];                        // bytes from the chunk's scratch to this thread's places of the state and of U
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    s_off[nt] = (int)(cr_state_at(p, mine, KD, warp * 16 + row, col0 + nt * 8 + cc) - reinterpret_cast<uint8_t*>(mine));
    u_off[nt] = (int)(cr_u_at(p, mine, r0, col0 + nt * 8 + cc) - reinterpret_cast<uint8_t*>(mine));
  }
  Split lo, hi;
  auto put_split = [&](bf16* dst, int pitch, int plane, int r, int nt, const float* x) {
    const int at = (nt * 8 + cc) * pitch + (r & ~7) + 2 * (r & 3) + ((r >> 2) & 1);
    lo = cr_split(x[0], x[1]);
    hi = cr_split(x[2], x[3]);
    auto put = [&](bf16* d, uint32_t a, uint32_t b) {
      uint16_t* y = reinterpret_cast<uint16_t*>(d) + at;
      y[0] = (uint16_t)a; y[pitch] = (uint16_t)(a >> 16);
      y[8] = (uint16_t)b; y[pitch + 8] = (uint16_t)(b >> 16);
    };
    put(dst, lo.h, hi.h); put(dst + plane, lo.m, hi.m); put(dst + 2 * plane, lo.l, hi.l);
  };
  auto put_state = [&](float* keep) {              // for the next product, and for the outputs of the chunk it stands before
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      put_split(Ss, PS, NV * PS, warp * 16 + row, nt, s[nt]);
      const int cl = col0 + nt * 8 + cc;
      if (cl < p.v_ld_s) {
        uint8_t* to = reinterpret_cast<uint8_t*>(keep) + s_off[nt];
        cr_put(to, part, lo);
        cr_put(to + 8 * 128, part, hi);
      }
    }
  };
  if (warp < MW) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = warp * 16 + row + (e >> 1) * 8, c = col0 + nt * 8 + cc + (e & 1);
        s[nt][e] = (d < p.dim && c < p.vdim) ? S[(size_t)d * p.vdim + c] : 0.f;
      }
    put_state(mine);
  }
  // 16 rows of `left` times the split right operand [3][NV][rp], over KSTEPS * 16 places
  auto product = [&](uint32_t left, int pitch, uint32_t right, int rp, auto ksteps, float (*acc)[4]) {
#pragma unroll
    for (int ks = 0; ks < decltype(ksteps)::value; ++ks) {
      Left a;
      Right b[NT];
      cr_left(left + 64 * ks, pitch, lane, a);
      auto part = [&](uint32_t plane, auto get) {
        if constexpr (NT == 1) {
          uint32_t* r = get(b[0]);
          asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                       : "=r"(r[0]), "=r"(r[1]) : "r"(plane + 2 * ((lane & 7) * rp + ((lane >> 3) & 1) * 8) + 32 * ks));
        } else {
#pragma unroll
          for (int n2 = 0; n2 < NT / 2; ++n2) {
            uint32_t *r = get(b[2 * n2]), *q = get(b[2 * n2 + 1]);
            ldmatrix_x4(plane + 2 * ((16 * n2 + (lane >> 4) * 8 + (lane & 7)) * rp + ((lane >> 3) & 1) * 8) + 32 * ks, r[0], r[1], q[0], q[1]);
          }
        }
      };
      part(right, [](Right& x) { return x.h; });
      part(right + 2 * NV * rp, [](Right& x) { return x.m; });
      part(right + 4 * NV * rp, [](Right& x) { return x.l; });
      cr_step<NT>(acc, a, b);
    }
  };
  struct HalfK { enum { value = KD / 32 }; };
  struct Tokens { enum { value = CR_C / 16 }; };

  for (int c = c_lo; c < c_hi; ++c) {
    const int buf = (c - c_lo) & 1;
    const uint32_t w_a = wk_a + buf * WK * 4, k_a = w_a + 4 * CR_C * PK;
    float u[NT][4];
    const float gam0 = g_next[0], gam1 = g_next[1];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) u[nt][e] = u_next[nt][e];
    cp_async_wait<0>();
    __syncthreads();                               // W and K have landed, the state is in place, the chunk before is through
    if (c + 1 < c_hi) { fetch(buf ^ 1, mine + stride); request(mine + stride); }
    float y[NT][4] = {};
    const int k0 = (warp >> 2) * (KD / 2);         // this warp's half of the places
    product(w_a + 4 * ((warp & 3) * 16 * PK + k0), PK, s_a + 2 * k0, PS, HalfK(), y);
    if (warp >= 4) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) *reinterpret_cast<float2*>(Y + (r0 + e2 * 8) * PY + nt * 8 + cc) = make_float2(y[nt][2 * e2], y[nt][2 * e2 + 1]);
    }
    __syncthreads();                               // the state is read
    if (warp < 4) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int cl = col0 + nt * 8 + cc;
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
          const float2 z = *reinterpret_cast<const float2*>(Y + (r0 + e2 * 8) * PY + nt * 8 + cc);
          u[nt][2 * e2] -= y[nt][2 * e2] + z.x;
          u[nt][2 * e2 + 1] -= y[nt][2 * e2 + 1] + z.y;
        }
        put_split(Us, PU, NV * PU, r0, nt, u[nt]);
        if (cl < p.v_ld_s) {
          if (!(cr_finite(u[nt][0]) && cr_finite(u[nt][1]) && cr_finite(u[nt][2]) && cr_finite(u[nt][3]))) {
            float x[4];                            // rare: the outputs' product meets it with the zeros of earlier tokens
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              x[e] = cr_finite(u[nt][e]) ? u[nt][e] : 0.f;
              if (!cr_finite(u[nt][e])) atomicMin(reinterpret_cast<int*>(mine) + p.off_f + cl + (e & 1), r0 + 8 * (e >> 1));
            }
            lo = cr_split(x[0], x[1]);
            hi = cr_split(x[2], x[3]);
          }
          uint8_t* to = reinterpret_cast<uint8_t*>(mine) + u_off[nt];
          cr_put(to, part, lo);
          cr_put(to + 8 * 128, part, hi);
        }
      }
    }
    __syncthreads();                               // U is in place
    mine += stride;
    if (warp < MW) {
      float x[NT][4] = {};
      product(k_a + 4 * warp * 16 * CR_PT, CR_PT, u_a, PU, Tokens(), x);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[nt][e] = fmaf(e < 2 ? gam0 : gam1, s[nt][e], x[nt][e]);
      if (c + 1 < c_hi) put_state(mine);
    }
  }
  if (warp < MW) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = warp * 16 + row + (e >> 1) * 8, c = col0 + nt * 8 + cc + (e & 1);
        if (d < p.dim && c < p.vdim) S[(size_t)d * p.vdim + c] = s[nt][e];
      }
  }
}

template <typename K>
static cudaError_t cr_allow(K kernel, int floats) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, floats * (int)sizeof(float));
}

template <int KD, int NV>
static cudaError_t launch_chunk_walk(const ChunkParams& p, int nslots, cudaStream_t stream) {
  constexpr int floats = cr_walk_floats(KD, NV);
  static const cudaError_t cfg = cr_allow(chunk_walk_kernel<KD, NV>, floats);
  if (cfg != cudaSuccess) return cfg;
  return launch(chunk_walk_kernel<KD, NV>, dim3((p.vdim + NV - 1) / NV, p.heads, p.num_seqs), dim3(CR_WALK), floats * sizeof(float), stream, p, nslots);
}

template <int KIND, int KD>
static cudaError_t launch_solve(const ChunkParams& p, int nslots, cudaStream_t stream) {
  constexpr int floats = cr_solve_floats(KIND, KD);
  static const cudaError_t cfg = cr_allow(chunk_solve_kernel<KIND, KD>, floats);
  if (cfg != cudaSuccess) return cfg;
  return launch(chunk_solve_kernel<KIND, KD>, dim3(nslots, p.heads), dim3(CR_THREADS), floats * sizeof(float), stream, p);
}

template <int KD>
static cudaError_t launch_chunks(int kind, const ChunkParams& p, int nslots, cudaStream_t stream) {
  cudaError_t e;
  if (cr_delta(kind)) {
    e = kind == CR_DELTA ? launch_solve<CR_DELTA, KD>(p, nslots, stream) : launch_solve<CR_CHANNELS, KD>(p, nslots, stream);
    if (e != cudaSuccess) return e;
    count_launch();
    if (p.wide) {
      e = cr_launch_walk(p, nslots, stream);
    } else {
      // Fewer columns a CTA where those with 32 leave SMs idle.  Of 128 rows CTAs of 16 columns are always more than there are SMs: with
      // fewer the wide walk runs.
      constexpr int least = KD == 64 ? 8 : 16;
      int nv = 32;
      while (nv > least && (long long)p.num_seqs * p.heads * ((p.vdim + nv - 1) / nv) < 100) nv /= 2;
      if (nv == 32) e = launch_chunk_walk<KD, 32>(p, nslots, stream);
      else if (KD == 128 || nv == 16) e = launch_chunk_walk<KD, 16>(p, nslots, stream);
      else e = launch_chunk_walk<KD, least>(p, nslots, stream);
    }
  } else {
    e = cr_launch_states(kind, p, nslots, stream);
    if (e != cudaSuccess) return e;
    count_launch();
    e = launch(chunk_scan_kernel, dim3((KD * (p.v_ld_s / 4) + CR_SCAN - 1) / CR_SCAN, p.heads, p.num_seqs), dim3(CR_SCAN), 0, stream, p, nslots, KD);
  }
  if (e != cudaSuccess) return e;
  count_launch();
  return cr_launch_outputs(kind, p, nslots, stream);
}

// floats of scratch a (chunk, head); the arrays' offsets, in whole 16-byte pieces
static long long cr_layout(ChunkParams& p, int kind) {
  const int kd = p.dim <= 64 ? 64 : 128, vt = cr_tile(p.vdim), tiles = (p.vdim + vt - 1) / vt;
  p.v_ld_s = (p.vdim + 7) / 8 * 8;
  int at = cr_delta(kind) ? 0 : kd * p.v_ld_s;
  p.off_w = at;
  if (cr_delta(kind)) at += kd == 128 ? CR_C * kd * 3 / 2 : CR_C * (kd + 4);       // of 128 rows: of either walk's form
  p.off_k = at;
  if (cr_delta(kind)) at += kd == 128 ? CR_C * kd * 3 / 2 : kd * CR_PT;
  p.off_u = at;
  if (cr_delta(kind)) at += CR_C * p.v_ld_s;
  p.off_s = at;
  at += tiles * kd * vt * 3 / 2;
  p.off_up = at;
  at += tiles * CR_C * vt * 3 / 2;
  p.off_f = at;
  at += tiles * vt;
  p.off_g = at;
  p.per_head = at + kd;
  return p.per_head;
}

}  // namespace lb

// Floats of scratch that one chunk of 64 tokens takes (all heads); 0: sizes the kernels do not take.
LB_EXPORT long long lb_chunk_recurrence_scratch(int kind, int heads, int dim, int vdim) {
  if (kind < 0 || kind > lb::CR_CHANNELS || heads <= 0 || heads > 65535 || dim <= 0 || dim > 128 || vdim <= 0 || vdim > 4096) return 0;
  lb::ChunkParams p;
  p.dim = dim; p.vdim = vdim;
  return lb::cr_layout(p, kind) * heads;
}

namespace lb {

static int run_chunks(int kind, const float* q, long long q_ld, const float* k, long long k_ld, const float* v, long long v_ld, const float* a,
                      long long a_ld, const float* b, long long b_ld, const float* A_log, const float* dt_bias, const float* D, const float* bias,
                      const float* lower, const float* decay, float* state, float* out, long long out_ld, const int* cu_tokens, const int* slots,
                      const int* seqs, const int* seq_tokens, int num_long, int heads, int groups, int dim, int vdim, int unit_norm, float q_scale,
                      float unit_eps, int act, float* scratch, int scratch_chunks, cudaStream_t stream, int hold, unsigned long long wait_cycles) {
  LB_CHECK_ARG(lb_chunk_recurrence_scratch(kind, heads, dim, vdim) > 0, "chunk_recurrence: kind %d with %d heads of %d x %d", kind, heads, dim, vdim);
  LB_CHECK_ARG(q && k && v && state && out && cu_tokens && slots && seqs && seq_tokens && scratch && scratch_chunks > 0, "chunk_recurrence: null argument");
  LB_CHECK_ARG(groups > 0 && heads % groups == 0, "chunk_recurrence: %d heads are not a multiple of %d groups", heads, groups);
  LB_CHECK_ARG(kind != lb::CR_FIXED || decay, "chunk_recurrence: no decays");
  LB_CHECK_ARG((kind != lb::CR_SSM && kind != lb::CR_DELTA) || (a && A_log && dt_bias), "chunk_recurrence: null argument");
  LB_CHECK_ARG(!lb::cr_delta(kind) || (a && b), "chunk_recurrence: null argument");
  LB_CHECK_ARG(kind != lb::CR_HGRN2 || (bias && lower), "chunk_recurrence: null argument");
  LB_CHECK_ARG(((uintptr_t)scratch & 15) == 0, "chunk_recurrence: scratch is not aligned");
  for (int i = 0; i < num_long; ++i) LB_CHECK_ARG(seq_tokens[i] > 0, "chunk_recurrence: a sequence without tokens");
  lb::ChunkParams p = {};
  p.q = q; p.k = k; p.v = v; p.a = a; p.b = b; p.q_ld = q_ld; p.k_ld = k_ld; p.v_ld = v_ld; p.a_ld = a_ld; p.b_ld = b_ld;
  p.A_log = A_log; p.dt_bias = dt_bias; p.D = D; p.bias = bias; p.lower = lower; p.decay = decay;
  p.state = state; p.out = out; p.out_ld = out_ld; p.cu_tokens = cu_tokens; p.slots = slots;
  p.heads = heads; p.groups = groups; p.dim = dim; p.vdim = vdim; p.unit_norm = unit_norm; p.act = act;
  p.q_scale = q_scale; p.unit_eps = unit_eps; p.scratch = scratch; p.hold = hold; p.wait_cycles = wait_cycles;
  auto aligned = [](const float* x, long long ld) { return (uintptr_t)x % 16 == 0 && ld % 4 == 0; };
  p.vec = dim % 4 == 0 && aligned(q, q_ld) && aligned(k, k_ld) && (kind != lb::CR_CHANNELS || aligned(a, a_ld));
  p.vecv = vdim % 4 == 0 && aligned(v, v_ld);
  lb::cr_layout(p, kind);
  int sms = 0;
  if (cudaError_t e = lb::cr_sms(&sms)) { lb::set_error("chunk_recurrence: %s", cudaGetErrorString(e)); return 2; }
  for (int done = 0; done < num_long;) {
    const int ns = num_long - done < lb::CR_SEQS ? num_long - done : lb::CR_SEQS;
    p.num_seqs = ns;
    // The walk on tcgen05 has a CTA for 16 columns and one CTA an SM: where all of them run at once it is the faster (16 heads of 128 x 128,
    // one prompt of 2048 tokens, 92 -> 68 us), in more than one round the one with 32 columns a CTA is (32 heads, two rounds, 136 | 125).
    p.wide = lb::cr_delta(kind) && dim > 64 && (long long)ns * heads * ((vdim + 15) / 16) <= sms;
    if (!p.wide) p.off_k = p.off_w + lb::CR_C * ((dim <= 64 ? 64 : 128) + 4);      // right behind W: one copy
    else p.off_k = p.off_w + lb::CR_C * 128 * 3 / 2;
    p.base[0] = 0;
    for (int i = 0; i < ns; ++i) {
      p.seq[i] = seqs[done + i];
      p.base[i + 1] = p.base[i] + (seq_tokens[done + i] + lb::CR_C - 1) / lb::CR_C;
    }
    const int total = p.base[ns], turns = (total + scratch_chunks - 1) / scratch_chunks;
    for (int turn = 0; turn < turns; ++turn) {
      const int lo = (int)((long long)total * turn / turns), hi = (int)((long long)total * (turn + 1) / turns);
      p.slot0 = lo;
      const cudaError_t e = dim <= 64 ? lb::launch_chunks<64>(kind, p, hi - lo, stream) : lb::launch_chunks<128>(kind, p, hi - lo, stream);
      if (e != cudaSuccess) { lb::set_error("chunk_recurrence: %s", cudaGetErrorString(e)); return 2; }
      LB_CHECK_LAUNCH("chunk_recurrence");
    }
    done += ns;
  }
  return 0;
}

}  // namespace lb

// The sequences seqs[0 .. num_long - 1] of the step (host array; with seq_tokens[i] tokens each, which must be what cu_tokens
// says), all their tokens.  `scratch` holds scratch_chunks chunks; more are worked off in turns.  fixed: `decay`; ssm: a, A_log,
// dt_bias, D; delta: a, b, A_log, dt_bias; hgrn2: k (the gate's input), bias, lower; channels: a (the decays), b.
LB_EXPORT int lb_chunk_recurrence(int kind, const float* q, long long q_ld, const float* k, long long k_ld, const float* v, long long v_ld,
                                  const float* a, long long a_ld, const float* b, long long b_ld, const float* A_log, const float* dt_bias,
                                  const float* D, const float* bias, const float* lower, const float* decay, float* state, float* out,
                                  long long out_ld, const int* cu_tokens, const int* slots, const int* seqs, const int* seq_tokens,
                                  int num_long, int heads, int groups, int dim, int vdim, int unit_norm, float q_scale, float unit_eps,
                                  int act, float* scratch, int scratch_chunks, cudaStream_t stream) {
  return lb::run_chunks(kind, q, q_ld, k, k_ld, v, v_ld, a, a_ld, b, b_ld, A_log, dt_bias, D, bias, lower, decay, state, out, out_ld, cu_tokens,
                        slots, seqs, seq_tokens, num_long, heads, groups, dim, vdim, unit_norm, q_scale, unit_eps, act, scratch, scratch_chunks,
                        stream, 0, lb::CR_WAIT_CYCLES);
}

// For tests of the give-up paths: the same of at most four chunks, with what `hold` names (CrHold) left out and a wait limit of `wait_cycles`
// clock cycles.  The first wait that depends on it runs out, the roles of each CTA leave once what they have in flight has landed, its code goes to
// the error flag (lb_chunk_device_error), no output and, by the wide walk, no state is stored, and the context stays usable.
LB_EXPORT int lb_chunk_recurrence_wait_test(int kind, const float* q, long long q_ld, const float* k, long long k_ld, const float* v, long long v_ld,
                                            const float* a, long long a_ld, const float* b, long long b_ld, const float* A_log, const float* dt_bias,
                                            const float* D, const float* bias, const float* lower, const float* decay, float* state, float* out,
                                            long long out_ld, const int* cu_tokens, const int* slots, const int* seqs, const int* seq_tokens,
                                            int num_long, int heads, int groups, int dim, int vdim, int unit_norm, float q_scale, float unit_eps,
                                            int act, float* scratch, int scratch_chunks, cudaStream_t stream, int hold,
                                            unsigned long long wait_cycles) {
  LB_CHECK_ARG(hold > 0 && hold < 32 && wait_cycles > 0 && wait_cycles <= lb::CR_WAIT_CYCLES, "chunk_recurrence_wait_test: hold %d, limit %llu", hold, wait_cycles);
  LB_CHECK_ARG(num_long == 1 && seq_tokens && seq_tokens[0] <= lb::CR_C * (scratch_chunks < 4 ? scratch_chunks : 4),
               "chunk_recurrence_wait_test: one sequence of at most four chunks, all of them at once");
  return lb::run_chunks(kind, q, q_ld, k, k_ld, v, v_ld, a, a_ld, b, b_ld, A_log, dt_bias, D, bias, lower, decay, state, out, out_ld, cu_tokens,
                        slots, seqs, seq_tokens, num_long, heads, groups, dim, vdim, unit_norm, q_scale, unit_eps, act, scratch, scratch_chunks,
                        stream, hold, wait_cycles);
}
