// The products of the chunked recurrences that stand by themselves, every (chunk of 64 tokens, head) apart, on the tensor cores
// (chunk_recurrence.cu has the formulas and the walk from chunk to chunk): K^T U of the kinds without the delta rule
// (chunk_states_kernel), and o = Q S0 + A U with A = Q K^T under the decays (chunk_outputs_kernel).
//
// Operands are 32-bit and keep all 24 bits: each is cut into three bfloat16 parts once, on its way into shared memory, and tcgen05.mma forms
// the six products of parts that are not below 2^-25 of a term.  The tensor core cuts its sums, so the products of the largest
// parts are summed over 16 places only, in columns of tensor memory of their own, and the small ones in one sum apart, whose cuts do not
// show; the sums meet in ordinary additions.  Over 128 places of positive numbers, rms against 64 bits: sums of 16 places 5.2e-8 of
// the result, of 32 5.6e-8, of 64 9.0e-8, of 128 1.8e-7, all but the first leaning towards zero by up to as much.  (With the small
// products in the same columns, or sums of 32 places, outputs of positive operands were 1.2 times as far off as with mma.sync.)
//
// The results lie transposed in tensor memory, value columns on the lanes: a warp's 32 lanes then write 128 bytes of a row, and
// both the state and U, [places][columns] in memory, are read as they lie (the "MN-major" form of an operand).  The scan and the walk
// leave the states and U already cut, in the form in which they are read here by one copy a half.
//
// Measured (16 heads of 128 x 128, us, mma.sync with the operands cut by every warp that reads them | here): outputs of 2048 tokens, HGRN2
// 96 | 83, delta rule 78 | 54; of four prompts of 1654 tokens, fixed decays, 79 | 43; K^T U of these 46 | 28, HGRN2 43 | 27; the scan, which cuts
// the states now, 10.5 | 13.6.  One prompt of 160 tokens, 8 heads, fixed decays, all launches: 62 | 25.
// What bounds it: a CTA of the outputs holds 216 KB, so one runs on an SM, and its (chunk, head) takes 10 us: loads of q and k that wait for room
// beside the operands (3 us), their silu or norm and cutting, and the read-out, around 4 us of products.  With a decay for every
// row the pairs inside the blocks and the rows' versions against other blocks come to it (6 us).
#include "attention_tcgen05.cuh"
#include "chunk_recurrence.cuh"

namespace lb {

static_assert(CR_WAIT_CYCLES == TA_WAIT_CYCLES, "one limit for all waits");
constexpr int CT_THREADS = 512;                    // that compute
constexpr int CT_OUT_THREADS = CT_THREADS + 128;   // and, of the outputs, a warp for the products, one for S and U, two for the tokens' numbers
enum CtError : int { CT_ERR_STATES = 401, CT_ERR_OUT = 410, CW_ERR = 450 };      // and the barrier's number
// Barriers of the outputs.  The first ones count an arrival of every warp that computes.
enum CtBar : int {
  CT_READY_QK, CT_READY_Q, CT_READY_A,             // operands are in shared memory
  CT_FREE_A, CT_FREE_S, CT_FREE_T,                 // sums are read: of a part of the scores, of Q S0, of a tile of columns
  CT_FREE_R, CT_FREE_G, CT_FREE_N, CT_FREE_N1,     // 32-bit rows, G(j, i), place and c_i are read
  CT_WARP_BARS,
  CT_SCORES = CT_WARP_BARS, CT_STATES = CT_SCORES + 3, CT_OUT = CT_STATES + 3,           // products are done
  CT_FULL_S, CT_FULL_S1, CT_FULL_U,                // S and U have landed
  CT_READY_G, CT_PLACE, CT_DRAIN = CT_PLACE + 4, CT_BARS
};

__device__ __forceinline__ void ct_put4(uint8_t* dst, int part, float4 x) {
  const Split a = cr_split(x.x, x.y), b = cr_split(x.z, x.w);
  *reinterpret_cast<uint2*>(dst) = make_uint2(a.h, b.h);
  *reinterpret_cast<uint2*>(dst + part) = make_uint2(a.m, b.m);
  *reinterpret_cast<uint2*>(dst + 2 * part) = make_uint2(a.l, b.l);
}
__device__ __forceinline__ void ct_put2(uint8_t* dst, int part, float x, float y) {
  const Split a = cr_split(x, y);
  *reinterpret_cast<uint32_t*>(dst) = a.h;
  *reinterpret_cast<uint32_t*>(dst + part) = a.m;
  *reinterpret_cast<uint32_t*>(dst + 2 * part) = a.l;
}

// D float32, A and B bfloat16, M = m, N = n; a_mn, b_mn: MN-major.
__host__ __device__ constexpr uint32_t ct_idesc(int a_mn, int b_mn, int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// An operand at shared address `at` (first part), parts `part` bytes and 64 places `half` bytes apart; 64-column blocks of `rows` rows.
struct CtOperand { uint32_t at; int part, half, rows, mn; };
__device__ __forceinline__ uint64_t ct_desc(const CtOperand& o, int p, int ks) {           // places 16 ks .. 16 ks + 15
  const uint32_t a = o.at + p * o.part + (ks >> 2) * o.half;
  return o.mn ? ta_desc_mnmajor(a + (ks & 3) * 2048, o.rows * 128) : ta_desc_kmajor(a + (ks & 3) * 32);
}
// Steps ks .. ks + n - 1 of 16 places each: the products of the largest parts in sums of their own, into columns d, d + stride, ..., the small
// ones all in one, behind them.  One thread.
__device__ __forceinline__ void ct_product(uint32_t d, int stride, int ks, int n, const CtOperand& a, const CtOperand& b, uint32_t idesc) {
  const uint32_t small = d + n * stride;
  uint32_t more = 0;
#pragma unroll 1
  for (const int end = ks + n; ks < end; ++ks, d += stride, more = 1) {
    uint64_t A[3], B[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) { A[i] = ct_desc(a, i, ks); B[i] = ct_desc(b, i, ks); }
    ta_umma(small, A[2], B[0], idesc, more);
    ta_umma(small, A[0], B[2], idesc, 1);
    ta_umma(small, A[1], B[1], idesc, 1);
    ta_umma(small, A[1], B[0], idesc, 1);
    ta_umma(small, A[0], B[1], idesc, 1);
    ta_umma(d, A[0], B[0], idesc, 0);
  }
}

// 32 lanes (this warp's quarter) x 8 columns.  The caller waits with ct_wait_ld() before it looks.
__device__ __forceinline__ void ct_ld8(uint32_t at, float* x) {
  uint32_t* r = reinterpret_cast<uint32_t*>(x);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(at) : "memory");
}
// The first 16 lanes of the warp's quarter (all that M = 64 fills) x 16 columns, spread over the warp: x[4 n + e] is lane l / 4 + 8 (e / 2),
// column 8 n + 2 (l % 4) + e % 2.
__device__ __forceinline__ void ct_ld16_half(uint32_t at, float* x) {
  uint32_t* r = reinterpret_cast<uint32_t*>(x);
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(at) : "memory");
}
__device__ __forceinline__ void ct_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// What ct_product has left of STEPS steps, added up: 8 columns (HALF: 16, in ct_ld16_half's form); ADD: to what is there.
template <int STEPS, int STRIDE, bool HALF, bool ADD>
__device__ __forceinline__ void ct_sums8(uint32_t at, float* out) {
  float x[2][8], y[8];
  auto load = [&](int region, float* to) { HALF ? ct_ld16_half(at + STRIDE * region, to) : ct_ld8(at + STRIDE * region, to); };
#pragma unroll
  for (int g = 0; g <= STEPS; g += 2) {
    load(g, x[0]);
    if (g < STEPS) load(g + 1, x[1]);
    ct_wait_ld();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float z = g < STEPS ? x[0][i] + x[1][i] : x[0][i];
      y[i] = g ? y[i] + z : z;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = ADD ? out[i] + y[i] : y[i];
}
// The same of 16 columns: 16 values, or 8 (HALF).
template <int STEPS, int STRIDE, bool HALF, bool ADD = false>
__device__ __forceinline__ void ct_sums(uint32_t at, float* out) {
  ct_sums8<STEPS, STRIDE, HALF, ADD>(at, out);
  if (!HALF) ct_sums8<STEPS, STRIDE, HALF, ADD>(at + 8, out + 8);
}

__device__ __forceinline__ void ct_publish() {       // what this thread wrote into shared memory, to the tensor cores
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// A barrier of `threads` threads that says to all of them whether any came with a value.
__device__ __forceinline__ bool ct_any(int id, int threads, int value) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %3, 0;\n\tbarrier.cta.red.or.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(any) : "r"(id), "r"(threads), "r"(value) : "memory");
  return any != 0;
}
__device__ __forceinline__ void ct_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ct_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
template <int COLS>
__device__ __forceinline__ void ct_alloc(uint32_t slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "n"(COLS) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLS>
__device__ __forceinline__ void ct_free(uint32_t tmem) { asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS)); }

// Contiguous bytes (multiples of 16) into shared memory, counted by a barrier; and out of it.
__device__ __forceinline__ void ct_bulk_in(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void ct_bulk_out(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void ct_bulk_out_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// Four neighbours of a row, zeros where there are none.
__device__ __forceinline__ float4 ct_load4(const float* row, bool real, int c, int cols, bool vec) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (real && c < cols) {
    if (vec) x = *reinterpret_cast<const float4*>(row + c);
    else {
      x.x = row[c];
      if (c + 1 < cols) x.y = row[c + 1];
      if (c + 2 < cols) x.z = row[c + 2];
      if (c + 3 < cols) x.w = row[c + 3];
    }
  }
  return x;
}
// A thread's pieces of 64 rows of COLS floats: four neighbours of rows t0, t0 + STEP, ...
template <int COLS>
struct CtRows {
  static constexpr int LANES = COLS / 4, STEP = CT_THREADS / LANES, N = CR_C / STEP;
  static __device__ __forceinline__ int row(int tid, int i) { return tid / LANES + i * STEP; }
  static __device__ __forceinline__ int col(int tid) { return (tid % LANES) * 4; }
  static __device__ __forceinline__ void load(const float* src, long long ld, int m, int cols, bool vec, int tid, float4* x) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = ct_load4(src + (size_t)row(tid, i) * ld, row(tid, i) < m, col(tid), cols, vec);
  }
  static __device__ __forceinline__ void put(uint8_t* dst, int part, int tid, const float4* x) {
#pragma unroll
    for (int i = 0; i < N; ++i) ct_put4(dst + cr_at(row(tid, i), col(tid), CR_C), part, x[i]);
  }
};
// A row's elements to unit length (its lanes hold four each).
template <int LANES>
__device__ __forceinline__ float4 ct_unit(float4 x, float eps, float scale) {
  float s = (x.x * x.x + x.y * x.y) + (x.z * x.z + x.w * x.w);
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  float f, rest;
  cr_unit(s + eps, scale, f, rest);
  return cr_map(x, [&](float y) { return fmaf(y, f, y * rest); });
}
// hgrn2: the decay from the gate's input.
__device__ __forceinline__ float ct_gate(float x, float low, float bias) { return fmaf(1.f - low, cr_sigmoid(x + bias), low); }

// ---- every chunk by itself: K^T U of the kinds without the delta rule --------------------------------------------------------
// Two CTAs an SM.  Reads k and v (64 KB a chunk and head of 128 x 128), writes 64 KB.  D[v][d]: 64 rows of the state at a time, four sums of
// 16 tokens each.
__host__ __device__ constexpr int ct_states_bytes(int kind, int kd, int vt) {
  return 1024 + 3 * CR_C * (kd + vt) * 2 + 4 * CR_C * 4 + vt * 4 + (cr_rows(kind) ? 8 * kd * 4 : 0);
}

template <int KIND, int KD, int VT>
__global__ void __launch_bounds__(CT_THREADS, 2) chunk_states_kernel(const __grid_constant__ ChunkParams p) {
  constexpr bool ROWS = cr_rows(KIND);
  constexpr int KPART = CR_C * KD * 2, UPART = CR_C * VT * 2;
  extern __shared__ uint8_t ct_raw[];
  __shared__ uint64_t bar_s;
  __shared__ uint32_t tmem_s;
  __shared__ int abort_s;
  uint8_t* Ks = ct_raw + ((1024u - (ta_smem_u32(ct_raw) & 1023u)) & 1023u);      // [3][64 tokens][KD]
  uint8_t* Us = Ks + 3 * KPART;                                                  // [3][64 tokens][VT]
  float* gs = reinterpret_cast<float*>(Us + 3 * UPART);
  float* ws = gs + CR_C;
  float* ts = ws + CR_C;                           // w_j G(j, 63)
  float* cs = ts + CR_C;                           // c_63
  int* from = reinterpret_cast<int*>(cs + CR_C);   // [VT]: first token whose U is not finite
  float* Pg = reinterpret_cast<float*>(from + VT); // [8][KD]: product of the decays of eight tokens
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, grp = h / (p.heads / p.groups);
  const uint32_t bar = ta_smem_u32(&bar_s);
  if (tid == 0) {
    abort_s = 0;
    ta_mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) ct_alloc<256>(ta_smem_u32(&tmem_s));
  if (tid < VT) from[tid] = CR_C;
  pdl_wait();
  const ChunkPlace c = cr_place(p, blockIdx.x);
  float* mine = p.scratch + ((size_t)blockIdx.x * p.heads + h) * p.per_head;
  const float* vsrc = p.v + (size_t)c.first * p.v_ld + (size_t)h * p.vdim;
  const float* ksrc = p.k + (size_t)c.first * p.k_ld + (size_t)grp * p.dim;
  float4 u4[CtRows<VT>::N];
  CtRows<VT>::load(vsrc, p.v_ld, c.m, min(VT, p.vdim), p.vecv, tid, u4);
  auto put_values = [&] {
    bool finite = true;
#pragma unroll
    for (int i = 0; i < CtRows<VT>::N; ++i) {
      if (KIND == CR_FIXED && p.act) u4[i] = cr_map(u4[i], cr_silu);
      finite &= cr_finite(u4[i].x) && cr_finite(u4[i].y) && cr_finite(u4[i].z) && cr_finite(u4[i].w);
    }
    if (!finite) {                                 // rare: the outputs' product meets it with the zeros of earlier tokens
#pragma unroll
      for (int i = 0; i < CtRows<VT>::N; ++i) {
        float* x = reinterpret_cast<float*>(&u4[i]);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (!cr_finite(x[e])) { x[e] = 0.f; atomicMin(&from[CtRows<VT>::col(tid) + e], CtRows<VT>::row(tid, i)); }
      }
    }
    CtRows<VT>::put(Us, UPART, tid, u4);
  };
  if constexpr (!ROWS) {
    float4 k4[CtRows<KD>::N];
    CtRows<KD>::load(ksrc, p.k_ld, c.m, p.dim, p.vec, tid, k4);
    cr_numbers<KIND>(p, c, h, gs, ws, tid);
    __syncthreads();
    put_values();
    if (tid < CR_C) {
      Product d;
#pragma unroll 16
      for (int i = 1; i < CR_C; ++i) { const float x = gs[i]; if (i > tid) d.times(x); }
      ts[tid] = d.value() * ws[tid];
      if (tid == 0) { d.times(gs[0]); cs[0] = d.value(); }
    }
    if (KIND == CR_FIXED && p.act) {
#pragma unroll
      for (int i = 0; i < CtRows<KD>::N; ++i) k4[i] = cr_map(k4[i], cr_silu);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < CtRows<KD>::N; ++i) {
      const float g = ts[CtRows<KD>::row(tid, i)];
      k4[i] = cr_map(k4[i], [&](float x) { return x * g; });
    }
    CtRows<KD>::put(Ks, KPART, tid, k4);
    if (tid < KD) mine[p.off_g + tid] = cs[0];
  } else {
    // a thread two neighbouring channels of eight tokens: k_j G(j, 63) from the last token back
    const int d = (tid % (KD / 2)) * 2, part = tid / (KD / 2);
    float g[8][2];
    if (part < 8) {
      float low[2] = {1.f, 1.f}, bi[2] = {0.f, 0.f};                     // rows beyond dim: decay 1
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (d + e < p.dim) { low[e] = p.lower[h * p.dim + d + e]; bi[e] = p.bias[h * p.dim + d + e]; }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float* x = ksrc + (size_t)(8 * part + i) * p.k_ld + d;
        const bool real = 8 * part + i < c.m;
        if (p.vec && d < p.dim) {
          const float2 y = real ? *reinterpret_cast<const float2*>(x) : make_float2(0.f, 0.f);
          g[i][0] = y.x; g[i][1] = y.y;
        } else {
#pragma unroll
          for (int e = 0; e < 2; ++e) g[i][e] = real && d + e < p.dim ? x[e] : 0.f;
        }
      }
      float all[2] = {1.f, 1.f};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          g[i][e] = 8 * part + i < c.m ? ct_gate(g[i][e], low[e], bi[e]) : 1.f;
          all[e] *= g[i][e];
        }
      *reinterpret_cast<float2*>(Pg + part * KD + d) = make_float2(all[0], all[1]);
    }
    __syncthreads();
    put_values();
    if (part < 8) {
      float2 x = make_float2(1.f, 1.f);
      for (int i = 7; i > part; --i) {
        const float2 y = *reinterpret_cast<const float2*>(Pg + i * KD + d);
        x.x *= y.x; x.y *= y.y;
      }
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        ct_put2(Ks + cr_at(8 * part + i, d, CR_C), KPART, (1.f - g[i][0]) * x.x, (1.f - g[i][1]) * x.y);
        x.x *= g[i][0]; x.y *= g[i][1];
      }
      if (part == 0) { mine[p.off_g + d] = x.x; mine[p.off_g + d + 1] = x.y; }
    }
  }
  ct_publish();
  ct_before_sync();
  __syncthreads();
  ct_after_sync();
  const uint32_t tmem = tmem_s;
  const CtOperand U = {ta_smem_u32(Us), UPART, 0, CR_C, 1};
  const int quad = warp & 3, cols = 16 * (warp >> 2);
  uint32_t parity = 0;
  bool aborted = false;                            // the same in all threads
  for (int v0 = 0; v0 < p.vdim && !aborted; v0 += VT) {
    if (v0 > 0) {
      CtRows<VT>::load(vsrc + v0, p.v_ld, c.m, min(VT, p.vdim - v0), p.vecv, tid, u4);
      if (tid == 0) ct_bulk_out_read();
      if (tid < VT) from[tid] = CR_C;
      __syncthreads();                             // U's copy has left
      put_values();
      ct_publish();
      __syncthreads();
    }
    if (tid == 0) ct_bulk_out(mine + p.off_up + v0 / VT * (3 * UPART / 4), ta_smem_u32(Us), 3 * UPART);
    if (tid < VT) reinterpret_cast<int*>(mine)[p.off_f + v0 + tid] = from[tid];
#pragma unroll 1
    for (int d0 = 0; d0 < KD && !aborted; d0 += 64) {
      float x[16];
#pragma unroll
      for (int ks = 0; ks < 4; ks += 2) {
        if (warp == 0 && elect_one()) {
          const CtOperand K = {ta_smem_u32(Ks) + d0 * 128, KPART, 0, CR_C, 1};   // 64 rows of the state: one block of 64 columns
          ct_product(tmem, 64, ks, 2, U, K, ct_idesc(1, 1, VT, 64));
          if (!(p.hold & CR_HOLD_STATES)) ta_commit(bar);
        }
        __syncwarp();
        ta_mbar_wait(bar, parity, &abort_s, CT_ERR_STATES, p.wait_cycles);
        parity ^= 1;
        ct_after_sync();
        const uint32_t at = tmem + ((uint32_t)(32 * quad) << 16) + cols;
        if (ks == 0) ct_sums<2, 64, VT == 64>(at, x);
        else ct_sums<2, 64, VT == 64, true>(at, x);
        ct_before_sync();
        if (ks == 0) __syncthreads();              // the sums are read
        else aborted = __syncthreads_or(abort_s);  // and whoever gave up, all leave
        ct_after_sync();
      }
      const int cols_left = aborted ? 0 : p.v_ld_s - v0;
      constexpr int N = VT == 64 ? 8 : 16;
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int v = VT == 128 ? 32 * quad + lane : 16 * quad + (lane >> 2) + 8 * ((i >> 1) & 1);
        const int d = VT == 128 ? i : 8 * (i >> 2) + 2 * (lane & 3) + (i & 1);
        if (v < cols_left) mine[(size_t)(d0 + cols + d) * p.v_ld_s + v0 + v] = from[v] < CR_C ? __int_as_float(0x7fffffff) : x[i];
      }
    }
    __syncthreads();                               // from[] is read
  }
  if (tid == 0) ct_bulk_out_read();
  if (aborted) {                                   // the products that were waited for last
    if (warp == 0 && elect_one()) ta_commit(bar);
    __syncwarp();
    ta_mbar_drain(bar, parity ^ 1u);
  }
  if (warp == 0) ct_free<256>(tmem);
}

// sum_d q_id k_jd G(j, i)_d inside the blocks of 16: a warp four columns j of a block, a lane KD / 32 neighbouring channels.  k_j G(j, i) is
// carried along from row to row, so that a row of q and of the decays is read once for all four; the four sums of a row are
// added up over the lanes together.  out[i][j % 16], 17 floats a row; entries above the diagonal are not written.
template <int KD>
__device__ __forceinline__ void ct_pairs(const float* Q, const float* K, const float* G, float* out, int warp, int lane) {
  constexpr int N = KD / 64;                       // pairs of channels
  const int b0 = 16 * (warp >> 2), j0 = 4 * ((warp + (warp >> 2)) & 3);          // long and short columns on every scheduler
  auto load = [&](const float* x, int t, uint64_t* to) {
    x += (b0 + t) * KD + 2 * N * lane;
    if constexpr (N == 2) {
      const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(x);
      to[0] = y.x; to[1] = y.y;
    } else {
      to[0] = *reinterpret_cast<const unsigned long long*>(x);
    }
  };
  uint64_t kk[4][N];
  float s[16];                                     // [row of four][column of four]
  auto row = [&](int i, int r, int columns, bool first) {        // `columns` columns carried on to row i; a new one begins there
    uint64_t q[N], g[N];
    load(Q, i, q);
    if (columns) load(G, i, g);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s[4 * r + u] = 0.f;
      if (u > columns || (u == columns && !first)) continue;
      if (u == columns) load(K, i, kk[u]);
      uint64_t sum = ta_pack2(0.f, 0.f);
#pragma unroll
      for (int e = 0; e < N; ++e) {
        if (u < columns) kk[u][e] = ta_mul2(kk[u][e], g[e]);
        sum = ta_fma2(q[e], kk[u][e], sum);
      }
      float x, y;
      ta_unpack2(sum, x, y);
      s[4 * r + u] = x + y;
    }
  };
  auto leave = [&](int i0) {                       // sixteen sums over the lanes: half of them at each of four exchanges
#pragma unroll
    for (int half = 8, o = 16; half >= 1; half >>= 1, o >>= 1) {
      const bool high = lane & o;
#pragma unroll
      for (int e = 0; e < half; ++e) s[e] = (high ? s[e + half] : s[e]) + __shfl_xor_sync(0xffffffffu, high ? s[e] : s[e + half], o);
    }
    s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
    const int i = i0 + (lane >> 3), j = j0 + ((lane >> 1) & 3);
    if (!(lane & 1) && j <= i) out[(b0 + i) * 17 + j] = s[0];
  };
#pragma unroll
  for (int r = 0; r < 4; ++r) row(j0 + r, r, r, true);
  leave(j0);
#pragma unroll 1
  for (int i0 = j0 + 4; i0 < 16; i0 += 4) {
#pragma unroll
    for (int r = 0; r < 4; ++r) row(i0 + r, r, 4, false);
    leave(i0);
  }
}

// ---- every chunk by itself: the outputs ---------------------------------------------------------------------------------------
// A CTA an SM takes (chunk, head) after (chunk, head).  In shared memory, three parts each: S of VT columns, 64 rows of the state after the
// other; Q; K and then U; A.  A decay for every row: where S comes lie q, k and the decays in 32 bits, for the pairs inside blocks of
// 16 tokens, and where Q and A come, q G(block before, i) of the blocks against the one, two and three blocks before them (96 rows, one
// product with the keys' 48).
template <int KIND, int KD, int VT>
struct CtOut {
  static constexpr bool ROWS = cr_rows(KIND);
  static constexpr int QPART = CR_C * KD * 2, UPART = CR_C * VT * 2, APART = CR_C * CR_C * 2;      // U and 64 rows of S are of one size
  static constexpr int XPART = 96 * KD * 2, KROWS = ROWS ? 48 : CR_C, KPART = KROWS * KD * 2;
  static constexpr int most(int a, int b) { return a > b ? a : b; }
  static constexpr int Q_OFF = most(KD / 64 * 3 * UPART, ROWS ? 3 * CR_C * KD * 4 : 0);            // S lies in front
  static constexpr int A_OFF = Q_OFF + 3 * QPART;
  static constexpr int K_OFF = Q_OFF + most(3 * QPART + 3 * APART, ROWS ? 3 * XPART : 0);
  static constexpr int F_OFF = K_OFF + most(3 * KPART, 3 * UPART);       // 32-bit values
  static constexpr int FLOATS = 4 * CR_C + 8 + (ROWS ? CR_C * 17 + 4 * KD : CR_C * (CR_C + 1) / 2);
  static constexpr int BYTES = 1024 + F_OFF + 4 * FLOATS;
  // M = 128 reads 128 of the 96 rows' parts: the last one's rows end inside the keys' part behind it
  static_assert(!ROWS || Q_OFF + 2 * XPART + (KD / 64 - 1) * 96 * 128 + 128 * 128 <= F_OFF, "rows read beyond the operand lie in shared memory");
};

template <int KIND, int KD, int VT>
__global__ void __launch_bounds__(CT_OUT_THREADS, 1) chunk_outputs_kernel(const __grid_constant__ ChunkParams p, int units) {
  using L = CtOut<KIND, KD, VT>;
  constexpr bool ROWS = L::ROWS;
  using QK = CtRows<KD>;
  constexpr int HALVES = KD / 64;
  // The scores and Q S0 are formed in parts of three steps of 16 places, three and two (or two and two), in columns 0 .. 255 and 256 .. 511 of
  // tensor memory by turns (the last, of 192 columns, at 320): each is read while the next one is formed.  A U takes columns 0 .. 319.
  constexpr int PASSES = HALVES + 1, STEPS = HALVES + 1;
  extern __shared__ uint8_t ct_raw[];
  __shared__ uint64_t bars_s[CT_BARS];
  __shared__ uint32_t tmem_s;
  __shared__ int abort_s;
  uint8_t* base = ct_raw + ((1024u - (ta_smem_u32(ct_raw) & 1023u)) & 1023u);
  uint8_t *Sp = base, *Qp = base + L::Q_OFF, *Ap = base + L::A_OFF, *Kp = base + L::K_OFF;
  float* cs = reinterpret_cast<float*>(base + L::F_OFF);         // [2][64]: c_i of this and of the next
  float* gs = cs + 2 * CR_C;
  float* ws = gs + CR_C;
  int* place = reinterpret_cast<int*>(ws + CR_C);  // [4][2]: first token, tokens
  float* Gs = reinterpret_cast<float*>(place + 8); // one decay a token: G(j, i) (w_j), the rows j <= i one behind the other
  float* Dg = Gs;                                  // a decay for every row: scores inside the blocks [64][17]
  float* Bs = Dg + CR_C * 17;                      // and the products of the blocks' decays [4][KD]
  float *Qf = reinterpret_cast<float*>(Sp), *Kf = Qf + CR_C * KD, *Gf = Kf + CR_C * KD;
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t bar = ta_smem_u32(bars_s);
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < CT_BARS; ++i) ta_mbar_init(bar + 8 * i, i < CT_WARP_BARS ? CT_THREADS / 32 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) ct_alloc<512>(ta_smem_u32(&tmem_s));
  ct_before_sync();
  __syncthreads();
  ct_after_sync();
  const uint32_t tmem = tmem_s;
  pdl_wait();
  // Every barrier advances once a (chunk, head) or a tile of columns; bit b of `phases` is the parity this thread waits for next.
  uint32_t phases = 0;
  // Where one gives up, abort_s is set, and every other wait that is not served gives up as well; a role leaves at the end of the (chunk, head)
  // or tile in which it did, and nothing is stored.
  volatile int* const gave_up = &abort_s;
  bool ok = true;                                  // of the roles that are one thread, or two warps
  auto wait = [&](int b) {
    const bool served = ta_mbar_wait(bar + 8 * b, (phases >> b) & 1u, gave_up, CT_ERR_OUT + b, p.wait_cycles);
    phases ^= 1u << b;
    return served;
  };
  auto wait_idle = [&](int b) {
    ok &= ta_mbar_wait_idle(bar + 8 * b, (phases >> b) & 1u, gave_up, CT_ERR_OUT + b, p.wait_cycles);
    phases ^= 1u << b;
  };

  if (warp == CT_THREADS / 32) {
    // ---- the products, one thread: scores and Q S0 by turns (each one's sums are read while the other's are formed), then A U
    if (elect_one()) {
      const CtOperand oS = {ta_smem_u32(Sp), L::UPART, 3 * L::UPART, 64, 1}, oQ = {ta_smem_u32(Qp), L::QPART, CR_C * 128, CR_C, 0},
                      oU = {ta_smem_u32(Kp), L::UPART, 0, CR_C, 1}, oA = {ta_smem_u32(Ap), L::APART, 0, CR_C, 0},
                      oK = {ta_smem_u32(Kp), L::KPART, L::KROWS * 128, L::KROWS, 0}, oX = {ta_smem_u32(Qp), L::XPART, 96 * 128, 96, 0};
      auto steps = [](int pass) { return pass < PASSES - 1 ? STEPS : 2; };
      auto scores = [&](int pass) {
        if (pass >= 2) ok &= wait(CT_FREE_A);
        ct_after_sync();
        if (ROWS) ct_product(tmem, 48, 0, KD / 16, oX, oK, ct_idesc(0, 0, 128, 48));
        else ct_product(tmem + 256 * (pass & 1), 64, pass * STEPS, steps(pass), oQ, oK, ct_idesc(0, 0, 64, 64));
        ta_commit(bar + 8 * (CT_SCORES + pass));
      };
      auto states = [&](int pass, bool behind_scores) {
        if (pass < HALVES) ok &= wait(CT_FULL_S + pass);
        if (behind_scores || pass >= 2) ok &= wait((PASSES + pass) & 1 ? CT_FREE_S : CT_FREE_A);
        ct_after_sync();
        ct_product(tmem + (pass == PASSES - 1 ? 320 : 256 * ((PASSES + pass) & 1)), 64, pass * STEPS, steps(pass), oS, oQ, ct_idesc(1, 0, VT, 64));
        ta_commit(bar + 8 * (CT_STATES + pass));
      };
      const int have = p.hold & CR_HOLD_OUT ? 0 : units;
      for (int u = blockIdx.x; u < have && ok; u += gridDim.x) {
        ok &= wait(CT_READY_QK);
#pragma unroll 1
        for (int pass = 0; pass < (ROWS ? 1 : PASSES); ++pass) scores(pass);
        if (ROWS) ok &= wait(CT_READY_Q);                // in the place of the scores' operand
        for (int v0 = 0; v0 < p.vdim && ok; v0 += VT) {
          if (v0 > 0) ok &= wait(CT_FREE_T);
#pragma unroll 1
          for (int pass = 0; pass < PASSES; ++pass) states(pass, !ROWS && v0 == 0);
          ok &= wait(CT_FREE_A);
          ok &= wait(CT_FULL_U);
          if (v0 == 0) ok &= wait(CT_READY_A);
          ct_after_sync();
          ct_product(tmem, 64, 0, 4, oU, oA, ct_idesc(1, 0, VT, 64));
          ta_commit(bar + 8 * CT_OUT);
        }
      }
      ta_commit(bar + 8 * CT_DRAIN);               // nobody else may have waited for what was issued last
      ta_mbar_drain(bar + 8 * CT_DRAIN, 0);
    }
    __syncwarp();
  } else if (warp == CT_THREADS / 32 + 1) {
    // ---- S and U, as soon as their places are free, one thread
    if (elect_one()) {
      bool first = true;
      int copies[3] = {};                          // asked for so far: the halves of S, U
      auto copy = [&](int i, uint32_t to, const float* from) {
        ta_mbar_expect_tx(bar + 8 * (CT_FULL_S + i), 3 * L::UPART);
        ct_bulk_in(to, from, 3 * L::UPART, bar + 8 * (CT_FULL_S + i));
        ++copies[i];
      };
      const int have = p.hold & CR_HOLD_OUT_COPIES ? 0 : units;
      for (int u = blockIdx.x; u < have && ok; u += gridDim.x) {
        const float* mine = p.scratch + (size_t)u * p.per_head;
        for (int v0 = 0; v0 < p.vdim && ok; v0 += VT, first = false) {
#pragma unroll
          for (int i = 0; i < HALVES; ++i) {
            if (!first) wait_idle(CT_STATES + PASSES - HALVES + i);
            if (ROWS && v0 == 0 && i == 0) wait_idle(CT_FREE_R);
            if (ok) copy(i, ta_smem_u32(Sp) + i * 3 * L::UPART, mine + p.off_s + (v0 / VT * HALVES + i) * (3 * L::UPART / 4));
          }
          if (!first) wait_idle(CT_OUT);
          if (v0 == 0) wait_idle(CT_SCORES + (ROWS ? 0 : PASSES - 1));
          if (ok) copy(2, ta_smem_u32(Kp), mine + p.off_up + v0 / VT * (3 * L::UPART / 4));
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)                  // nobody leaves while a copy of its own is in flight
        if (copies[i] > 0) ta_mbar_drain(bar + 8 * (CT_FULL_S + i), (copies[i] - 1) & 1);
    }
    __syncwarp();
  } else if (warp >= CT_THREADS / 32 + 2) {
    // ---- places, two (chunk, head)s ahead, and, one decay a token, the decays' products: two warps, a lane a token, then a column
    const int j = tid - CT_THREADS - 64;
    auto put_place = [&](int n) {
      const int u = blockIdx.x + n * gridDim.x;
      if (j != 0 || u >= units) return;
      const ChunkPlace c = cr_place(p, u / p.heads);
      place[2 * (n & 3)] = c.first;
      place[2 * (n & 3) + 1] = c.m;
      ta_mbar_arrive(bar + 8 * (CT_PLACE + (n & 3)));
    };
    put_place(0);
    put_place(1);
    int n = 0;
    for (int u = blockIdx.x; u < units && (!ROWS || ok); u += gridDim.x, ++n) {
      const int buf = n & 1;
      if (n >= 2) wait_idle(CT_FREE_N + buf);      // the one before the one before is through
      put_place(n + 2);
      if (!ROWS) {
        const ChunkPlace c = cr_place(p, u / p.heads);
        cr_numbers<KIND>(p, c, u % p.heads, gs, ws, j);
        if (n >= 1) wait_idle(CT_FREE_G);
        if (ct_any(2, 64, !ok)) break;             // both warps or none
        Product d, all;
        const float w = KIND == CR_SSM ? ws[j] : 1.f;
        float* to = Gs + j;
#pragma unroll 1
        for (int i0 = 0; i0 < CR_C; i0 += 8) {
          float g[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) g[i] = gs[i0 + i];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            all.times(g[i]);
            d.times(i0 + i > j ? g[i] : 1.f);
            if (i0 + i >= j) to[(i0 + i) * (i0 + i + 1) / 2] = d.value() * w;
            if (j == 0) cs[buf * CR_C + i0 + i] = all.value();
          }
        }
        asm volatile("bar.sync 2, 64;" ::: "memory");
        if (j == 0) ta_mbar_arrive(bar + 8 * CT_READY_G);
      }
    }
  } else {
    const int quad = warp & 3, c0 = 16 * (warp >> 2);
    const uint32_t at = tmem + ((uint32_t)(32 * quad) << 16) + c0;
    float4 q4[QK::N], k4[QK::N], g4[KIND == CR_CHANNELS ? QK::N : 1];          // hgrn2: k is 1 - decay, and the decay is what is kept
    auto arrive = [&](int b) {
      __syncwarp();
      if (lane == 0) ta_mbar_arrive(bar + 8 * b);
    };
    auto barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(CT_THREADS) : "memory"); };
    ChunkPlace c = {};
    float4 low, bi;                                // hgrn2's gate
    // q, then k (and the decays) of the next one: no more than fits beside the operands at a time, or the loads wait for one another
    auto request_q = [&](int u, int n) {
      const int grp = u % p.heads / (p.heads / p.groups);
      const bool served = wait(CT_PLACE + (n & 3));
      c.first = served ? place[2 * (n & 3)] : 0;       // without a place no token is read
      c.m = served ? place[2 * (n & 3) + 1] : 0;
      QK::load(p.q + (size_t)c.first * p.q_ld + (size_t)grp * p.dim, p.q_ld, c.m, p.dim, p.vec, tid, q4);
    };
    auto request_k = [&](int u) {
      const int h = u % p.heads, grp = h / (p.heads / p.groups);
      QK::load(p.k + (size_t)c.first * p.k_ld + (size_t)grp * p.dim, p.k_ld, c.m, p.dim, p.vec, tid, k4);
      if constexpr (KIND == CR_CHANNELS) QK::load(p.a + (size_t)c.first * p.a_ld + (size_t)h * p.dim, p.a_ld, c.m, p.dim, p.vec, tid, g4);
      if (KIND == CR_HGRN2) {
        low = ct_load4(p.lower + h * p.dim, true, QK::col(tid), p.dim, false);
        bi = ct_load4(p.bias + h * p.dim, true, QK::col(tid), p.dim, false);
      }
    };
    auto form_q = [&] {                            // as the products take them
#pragma unroll
      for (int i = 0; i < QK::N; ++i) {
        if (KIND == CR_FIXED && p.act) q4[i] = cr_map(q4[i], cr_silu);
        if (cr_delta(KIND) && p.unit_norm) q4[i] = ct_unit<QK::LANES>(q4[i], p.unit_eps, p.q_scale);
        if (KIND == CR_HGRN2) q4[i] = cr_map(q4[i], cr_silu);
      }
    };
    auto form_k = [&] {
      const int have = p.dim - QK::col(tid);       // rows beyond dim: decay 1
#pragma unroll
      for (int i = 0; i < QK::N; ++i) {
        const bool real = QK::row(tid, i) < c.m;
        if (KIND == CR_FIXED && p.act) k4[i] = cr_map(k4[i], cr_silu);
        if (cr_delta(KIND) && p.unit_norm) k4[i] = ct_unit<QK::LANES>(k4[i], p.unit_eps, 1.f);
        float4& g = KIND == CR_HGRN2 ? k4[i] : g4[KIND == CR_CHANNELS ? i : 0];
        if (KIND == CR_HGRN2) g = make_float4(ct_gate(k4[i].x, low.x, bi.x), ct_gate(k4[i].y, low.y, bi.y), ct_gate(k4[i].z, low.z, bi.z), ct_gate(k4[i].w, low.w, bi.w));
        if (ROWS) g = make_float4(real && have > 0 ? g.x : 1.f, real && have > 1 ? g.y : 1.f, real && have > 2 ? g.z : 1.f, real && have > 3 ? g.w : 1.f);
      }
    };
    request_q(blockIdx.x, 0);
    request_k(blockIdx.x);
    form_q();
    form_k();

    int n = 0;
#pragma unroll 1
    for (int u = blockIdx.x; u < units; u += gridDim.x, ++n) {
      const int buf = n & 1;
      const ChunkPlace here = c;
      const bool more = u + (int)gridDim.x < units;
      float o[16];
      if constexpr (!ROWS) {
        if (__any_sync(0xffffffffu, *gave_up)) break;
        QK::put(Qp, L::QPART, tid, q4);
        QK::put(Kp, L::KPART, tid, k4);
        ct_publish();
        ct_before_sync();
        arrive(CT_READY_QK);
        if (more) request_q(u + gridDim.x, n + 1);
        float sc[8], gd[8];
        const int i0 = 16 * quad + (lane >> 2), j0 = c0 + 2 * (lane & 3);        // sc[e]: (i0 + 8 (e / 2 % 2), j0 + 8 (e / 4) + e % 2)
        wait(CT_READY_G);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int i = i0 + 8 * ((e >> 1) & 1), j = j0 + 8 * (e >> 2) + (e & 1);
          gd[e] = j <= i ? Gs[i * (i + 1) / 2 + j] : 0.f;
        }
        arrive(CT_FREE_G);
#pragma unroll
        for (int pass = 0; pass < PASSES; ++pass) {
          wait(CT_SCORES + pass);
          ct_after_sync();
          const uint32_t from = at + 256 * (pass & 1);
          if (pass == 0) ct_sums<STEPS, 64, true>(from, sc);
          else if (pass < PASSES - 1) ct_sums<STEPS, 64, true, true>(from, sc);
          else ct_sums<2, 64, true, true>(from, sc);
          ct_before_sync();
          arrive(pass & 1 ? CT_FREE_S : CT_FREE_A);
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const int i = i0 + 8 * ((e >> 1) & 1), j = j0 + 8 * (e >> 2);
          ct_put2(Ap + cr_at(i, j, CR_C), L::APART, j <= i ? sc[e] * gd[e] : 0.f, j + 1 <= i ? sc[e + 1] * gd[e + 1] : 0.f);
        }
      } else {
        // two channels (ch, ch + 1) of four tokens of block a and four of block 3 - a: q c_i
        float qt[2][4][2], sc[16];
        const int ch = (tid % (KD / 2)) * 2, part = tid / (KD / 2), a = (part >> 2) & 1, t4 = 4 * (part & 3);
#pragma unroll
        for (int i = 0; i < QK::N; ++i) {
          const int at4 = QK::row(tid, i) * KD + QK::col(tid);
          *reinterpret_cast<float4*>(Qf + at4) = q4[i];
          *reinterpret_cast<float4*>(Kf + at4) = KIND == CR_HGRN2 ? cr_map(k4[i], [](float g) { return 1.f - g; }) : k4[i];
          *reinterpret_cast<float4*>(Gf + at4) = KIND == CR_HGRN2 ? k4[i] : g4[KIND == CR_CHANNELS ? i : 0];
        }
        if (ct_any(1, CT_THREADS, *gave_up)) break;              // all warps or none: they meet again below
        // q G(block's start, i), k G(j, block's end)
        if (part < 8) {
          auto of = [&](const float* m, int t) { return *reinterpret_cast<const float2*>(m + t * KD + ch); };
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int I = e ? 3 - a : a, b0 = 16 * I;
            float g[4][2], x[2] = {1.f, 1.f};
#pragma unroll
            for (int i = 0; i < 4; ++i) { const float2 y = of(Gf, b0 + t4 + i); g[i][0] = y.x; g[i][1] = y.y; }
#pragma unroll 4
            for (int i = 0; i < t4; ++i) { const float2 y = of(Gf, b0 + i); x[0] *= y.x; x[1] *= y.y; }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 y = of(Qf, b0 + t4 + i);
              x[0] *= g[i][0]; x[1] *= g[i][1];
              qt[e][i][0] = y.x * x[0]; qt[e][i][1] = y.y * x[1];
              if (I > 0) ct_put2(Qp + cr_at(b0 - 16 + t4 + i, ch, 96), L::XPART, qt[e][i][0], qt[e][i][1]);
            }
            if (t4 == 12) *reinterpret_cast<float2*>(Bs + I * KD + ch) = make_float2(x[0], x[1]);
            if (I < 3) {
              x[0] = x[1] = 1.f;
#pragma unroll 4
              for (int i = 15; i >= t4 + 4; --i) { const float2 y = of(Gf, b0 + i); x[0] *= y.x; x[1] *= y.y; }
#pragma unroll
              for (int i = 3; i >= 0; --i) {
                const float2 y = of(Kf, b0 + t4 + i);
                ct_put2(Kp + cr_at(b0 + t4 + i, ch, 48), L::KPART, y.x * x[0], y.y * x[1]);
                x[0] *= g[i][0]; x[1] *= g[i][1];
              }
            }
          }
        }
        barrier();
        if (part < 8) {                            // against the blocks further back; last, all the way to the chunk's start
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int I = e ? 3 - a : a;
#pragma unroll 1
            for (int J = I - 1; J >= 0; --J) {
              const float2 b = *reinterpret_cast<const float2*>(Bs + J * KD + ch);
              const int row = I == 2 ? 48 : J == 2 ? 64 : 80;    // of (2 | 0), (3 | 1), (3 | 0)
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                qt[e][i][0] *= b.x; qt[e][i][1] *= b.y;
                if (J > 0) ct_put2(Qp + cr_at(row + t4 + i, ch, 96), L::XPART, qt[e][i][0], qt[e][i][1]);
              }
            }
          }
        }
        ct_publish();
        ct_before_sync();
        arrive(CT_READY_QK);
        ct_pairs<KD>(Qf, Kf, Gf, Dg, warp, lane);
        ct_publish();                              // what is read here is overwritten by a copy
        arrive(CT_FREE_R);
        barrier();                                 // the scores inside the blocks are in place
        const bool some = quad < 3 && c0 < 48;
        wait(CT_SCORES);
        ct_after_sync();
        if (some) ct_sums<KD / 16, 48, false>(at, sc);
        if (part < 8) {
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i) ct_put2(Qp + cr_at(16 * (e ? 3 - a : a) + t4 + i, ch, CR_C), L::QPART, qt[e][i][0], qt[e][i][1]);
        }
        ct_publish();
        ct_before_sync();
        arrive(CT_READY_Q);
        if (more) request_q(u + gridDim.x, n + 1);
        if (some) {                                // block I against block J, a lane a token
          const int r = 32 * quad + lane, b = r >> 4, I = b < 3 ? b + 1 : b == 3 ? 2 : 3, J = b < 3 ? b : b == 4 ? 1 : 0;
          if (16 * J == c0) {
#pragma unroll
            for (int e = 0; e < 16; e += 4)
              ct_put4(Ap + cr_at(16 * I + (r & 15), c0 + (e & 8), CR_C) + 2 * (e & 4), L::APART, make_float4(sc[e], sc[e + 1], sc[e + 2], sc[e + 3]));
          }
        }
        if (tid >= CT_THREADS - 4 * CR_C) {        // inside the blocks, and the zeros above
          const int i = (tid - (CT_THREADS - 4 * CR_C)) >> 2, J = tid & 3;
          if (J >= i >> 4) {
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
              float x[4];
#pragma unroll
              for (int f = 0; f < 4; ++f) x[f] = J == i >> 4 && e + f <= (i & 15) ? Dg[i * 17 + e + f] : 0.f;
              ct_put4(Ap + cr_at(i, 16 * J + (e & 8), CR_C) + 2 * (e & 4), L::APART, make_float4(x[0], x[1], x[2], x[3]));
            }
          }
        }
      }
      ct_publish();
      ct_before_sync();
      arrive(CT_READY_A);
      const int h = u % p.heads;
      if (more) request_k(u + gridDim.x);
      // a thread's places of the read-out: columns v (and v + 8), tokens t0 + 0 .. 15, or t0 + 0, 1, 8, 9
      constexpr int N = VT == 64 ? 8 : 16;
      const int v = VT == 128 ? 32 * quad + lane : 16 * quad + (lane >> 2), t0 = VT == 128 ? c0 : c0 + 2 * (lane & 3);
#pragma unroll 1
      for (int v0 = 0; v0 < p.vdim; v0 += VT) {
        const int* from = reinterpret_cast<const int*>(p.scratch + (size_t)u * p.per_head) + p.off_f + v0 + v;
        const int bad0 = from[0], bad1 = VT == 64 ? from[8] : 0;
        const bool last = v0 + VT >= p.vdim;
#pragma unroll
        for (int pass = 0; pass < PASSES - 1; ++pass) {
          if (more && last && pass == 0) form_q();               // while the products run
          wait(CT_STATES + pass);
          ct_after_sync();
          const uint32_t from = at + 256 * ((PASSES + pass) & 1);
          pass ? ct_sums<STEPS, 64, VT == 64, true>(from, o) : ct_sums<STEPS, 64, VT == 64>(from, o);
          ct_before_sync();
          arrive((PASSES + pass) & 1 ? CT_FREE_S : CT_FREE_A);
        }
        if (more && last) form_k();
        wait(CT_STATES + PASSES - 1);
        ct_after_sync();
        ct_sums<2, 64, VT == 64, true>(at + 320, o);
        wait(CT_OUT);
        ct_after_sync();
        const int m = *gave_up ? 0 : here.m;       // whoever it was: nothing is stored
        float* dst = p.out + (size_t)(here.first + t0) * p.out_ld + (size_t)h * p.vdim + v0 + v;
        const float* skip = KIND == CR_SSM ? p.v + (size_t)(here.first + t0) * p.v_ld + (size_t)h * p.vdim + v0 + v : nullptr;
        const float D = KIND == CR_SSM && p.D ? p.D[h] : 0.f;
#pragma unroll
        for (int i0 = 0; i0 < N; i0 += 8) {
          float x[8];
          ct_sums8<4, 64, VT == 64, false>(at + i0, x);
#pragma unroll
          for (int i = i0; i < i0 + 8; ++i) {
            const int dt = VT == 128 ? i : 8 * (i >> 2) + (i & 1), dv = VT == 128 ? 0 : 8 * ((i >> 1) & 1);
            float y = ROWS ? o[i] + x[i - i0] : fmaf(o[i], cs[buf * CR_C + t0 + dt], x[i - i0]);
            if (t0 + dt >= (dv ? bad1 : bad0)) y = __int_as_float(0x7fffffff);
            if (t0 + dt < m && v0 + v + dv < p.vdim) {
              if (KIND == CR_SSM && p.D) y = fmaf(D, skip[dt * p.v_ld + dv], y);
              dst[dt * p.out_ld + dv] = y;
            }
          }
        }
        ct_before_sync();
        if (v0 + VT < p.vdim) arrive(CT_FREE_T);
      }
      arrive(CT_FREE_N + buf);
    }
  }
  __syncthreads();
  if (warp == 0) ct_free<512>(tmem);
}

// ---- the states before the chunks of the delta rules, 128 rows: U = U' - W S, S <- diag(c) S + K^T U -----------------------------
// A CTA for every (16 value columns, head, sequence); the state's 128 x 16 numbers stay in registers, a row's eight columns a thread.  Both
// products of a chunk have W or K^T on the lanes and the three parts of S or U side by side, [h | m | l] of 16 columns each: a product with
// 16 columns takes the tensor cores as long as one with 48 (their left side's 4 KB from shared memory bound both), so three
// products a step of 16 places form all six: W_h [h | m | l], W_m [h | m], W_l h, 8 sums of 16 places apart.  W and K, which the solve
// leaves cut, are copied two chunks deep.  What bounds it is the path from chunk to chunk, 2.1 us (mma.sync, which cut W and K in every CTA, 2.9
// where it leaves the states cut as here): products 0.55 and 0.3 us at their rate, twice the read-out of tensor memory, cutting and handing
// over, and 96 KB a chunk and CTA out of L2, 5.7 TB/s over all CTAs.
constexpr int CW_COLS = 16, CW_THREADS = 256;        // that compute; and a warp for the products and one for the copies
constexpr int CW_PART = CR_C * 128 * 2;              // bytes of a part of W or K
constexpr int CW_STAGE = 6 * CW_PART;                // W, K
constexpr int CW_BYTES = 1024 + 2 * CW_STAGE + 128 * 128 + CR_C * 128;
enum CwBar : int { CW_READY_S, CW_READY_U, CW_WS, CW_KU, CW_FULL_W, CW_FULL_W1, CW_FULL_K, CW_FULL_K1, CW_FREE_W, CW_FREE_W1, CW_FREE_K, CW_FREE_K1, CW_DRAIN, CW_BARS };

// The first 16 lanes of the warp's quarter x 8 columns: x[e] is lane l / 4 + 8 (e / 2), column 2 (l % 4) + e % 2.
__device__ __forceinline__ void ct_ld8_half(uint32_t at, float* x) {
  uint32_t* r = reinterpret_cast<uint32_t*>(x);
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
// Sums of STEPS steps (48 columns each: large | small | small) of N values a step: the large ones pairwise, the small ones behind them.
template <int STEPS, int N, typename F>
__device__ __forceinline__ void cw_sums(uint32_t at, float* out, F load) {
  float x[STEPS][N], y[STEPS][2][N];
#pragma unroll
  for (int k = 0; k < STEPS; ++k) {
    load(at + 48 * k, x[k]);
    load(at + 48 * k + 16, y[k][0]);
    load(at + 48 * k + 32, y[k][1]);
  }
  ct_wait_ld();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float small = 0.f;
#pragma unroll
    for (int k = 0; k < STEPS; ++k) small += y[k][0][i] + y[k][1][i];
#pragma unroll
    for (int n = STEPS / 2; n >= 1; n /= 2)
#pragma unroll
      for (int k = 0; k < n; ++k) x[k][i] += x[k + n][i];
    out[i] = x[0][i] + small;
  }
}

__global__ void __launch_bounds__(CW_THREADS + 64, 1) chunk_walk_wide_kernel(const __grid_constant__ ChunkParams p, int nslots) {
  extern __shared__ uint8_t ct_raw[];
  __shared__ uint64_t bars_s[CW_BARS];
  __shared__ uint32_t tmem_s;
  __shared__ int abort_s;
  uint8_t* base = ct_raw + ((1024u - (ta_smem_u32(ct_raw) & 1023u)) & 1023u);
  uint8_t* Sp = base + 2 * CW_STAGE;                 // [128 rows of the state][3][16 columns], 128 bytes a row
  uint8_t* Up = Sp + 128 * 128;                      // [64 tokens][3][16 columns]
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int h = blockIdx.y, seq = p.seq[blockIdx.z], first = p.base[blockIdx.z];
  const int c_lo = max(0, p.slot0 - first), c_hi = min(p.base[blockIdx.z + 1], p.slot0 + nslots) - first;
  const uint32_t bar = ta_smem_u32(bars_s);
  if (c_lo >= c_hi) return;                          // the whole CTA
  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < CW_BARS; ++i) ta_mbar_init(bar + 8 * i, i <= CW_READY_U ? CW_THREADS / 32 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) ct_alloc<512>(ta_smem_u32(&tmem_s));
  ct_before_sync();
  __syncthreads();
  ct_after_sync();
  const uint32_t tmem = tmem_s;
  pdl_wait();
  const size_t stride = (size_t)p.heads * p.per_head;
  float* mine = p.scratch + ((size_t)(first + c_lo - p.slot0) * p.heads + h) * p.per_head;
  uint32_t phases = 0;                               // parities, as in the outputs; and as there, all leave where one gives up
  bool ok = true;
  auto wait = [&](int b) {
    ok &= ta_mbar_wait(bar + 8 * b, (phases >> b) & 1u, &abort_s, CW_ERR + b, p.wait_cycles);
    phases ^= 1u << b;
  };

  if (warp == CW_THREADS / 32) {
    if (elect_one()) {
      const uint32_t s_at = ta_smem_u32(Sp), u_at = ta_smem_u32(Up);
      auto step = [&](uint32_t d, const CtOperand& left, int ks, uint64_t right, int m) {
        ta_umma(d, ct_desc(left, 0, ks), right, ct_idesc(left.mn, 1, m, 48), 0);
        ta_umma(d + 16, ct_desc(left, 1, ks), right, ct_idesc(left.mn, 1, m, 32), 1);
        ta_umma(d + 32, ct_desc(left, 2, ks), right, ct_idesc(left.mn, 1, m, 16), 1);
      };
      const int end = p.hold & CR_HOLD_WALK ? c_lo : c_hi;
      for (int c = c_lo; c < end && ok; ++c) {
        const int buf = (c - c_lo) & 1;
        const uint32_t w_at = ta_smem_u32(base) + buf * CW_STAGE;
        const CtOperand W = {w_at, CW_PART, CR_C * 128, CR_C, 0}, K = {w_at + 3 * CW_PART, CW_PART, 0, CR_C, 1};
        wait(CW_FULL_W + buf);
        wait(CW_READY_S);
        ct_after_sync();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) step(tmem + 48 * ks, W, ks, ta_desc_mnmajor(s_at + ks * 2048, 128 * 128), 64);
        ta_commit(bar + 8 * CW_WS);
        ta_commit(bar + 8 * (CW_FREE_W + buf));
        wait(CW_FULL_K + buf);
        wait(CW_READY_U);
        ct_after_sync();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) step(tmem + 48 * ks, K, ks, ta_desc_mnmajor(u_at + ks * 2048, CR_C * 128), 128);
        ta_commit(bar + 8 * CW_KU);
        ta_commit(bar + 8 * (CW_FREE_K + buf));
      }
      ta_commit(bar + 8 * CW_DRAIN);
      ta_mbar_drain(bar + 8 * CW_DRAIN, 0);
    }
    __syncwarp();
  } else if (warp == CW_THREADS / 32 + 1) {
    if (elect_one()) {
      const float* from = mine;
      const int end = p.hold & CR_HOLD_WALK_COPIES ? c_lo : c_hi;
      int copies = 0;                                // W and K of chunk c_lo + i are copies 2 i and 2 i + 1
      for (int c = c_lo; c < end; ++c, from += stride) {
        const int buf = (c - c_lo) & 1;
        const uint32_t to = ta_smem_u32(base) + buf * CW_STAGE;
        if (c >= c_lo + 2) wait(CW_FREE_W + buf);
        if (!ok) break;
        ta_mbar_expect_tx(bar + 8 * (CW_FULL_W + buf), 3 * CW_PART);
        ct_bulk_in(to, from + p.off_w, 3 * CW_PART, bar + 8 * (CW_FULL_W + buf));
        ++copies;
        if (c >= c_lo + 2) wait(CW_FREE_K + buf);
        if (!ok) break;
        ta_mbar_expect_tx(bar + 8 * (CW_FULL_K + buf), 3 * CW_PART);
        ct_bulk_in(to + 3 * CW_PART, from + p.off_k, 3 * CW_PART, bar + 8 * (CW_FULL_K + buf));
        ++copies;
      }
      for (int i = max(0, copies - 4); i < copies; ++i)         // the last four may still be in flight
        ta_mbar_drain(bar + 8 * ((i & 1 ? CW_FULL_K : CW_FULL_W) + ((i >> 1) & 1)), (i >> 2) & 1);
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, hf = (warp >> 2) * 8;             // 32 rows of the state or 16 tokens; eight columns
    const int col0 = blockIdx.x * CW_COLS + hf;
    const uint32_t at = tmem + ((uint32_t)(32 * quad) << 16) + hf;
    const int part = 128 * cr_tile(p.vdim);
    const int d = 32 * quad + lane, t = 16 * quad + (lane >> 2), cc = 2 * (lane & 3);
    const bool there = col0 < p.v_ld_s;                          // a multiple of eight
    const int s_off = there ? (int)(cr_state_at(p, mine, 128, d, col0) - reinterpret_cast<uint8_t*>(mine)) : 0;
    const int u_off = there ? (int)(cr_u_at(p, mine, t, col0 + cc) - reinterpret_cast<uint8_t*>(mine)) : 0;
    auto arrive = [&](int b) {
      ct_publish();
      ct_before_sync();
      __syncwarp();
      if (lane == 0) ta_mbar_arrive(bar + 8 * b);
    };
    float s[8], g = 1.f;
    float2 u_next[2];
    auto request = [&](const float* src) {                       // U' and the row's decay over the chunk
#pragma unroll
      for (int e = 0; e < 2; ++e)
        u_next[e] = there ? *reinterpret_cast<const float2*>(src + p.off_u + (t + 8 * e) * p.v_ld_s + col0 + cc) : make_float2(0.f, 0.f);
      g = src[p.off_g + d];
    };
    auto put_state = [&](float* keep) {              // for the next product, and for the outputs of the chunk it stands before
      Split x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = cr_split(s[2 * i], s[2 * i + 1]);
      const uint4 hi = make_uint4(x[0].h, x[1].h, x[2].h, x[3].h), mi = make_uint4(x[0].m, x[1].m, x[2].m, x[3].m), lo = make_uint4(x[0].l, x[1].l, x[2].l, x[3].l);
      *reinterpret_cast<uint4*>(Sp + cr_at(d, hf, 128)) = hi;
      *reinterpret_cast<uint4*>(Sp + cr_at(d, 16 + hf, 128)) = mi;
      *reinterpret_cast<uint4*>(Sp + cr_at(d, 32 + hf, 128)) = lo;
      arrive(CW_READY_S);
      if (there) {
        uint8_t* to = reinterpret_cast<uint8_t*>(keep) + s_off;
        *reinterpret_cast<uint4*>(to) = hi;
        *reinterpret_cast<uint4*>(to + part) = mi;
        *reinterpret_cast<uint4*>(to + 2 * part) = lo;
      }
    };
    float* S = p.state + ((size_t)p.slots[seq] * p.heads + h) * p.dim * p.vdim + (size_t)d * p.vdim + col0;
    const int have = d < p.dim ? min(8, p.vdim - col0) : 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] = i < have ? S[i] : 0.f;
    put_state(mine);
    request(mine);
    for (int c = c_lo; c < c_hi && __all_sync(0xffffffffu, ok); ++c) {
      const float2 u0 = u_next[0], u1 = u_next[1];
      const float decay = g;
      float* const keep = mine;
      mine += stride;
      if (c + 1 < c_hi) request(mine);
      wait(CW_WS);
      ct_after_sync();
      float y[4];
      cw_sums<8, 4>(at, y, [](uint32_t a, float* x) { ct_ld8_half(a, x); });
      y[0] = u0.x - y[0]; y[1] = u0.y - y[1]; y[2] = u1.x - y[2]; y[3] = u1.y - y[3];
      Split a = cr_split(y[0], y[1]), b = cr_split(y[2], y[3]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const Split& x = e ? b : a;
        *reinterpret_cast<uint32_t*>(Up + cr_at(t + 8 * e, hf + cc, CR_C)) = x.h;
        *reinterpret_cast<uint32_t*>(Up + cr_at(t + 8 * e, 16 + hf + cc, CR_C)) = x.m;
        *reinterpret_cast<uint32_t*>(Up + cr_at(t + 8 * e, 32 + hf + cc, CR_C)) = x.l;
      }
      arrive(CW_READY_U);
      if (there) {
        if (!(cr_finite(y[0]) && cr_finite(y[1]) && cr_finite(y[2]) && cr_finite(y[3]))) {      // rare: the outputs' product meets it with the zeros of earlier tokens
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (!cr_finite(y[e])) { atomicMin(reinterpret_cast<int*>(keep) + p.off_f + col0 + cc + (e & 1), t + 8 * (e >> 1)); y[e] = 0.f; }
          a = cr_split(y[0], y[1]);
          b = cr_split(y[2], y[3]);
        }
        uint8_t* to = reinterpret_cast<uint8_t*>(keep) + u_off;
        cr_put(to, part, a);
        cr_put(to + 8 * 128, part, b);
      }
      wait(CW_KU);
      ct_after_sync();
      float x[8];
      cw_sums<4, 8>(at, x, [](uint32_t a, float* z) { ct_ld8(a, z); });
#pragma unroll
      for (int i = 0; i < 8; ++i) s[i] = fmaf(decay, s[i], x[i]);
      if (c + 1 < c_hi) put_state(mine);
    }
    const int keep = *(volatile int*)&abort_s ? 0 : have;              // whoever gave up: the request's state stays as it was
#pragma unroll
    for (int i = 0; i < 8; ++i) if (i < keep) S[i] = s[i];
  }
  ct_before_sync();
  __syncthreads();
  ct_after_sync();
  if (warp == 0) ct_free<512>(tmem);
}

template <typename K>
static cudaError_t ct_allow(K kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }

template <int KIND, int KD, int VT>
static cudaError_t launch_states(const ChunkParams& p, int nslots, cudaStream_t stream) {
  constexpr int bytes = ct_states_bytes(KIND, KD, VT);
  static const cudaError_t cfg = ct_allow(chunk_states_kernel<KIND, KD, VT>, bytes);
  if (cfg != cudaSuccess) return cfg;
  return launch(chunk_states_kernel<KIND, KD, VT>, dim3(nslots, p.heads), dim3(CT_THREADS), bytes, stream, p);
}
template <int KIND, int KD, int VT>
static cudaError_t launch_outputs(const ChunkParams& p, int nslots, cudaStream_t stream) {
  constexpr int bytes = CtOut<KIND, KD, VT>::BYTES;
  static const cudaError_t cfg = ct_allow(chunk_outputs_kernel<KIND, KD, VT>, bytes);
  if (cfg != cudaSuccess) return cfg;
  int sms = 0;
  if (cudaError_t e = cr_sms(&sms)) return e;
  const int units = nslots * p.heads;
  return launch(chunk_outputs_kernel<KIND, KD, VT>, dim3(units < sms ? units : sms), dim3(CT_OUT_THREADS), bytes, stream, p, units);
}

cudaError_t cr_launch_walk(const ChunkParams& p, int nslots, cudaStream_t stream) {
  static const cudaError_t cfg = ct_allow(chunk_walk_wide_kernel, CW_BYTES);
  if (cfg != cudaSuccess) return cfg;
  return launch(chunk_walk_wide_kernel, dim3((p.vdim + CW_COLS - 1) / CW_COLS, p.heads, p.num_seqs), dim3(CW_THREADS + 64), CW_BYTES, stream, p, nslots);
}

// Value columns up to 64 take tiles of 64, more than that of 128.
#define CT_SIZES(KIND, F)                                                                                        \
  (p.dim <= 64 ? (p.vdim <= 64 ? F<KIND, 64, 64>(p, nslots, stream) : F<KIND, 64, 128>(p, nslots, stream))       \
               : (p.vdim <= 64 ? F<KIND, 128, 64>(p, nslots, stream) : F<KIND, 128, 128>(p, nslots, stream)))

cudaError_t cr_launch_states(int kind, const ChunkParams& p, int nslots, cudaStream_t stream) {
  switch (kind) {
    case CR_FIXED: return CT_SIZES(CR_FIXED, launch_states);
    case CR_SSM: return CT_SIZES(CR_SSM, launch_states);
    case CR_HGRN2: return CT_SIZES(CR_HGRN2, launch_states);
    default: return cudaErrorInvalidValue;         // the delta rules' states come from a walk
  }
}
cudaError_t cr_launch_outputs(int kind, const ChunkParams& p, int nslots, cudaStream_t stream) {
  switch (kind) {
    case CR_FIXED: return CT_SIZES(CR_FIXED, launch_outputs);
    case CR_SSM: return CT_SIZES(CR_SSM, launch_outputs);
    case CR_DELTA: return CT_SIZES(CR_DELTA, launch_outputs);
    case CR_HGRN2: return CT_SIZES(CR_HGRN2, launch_outputs);
    case CR_CHANNELS: return CT_SIZES(CR_CHANNELS, launch_outputs);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace lb

// Code that a kernel of this file left when one of its bounded waits gave up (0: none), and clears it.
LB_EXPORT int lb_chunk_device_error() {
  int v = 0;
  const int zero = 0;
  if (cudaMemcpyFromSymbol(&v, lb::g_attention_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(lb::g_attention_tc_error, &zero, sizeof(int));
  return v;
}
