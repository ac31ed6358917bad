// The recurrences of linrec_segments.cu over prompts, in chunks of 128 tokens on the fifth-generation tensor cores, in 32-bit
// accuracy.
//
//   S_t = keep_t S_(t-1) + take_t k_t v_t^T        modes 0 (state space) and 1 (matrix memory): one number per head and token
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T             mode 3 (gated linear attention): a number per row
//
// Mode 2 (forget and write) stays with the segments: the error of its outputs against 64 bits was 1.2e-7 to 1.3e-7 here and 0.9e-7 to 1.0e-7 there
// (ordinary gates), and write gates near 1 took the blocks below one by one (512 tokens of 16 heads, 374 us against 68).
//
// With w(t, s) the decay from token s to token t (times what s takes) and w(t) that from the chunk's start S_0,
//   o_t = w(t) q_t^T S_0 + sum over s <= t of w(t, s) (q_t . k_s) v_s        S_128 = w(128) S_0 + sum over s of w(128, s) k_s v_s^T
// which are products of 128 x 128 x 128.  The chunks' sums do not depend on one another; only S_0 does:
//   1. lc_gates_kernel (modes 0, 1): the logarithms of the decays since the chunk's start, their sum in 64 bits, kept as two floats;
//   2. lc_ends_kernel: a block per chunk and head, U = sum over s of w(128, s) k_s v_s^T;
//   3. lc_scan_kernel: a thread per four numbers of the state, from chunk to chunk, leaves every chunk its S_0 where U was;
//   4. lc_out_kernel: a block per chunk and head: P^T = K Q^T, weights and mask on P^T as it comes from tensor memory, then
//      O^T = S_0^T Q^T and V^T P^T.
// Each 32-bit operand is split into three bfloat16 parts (as in gemm_f32_tc.cu) which stand in shared memory as [row][128] planes of 128-byte
// swizzled halves; whether a product reads them along the rows or across is a bit of its descriptors, so nothing is transposed.  Of
// the nine products of parts the six largest are formed, the small ones first.
//
// Mode 3: w(t, s) differs from row to row of the state, so it has to be in the operands: q_t b_t and k_s / b_s with b the
// product of the decays since a reference, the chunk's start while no row's decays multiply to less than LC_SMALL there.  Else
// blocks of 64 or 32 tokens take their own starts: for the queries of block j, keys of the blocks before it are multiplied by decays
// up to the start of j (at most 1), those of j itself divided by theirs; and the weights of a block of 32 that is still out of range
// are formed one by one in 32 bits.  Products of decays near 1 are carried by what they lack to 1 (lr_decay), as in linrec_segments.cu.
//
// What bounds it: none of the tensor cores (active for 12 to 15 % of lc_ends_kernel's and lc_out_kernel's time), memory (384 KB a block, 15 to 20 %
// of the DRAM rate) or issue slots (32 to 40 % used) alone, but one block an SM whose phases (rows in, parts, products, weights, rows
// out) follow one another.  Straight-line code is fetched once a block: with the products' loop unrolled the same block took 10 to 15 %
// longer.  Rows by bulk copies instead of loads into registers, and calls instead of inlined splits, changed nothing.
// Measured, 2,048 tokens of 16 heads of 128 x 128, the recurrence alone, us, segments first: gated linear attention 176 and 102, matrix memory 183
// and 96, state space 155 and 84.
//
// A value that is not finite would reach earlier tokens of its chunk through products with weights of 0: it is left out of
// the products, and its column is NaN from its token on.
#include "attention_tc.cuh"
#include "linrec.cuh"
#include "portions.cuh"

#define LC_T 128                       // tokens of a chunk, and the most rows and columns of a state
#define LC_THREADS 512
#define LC_PART 32768                  // bytes of one part of an operand: two halves of 128 rows x 64 columns
#define LC_HALF 16384
#define LC_PLANE (3 * LC_PART)
#define LC_SMALL 0x1p-90f             // the third part of a number of this size keeps its bits (2^-110 is the least)

struct LcArgs {
  const float* q; long q_stride;                     // [T][qk_heads * N]
  const float* k; long k_stride;                     // [T][qk_heads * N]
  const float* v; long v_stride;                     // [T][H * dv]
  const float* a; long a_stride;                     // mode 3: [T][qk_heads * N] decays
  const float* d_skip;                               // mode 0: [H]
  float q_scale;
  const int* cu_tokens;
  const int* state_slots;
  float* state; long state_stride; int num_slots;
  float* out; long out_stride;                       // [T][H * dv]; mode 1: before the division
  float* den;                                        // mode 1: [T][H], what the outputs are to be divided by
  float* gates;                                      // planes [T][H], see lc_gates_kernel
  float* ends;                                       // [chunks][H][N * dv]: U, then S_0
  float* vecs;                                       // [chunks][H][N]: mode 1 the sum of keys, then n at the start; mode 3 the rows' decay (lr_code)
  float* scale;                                      // [chunks][H][4]: the chunk's F (high, low); mode 1 also F + M
  int T, S, H, qk_heads, N, dv, chunks;
  int* err;
};

// ---------------------------------------------------------------- operands in shared memory
__device__ __forceinline__ unsigned char* lc_at(unsigned char* plane, int row, int col) {      // col even
  return plane + (col >> 6) * LC_HALF + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4) + (col & 7) * 2;
}
__device__ __forceinline__ void lc_put2(unsigned char* plane, int row, int col, float x, float y) {
  uint32_t p[3];
  at_split2(x, y, p[0], p[1], p[2]);
  unsigned char* d = lc_at(plane, row, col);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(d + i * LC_PART) = p[i];
}
__device__ __forceinline__ void lc_put4(unsigned char* plane, int row, int col, const float4& v) {
  uint2 p[3];
  at_split2(v.x, v.y, p[0].x, p[1].x, p[2].x);
  at_split2(v.z, v.w, p[0].y, p[1].y, p[2].y);
  unsigned char* d = lc_at(plane, row, col);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(d + i * LC_PART) = p[i];
}
// D = A B over 128 of K.  An operand is K-major (a row for every M or N) or MN-major (a row for every K).
// The tensor cores truncate what they add to an accumulator, so each 32 of K have one of their own, 128 columns apart: two large
// products each instead of eight in a row, and the four are added up in registers, rounded (lc_sum32).  Error of the outputs against 64
// bits, 777 tokens of 128 x 128, one accumulator, four, and the segments: row decays near 1 2.5e-7, 1.5e-7, 2.3e-7, ordinary ones 2.0e-7, 1.5e-7,
// 1.4e-7 (their state 8.1e-8, 8.4e-8, 1.2e-7); state space 9.6e-8, 6.8e-8, 4.4e-7.  It takes 1.5 % of a mixer's step (2,048 tokens, row decays, 221 ->
// 225 us).  What the operands' products lost to rounding, carried in the third parts, gave 1 to 3 % of the error for 1 to 5 % of the step: not kept.
template <bool A_MN, bool B_MN>
__device__ __forceinline__ void lc_product(uint32_t d, uint32_t a, uint32_t b, int n) {
  const uint32_t idesc = tc_idesc(128, n) | (A_MN ? 1u << 15 : 0u) | (B_MN ? TC_IDESC_B_MN : 0u);
  const uint64_t a0 = A_MN ? tc_desc_mn(a, LC_HALF, 1024) : tc_desc(a), b0 = B_MN ? tc_desc_mn(b, LC_HALF, 1024) : tc_desc(b);
#pragma unroll 1
  for (int j = 0; j < 6; ++j) {                       // parts (0, 2), (2, 0), (1, 1), (0, 1), (1, 0), (0, 0)
    const uint64_t aj = a0 + (uint64_t)((0x010120 >> 4 * j & 3) * (LC_PART >> 4)), bj = b0 + (uint64_t)((0x001102 >> 4 * j & 3) * (LC_PART >> 4));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t kmajor = ((k >> 2) * LC_HALF + (k & 3) * 32) >> 4, mnmajor = k * 2048 >> 4;
      tc_mma(d + (k >> 1) * 128, aj + (A_MN ? mnmajor : kmajor), bj + (B_MN ? mnmajor : kmajor), idesc, (j > 0 || (k & 1)) ? 1u : 0u);
    }
  }
}
// 32 columns of a lane, the four accumulators added up; eight columns at a time, for the registers' sake.
__device__ __forceinline__ void lc_sum32(uint32_t taddr, float* sum) {
#pragma unroll
  for (int c = 0; c < 32; c += 8) {
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      uint32_t u[16];
      tc_ld8_issue(taddr + i * 128 + c, u);
      tc_ld8_issue(taddr + i * 128 + 128 + c, u + 8);
      tc_ld_wait();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float pair = __uint_as_float(u[j]) + __uint_as_float(u[j + 8]);
        sum[c + j] = i == 0 ? pair : sum[c + j] + pair;
      }
    }
  }
}

// ---------------------------------------------------------------- 1: gates
// With F the sum of the logarithms of the decays since the chunk's start, mode 0 needs exp(F_t - F_s) dt_s.  Mode 1 needs exp(F_t - F_s +
// i_s - m_t) with the running maximum m_t = F_t + max(m before the chunk, M_t), M_t the largest i_s - F_s so far: exp((i_s - F_s) -
// max(m, M_t)), from which F_t has gone.  What is subtracted is kept as two floats of a 64-bit sum; so is F_t, because m_t itself is
// the outputs' floor exp(-m_t) and F_t and M_t, hundreds each, cancel there.
// Planes: mode 0 F (high, low), dt; mode 1 i - F (high, low), M (high, low), F (high, low).  A warp per (chunk, head), 32 tokens at a time.
template <int MODE>
__global__ void __launch_bounds__(128)
lc_gates_kernel(const float* __restrict__ ga, const float* __restrict__ gb, long g_stride, const float* __restrict__ p0,
                const float* __restrict__ p1, float cap, LcArgs A) {
  const int lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
  const Portion place = find_portion<false>(A.cu_tokens, A.S, 1, LC_T, blockIdx.x);
  if (h >= A.H || place.seq < 0) return;
  const int b0 = A.cu_tokens[place.seq] + ((int)blockIdx.x - place.before) * LC_T, b1 = min(A.cu_tokens[place.seq + 1], b0 + LC_T);
  const size_t TH = (size_t)A.T * A.H;
  if (MODE == 1 && lane == 0 && (int)blockIdx.x == place.before) {                  // the maximum before the step: one block of the scan overwrites
    const int slot = A.state_slots[place.seq];                                      // the slot while others may not have started
    A.den[TH + (size_t)blockIdx.x * A.H + h] =
        slot >= 0 && slot < A.num_slots ? A.state[(size_t)slot * A.state_stride + (size_t)A.H * A.N * (A.dv + 1) + h] : 0.f;
  }
  const double a_h = MODE == 0 ? (double)expf(p0[h]) : 0.0;
  double sum = 0.0, last = -INFINITY;                 // the sum before these 32; mode 1: the largest i - sum so far
  for (int t = b0; t < b1; t += 32) {
    const bool live = t + lane < b1;
    float x = 0.f, y = 0.f;
    if (live) {
      x = ga[(size_t)(t + lane) * g_stride + h];
      if (MODE == 1) y = gb[(size_t)(t + lane) * g_stride + h];
    }
    float take;
    double F;
    if (MODE == 0) {
      take = lr_softplus(x + p1[h]);
      F = live ? -a_h * (double)take : 0.0;
    } else {
      take = cap * tanhf((x + p0[h]) / cap);                                        // log input gate
      F = live ? (double)lr_logsigmoid(cap * tanhf((y + p1[h]) / cap)) : 0.0;       // log forget gate
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, F, o);
      if (lane >= o) F += up;
    }
    F += sum;
    double most = MODE == 1 && live ? (double)take - F : -INFINITY;
    if (MODE == 1) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, most, o);
        if (lane >= o) most = fmax(most, up);
      }
      most = fmax(most, last);
    }
    if (live) {
      const size_t at = (size_t)(t + lane) * A.H + h;
      const double x2 = MODE == 0 ? F : (double)take - F;
      const float hi = (float)x2;
      A.gates[at] = hi; A.gates[TH + at] = (float)(x2 - (double)hi);
      if (MODE == 0) {
        A.gates[2 * TH + at] = take;
      } else {
        const float mh = (float)most;
        const float fh = (float)F;
        A.gates[2 * TH + at] = mh; A.gates[3 * TH + at] = (float)(most - (double)mh);
        A.gates[4 * TH + at] = fh; A.gates[5 * TH + at] = (float)(F - (double)fh);
      }
    }
    sum = __shfl_sync(0xffffffffu, F, 31);
    last = __shfl_sync(0xffffffffu, most, 31);
  }
  if (lane == 0) {
    float* sc = A.scale + ((size_t)blockIdx.x * A.H + h) * 4;
    const double L = sum + last;
    sc[0] = (float)sum; sc[1] = (float)(sum - (double)sc[0]);
    sc[2] = (float)L; sc[3] = (float)(L - (double)sc[2]);
  }
}

// ---------------------------------------------------------------- what the two product kernels share
struct LcShared {
  uint64_t bar;
  uint32_t tmem;
  int abort;
  float hi[LC_T], lo[LC_T], take[LC_T];               // modes 0, 1: a token's F or i - F, and dt or exp(-m_t)
  float m[LC_T], ml[LC_T];                            // mode 1: max(m before the chunk, M)
  float by[LC_T];                                     // modes 0, 1: the weight of S_0 in a token's output
  float group[8][LC_T], lacks[8][LC_T];               // mode 3: the decay through 16 tokens and what it lacks to 1
  int bad[LC_T];                                      // the first token whose value in this column is not finite
  float qn[LC_T], den[4][LC_T];                       // mode 1
  int blocks;                                         // mode 3: blocks with references of their own
  int direct[4];                                      // those of 32 whose weights are formed one by one,
  float self[4][32][33];                              // and those: [block][s][t]
};

struct LcPlace { int s, c, nc, t0, cnt, h, hq; size_t at; };

__device__ __forceinline__ bool lc_place(const LcArgs& A, LcPlace& p) {
  const Portion place = find_portion<false>(A.cu_tokens, A.S, 1, LC_T, blockIdx.x);
  p.s = place.seq;
  if (p.s < 0) return false;
  p.c = (int)blockIdx.x - place.before;
  const int t0 = A.cu_tokens[p.s], t1 = A.cu_tokens[p.s + 1];
  p.nc = (t1 - t0 + LC_T - 1) / LC_T;
  p.t0 = t0 + p.c * LC_T;
  p.cnt = min(LC_T, t1 - p.t0);
  p.h = blockIdx.y; p.hq = p.h / (A.H / A.qk_heads);
  p.at = (size_t)blockIdx.x * A.H + p.h;
  return true;
}

// A 4-wide piece of row `t` (zeros behind the chunk and behind `width`).
__device__ __forceinline__ float4 lc_piece(const float* base, long stride, int t, int cnt, int col, int width) {
  return t < cnt && col < width ? *reinterpret_cast<const float4*>(base + (size_t)t * stride + col) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ bool lc_odd(float x) { return !(fabsf(x) < 3.38e38f); }       // not finite, or beyond bfloat16's largest
// The values: what is not finite stays out, and its column is marked from its token on.
__device__ __forceinline__ void lc_put_value(unsigned char* plane, LcShared& sh, int t, int col, float4 v) {
  if (lc_odd(v.x) || lc_odd(v.y) || lc_odd(v.z) || lc_odd(v.w)) {
    if (lc_odd(v.x)) { atomicMin(&sh.bad[col], t); v.x = 0.f; }
    if (lc_odd(v.y)) { atomicMin(&sh.bad[col + 1], t); v.y = 0.f; }
    if (lc_odd(v.z)) { atomicMin(&sh.bad[col + 2], t); v.z = 0.f; }
    if (lc_odd(v.w)) { atomicMin(&sh.bad[col + 3], t); v.w = 0.f; }
  }
  lc_put4(plane, t, col, v);
}

__device__ __forceinline__ void lc_set_up(LcShared& sh) {
  if (threadIdx.x == 0) {
    tc_mbar_init(&sh.bar, 1);
    sh.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < LC_T) sh.bad[threadIdx.x] = LC_T;
  if (threadIdx.x < 4) sh.direct[threadIdx.x] = 0;
  if (threadIdx.x == 0) sh.blocks = 1;
  if ((threadIdx.x >> 5) == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc_smem(&sh.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}
__device__ __forceinline__ void lc_tear_down(LcShared& sh, int* err) {
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(sh.tmem) : "memory");
  }
  if (threadIdx.x == 0 && sh.abort) report_error(err, PHOTON_DEV_WAIT_TIMEOUT, blockIdx.x, blockIdx.y, 0);
}
// What all threads wrote is there for the products, which warp 0 issues (`issue` runs in one of its lanes).
template <class F>
__device__ __forceinline__ void lc_run(LcShared& sh, F issue) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    if (tc_elect()) { issue(); tc_commit(&sh.bar); }
    __syncwarp();
  }
}
__device__ __forceinline__ void lc_done(LcShared& sh, uint32_t& parity) {
  tc_wait(&sh.bar, parity, &sh.abort);                // a wait that runs out raises the flag; what follows stays in bounds
  parity ^= 1;
  tc_fence_after();
}

// Mode 3, two rows of a token: the keys, and the decays.  Tokens behind the chunk and rows behind the state keep everything.
__device__ __forceinline__ void lc_row_gate(const LcArgs& A, const LcPlace& p, int t, int n, float2& key, float2& decay) {
  key = make_float2(0.f, 0.f); decay = make_float2(1.f, 1.f);
  if (t >= p.cnt || n >= A.N) return;
  key = *reinterpret_cast<const float2*>(A.k + (size_t)(p.t0 + t) * A.k_stride + (size_t)p.hq * A.N + n);
  decay = *reinterpret_cast<const float2*>(A.a + (size_t)(p.t0 + t) * A.a_stride + (size_t)p.hq * A.N + n);
}

// ---------------------------------------------------------------- 2: the chunks' sums
template <int MODE>
__global__ void __launch_bounds__(LC_THREADS, 1)
lc_ends_kernel(const LcArgs A) {
  extern __shared__ unsigned char lc_dyn[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)lc_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char *X = base, *Y = base + LC_PLANE;
  LcShared& sh = *reinterpret_cast<LcShared*>(base + 2 * LC_PLANE);
  LcPlace p;
  pdl_wait();
  if (!lc_place(A, p)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  lc_set_up(sh);
  const float* v0 = A.v + (size_t)p.t0 * A.v_stride + (size_t)p.h * A.dv;
  if (MODE < 2) {
    const float* k0 = A.k + (size_t)p.t0 * A.k_stride + (size_t)p.hq * A.N;
    const size_t TH = (size_t)A.T * A.H, g0 = (size_t)p.t0 * A.H + p.h;
    const size_t end = g0 + (size_t)(p.cnt - 1) * A.H + (MODE == 1 ? 2 * TH : 0);       // F, or M, at the chunk's end
    const float e_hi = A.gates[end], e_lo = A.gates[TH + end];
    float4 kk[8], vv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) kk[i] = lc_piece(k0, A.k_stride, warp + i * 16, p.cnt, lane * 4, A.N);
#pragma unroll
    for (int i = 0; i < 8; ++i) vv[i] = lc_piece(v0, A.v_stride, warp + i * 16, p.cnt, lane * 4, A.dv);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = warp + i * 16;                    // a warp takes a token at a time
      float w = 0.f;
      if (t < p.cnt) {
        const size_t at = g0 + (size_t)t * A.H;
        const float f = (e_hi - A.gates[at]) + (e_lo - A.gates[TH + at]);
        w = MODE == 0 ? expf(f) * A.gates[2 * TH + at] : expf(-f);
      }
      float4 k = kk[i];
      k.x *= w; k.y *= w; k.z *= w; k.w *= w;
      lc_put4(X, t, lane * 4, k);
      lc_put_value(Y, sh, t, lane * 4, vv[i]);
    }
  } else {
    const int n = (tid & 63) * 2, tg = tid >> 6;
    float2 key[16], e[16];
    float2 b = make_float2(1.f, 1.f), B = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) lc_row_gate(A, p, tg * 16 + i, n, key[i], e[i]);
    // the decay behind each token to the end of the 16, from the last on
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      const float2 decay = e[i];
      e[i] = b;
      lr_decay(decay.x * b.x, 1.0f - decay.x, b.x, B.x);
      lr_decay(decay.y * b.y, 1.0f - decay.y, b.y, B.y);
    }
    *reinterpret_cast<float2*>(&sh.group[tg][n]) = b;
    *reinterpret_cast<float2*>(&sh.lacks[tg][n]) = B;
    __syncthreads();
    b = make_float2(1.f, 1.f); B = make_float2(0.f, 0.f);
    for (int g = 7; g > tg; --g) {
      const float2 d = *reinterpret_cast<const float2*>(&sh.group[g][n]), l = *reinterpret_cast<const float2*>(&sh.lacks[g][n]);
      lr_decay(d.x * b.x, l.x, b.x, B.x);
      lr_decay(d.y * b.y, l.y, b.y, B.y);
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) lc_put2(X, tg * 16 + i, n, key[i].x * (e[i].x * b.x), key[i].y * (e[i].y * b.y));
    if (tg == 0) {
      const float2 d = *reinterpret_cast<const float2*>(&sh.group[0][n]), l = *reinterpret_cast<const float2*>(&sh.lacks[0][n]);
      lr_decay(d.x * b.x, l.x, b.x, B.x);
      lr_decay(d.y * b.y, l.y, b.y, B.y);
      float* vec = A.vecs + p.at * A.N;
      if (n < A.N) { vec[n] = lr_code(b.x, B.x); vec[n + 1] = lr_code(b.y, B.y); }
    }
    float4 vv[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) vv[i] = lc_piece(v0, A.v_stride, warp + i * 16, p.cnt, lane * 4, A.dv);
#pragma unroll
    for (int i = 0; i < 8; ++i) lc_put_value(Y, sh, warp + i * 16, lane * 4, vv[i]);
  }
  uint32_t parity = 0;
  lc_run(sh, [&]() { lc_product<true, true>(sh.tmem, tc_smem(Y), tc_smem(X), 128); });     // U^T [dv][n]: rows of tokens are K of both
  if (MODE == 1) {
    // the sum of the chunk's weighted keys: a thread per row and 32 tokens, parts as the products see them
    const int n = tid & 127, t1 = tid >> 7;
    float s = 0.f;
    for (int t = t1 * 32; t < t1 * 32 + 32; ++t) {
      const unsigned char* d = X + (n >> 6) * LC_HALF + t * 128 + ((((n & 63) >> 3) ^ (t & 7)) << 4) + (n & 7) * 2;
      s += (__bfloat162float(*reinterpret_cast<const bf16*>(d + 2 * LC_PART)) + __bfloat162float(*reinterpret_cast<const bf16*>(d + LC_PART))) +
           __bfloat162float(*reinterpret_cast<const bf16*>(d));
    }
    sh.den[t1][n] = s;
    __syncthreads();
    if (tid < A.N) A.vecs[p.at * A.N + tid] = (sh.den[0][tid] + sh.den[1][tid]) + (sh.den[2][tid] + sh.den[3][tid]);
  }
  lc_done(sh, parity);
  pdl_launch_dependents();
  {
    const int col = (warp & 3) * 32 + lane, n0 = (warp >> 2) * 32;
    float u[32];
    lc_sum32(sh.tmem + ((uint32_t)((warp & 3) * 32) << 16) + n0, u);
    if (col < A.dv) {
      float* dst = A.ends + p.at * A.N * A.dv + (size_t)n0 * A.dv + col;
      const bool bad = sh.bad[col] < LC_T;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (n0 + j < A.N) dst[(size_t)j * A.dv] = bad ? NAN : u[j];
    }
  }
  lc_tear_down(sh, A.err);
}

// ---------------------------------------------------------------- 3: from chunk to chunk
// Block (x, head, request): four numbers of the state a thread; the last x has mode 1's n and the running maximum.
template <int MODE>
__global__ void __launch_bounds__(256)
lc_scan_kernel(const LcArgs A) {
  pdl_wait();
  const int s = blockIdx.z, h = blockIdx.y;
  const int t0 = A.cu_tokens[s], t1 = A.cu_tokens[s + 1], nc = (t1 - t0 + LC_T - 1) / LC_T;
  if (nc <= 0) return;
  int before = 0;                                     // chunks of the requests in front
  for (int i = threadIdx.x & 31; i < s; i += 32) before += (A.cu_tokens[i + 1] - A.cu_tokens[i] + LC_T - 1) / LC_T;
  before = __reduce_add_sync(0xffffffffu, before);
  int slot = A.state_slots[s];
  if (slot >= A.num_slots) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && h == 0) report_error(A.err, PHOTON_DEV_BAD_SLOT, s, slot, A.num_slots);
    slot = -1;
  }
  float* row0 = slot >= 0 ? A.state + (size_t)slot * A.state_stride : nullptr;
  const int size = A.N * A.dv;
  const bool vec = MODE == 1 && blockIdx.x == gridDim.x - 1;
  const int i = vec ? threadIdx.x * 4 : (blockIdx.x * 256 + threadIdx.x) * 4, end = vec ? A.N : size;
  float* slot_at = row0 ? row0 + (vec ? (size_t)A.H * size + (size_t)h * A.N : (size_t)h * size) + i : nullptr;
  float* slot_m = row0 ? row0 + (size_t)A.H * size + (size_t)A.H * A.N + h : nullptr;
  float m = MODE == 1 ? A.den[(size_t)A.T * A.H + (size_t)before * A.H + h] : 0.f;  // from lc_gates_kernel
  float4 S = i < end && row0 ? *reinterpret_cast<const float4*>(slot_at) : make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t step = vec ? (size_t)A.H * A.N : (size_t)A.H * size;
  float* at = (vec ? A.vecs + ((size_t)before * A.H + h) * A.N : A.ends + ((size_t)before * A.H + h) * size) + i;
  const float* rows = A.vecs + ((size_t)before * A.H + h) * A.N + (i < size ? i / A.dv : 0);     // mode 3: the row's decay
  float* sc = A.scale + ((size_t)before * A.H + h) * 4;
  float4 next = make_float4(0.f, 0.f, 0.f, 0.f), after = next;
  if (i < end) { next = *reinterpret_cast<const float4*>(at); if (nc > 1) after = *reinterpret_cast<const float4*>(at + step); }
  for (int c = 0; c < nc; ++c, at += step, rows += (size_t)A.H * A.N, sc += 4 * A.H) {
    const float4 U = next;
    next = after;
    if (i < end && c + 2 < nc) after = *reinterpret_cast<const float4*>(at + 2 * step);
    float code, c2 = 1.f, m_start = m;
    auto near1 = [](float d) {                        // exp(d), d <= 0: near 1 what it lacks, with the sign that says so
      return d > -0.5f ? (d == 0.f ? -0.f : expm1f(d)) : expf(d);
    };
    if (MODE == 0) {
      code = near1(sc[0]);
      if (code >= 0.f && !(sc[0] == 0.f)) code = fmaf(code, sc[1], code);
    } else if (MODE == 1) {
      const double f = (double)sc[0] + (double)sc[1] + (double)m, L = (double)sc[2] + (double)sc[3];
      m = (float)fmax(f, L);
      const float d = (float)(f - (double)m);
      code = d <= 0.f ? near1(d) : expf(d);           // the rounding of m may have put it below f
      c2 = expf((float)(L - (double)m));
    } else {
      code = *rows;
    }
    if (i < end) {
      *reinterpret_cast<float4*>(at) = S;
      S.x = MODE == 1 ? fmaf(c2, U.x, lr_apply(code, S.x)) : lr_apply(code, S.x) + U.x;
      S.y = MODE == 1 ? fmaf(c2, U.y, lr_apply(code, S.y)) : lr_apply(code, S.y) + U.y;
      S.z = MODE == 1 ? fmaf(c2, U.z, lr_apply(code, S.z)) : lr_apply(code, S.z) + U.z;
      S.w = MODE == 1 ? fmaf(c2, U.w, lr_apply(code, S.w)) : lr_apply(code, S.w) + U.w;
    }
    if (vec && threadIdx.x == 0 && c > 0) A.den[(size_t)A.T * A.H + ((size_t)(before + c)) * A.H + h] = m_start;
  }
  pdl_launch_dependents();
  if (i < end && slot_at) *reinterpret_cast<float4*>(slot_at) = S;
  if (vec && threadIdx.x == 0 && slot_m) *slot_m = m;
}

// ---------------------------------------------------------------- 4: the outputs
template <int MODE>
__global__ void __launch_bounds__(LC_THREADS, 1)
lc_out_kernel(const LcArgs A) {
  extern __shared__ unsigned char lc_dyn[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)lc_dyn + 1023) & ~(uintptr_t)1023);
  unsigned char *X = base, *Y = base + LC_PLANE;
  LcShared& sh = *reinterpret_cast<LcShared*>(base + 2 * LC_PLANE);
  LcPlace p;
  pdl_wait();
  if (!lc_place(A, p)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  lc_set_up(sh);
  uint32_t parity = 0;
  const uint32_t x = tc_smem(X), y = tc_smem(Y);
  const uint32_t acc = sh.tmem;                       // in turn P^T, O^T from S_0, O^T from the chunk itself: each takes all columns
  const uint32_t mine = acc + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 32;
  const float* q0 = A.q + (size_t)p.t0 * A.q_stride + (size_t)p.hq * A.N;
  const float* v0 = A.v + (size_t)p.t0 * A.v_stride + (size_t)p.h * A.dv;
  const float* S0 = A.ends + p.at * A.N * A.dv;
  const float m0 = MODE == 1 ? A.den[(size_t)A.T * A.H + p.at] : 0.f;              // the running maximum before the chunk
  float4 ahead[8];                                    // S_0, on its way while the first products run
  auto fetch_state = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i) ahead[i] = lc_piece(S0, A.dv, warp + i * 16, A.N, lane * 4, A.dv);
  };
  auto put_state = [&]() {
#pragma unroll
    for (int i = 0; i < 8; ++i) lc_put4(Y, warp + i * 16, lane * 4, ahead[i]);
  };
  if (MODE < 2) {
    const float* k0 = A.k + (size_t)p.t0 * A.k_stride + (size_t)p.hq * A.N;
    if (tid < LC_T) {
      const size_t TH = (size_t)A.T * A.H, at = (size_t)(p.t0 + tid) * A.H + p.h;
      const bool in = tid < p.cnt;
      sh.hi[tid] = in ? A.gates[at] : 0.f;
      sh.lo[tid] = in ? A.gates[TH + at] : 0.f;
      if (MODE == 0) {
        sh.take[tid] = in ? A.gates[2 * TH + at] : 0.f;
        const float w = expf(sh.hi[tid]);
        sh.by[tid] = fmaf(w, sh.lo[tid], w);
      }
      if (MODE == 1) {
        const float mh = in ? A.gates[2 * TH + at] : 0.f, ml = in ? A.gates[3 * TH + at] : 0.f;
        const bool before = m0 > mh;                  // NaN: the token's own
        sh.m[tid] = before ? m0 : mh;
        sh.ml[tid] = before ? 0.f : ml;
        // high parts first: their sum is rounded relative to itself, however large they are
        sh.take[tid] = in ? expf(-((A.gates[4 * TH + at] + sh.m[tid]) + (A.gates[5 * TH + at] + sh.ml[tid]))) : 0.f;
        sh.by[tid] = expf((m0 - sh.m[tid]) - sh.ml[tid]);
      }
    }
    const float4 n0 = MODE == 1 && lane * 4 < A.N ? *reinterpret_cast<const float4*>(A.vecs + p.at * A.N + lane * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    float4 qq[8], kk[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      qq[i] = lc_piece(q0, A.q_stride, warp + i * 16, p.cnt, lane * 4, A.N);
      kk[i] = lc_piece(k0, A.k_stride, warp + i * 16, p.cnt, lane * 4, A.N);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = warp + i * 16;
      const float4 q = qq[i];
      lc_put4(X, t, lane * 4, q);
      lc_put4(Y, t, lane * 4, kk[i]);
      if (MODE == 1) {
        const float d = warp_sum((q.x * n0.x + q.y * n0.y) + (q.z * n0.z + q.w * n0.w));
        if (lane == 0) sh.qn[t] = d;
      }
    }
    lc_run(sh, [&]() { lc_product<false, false>(acc, y, x, 128); });               // P^T [s][t]
    fetch_state();
    lc_done(sh, parity);
  } else {
    // thread (pair of rows, 16 tokens)
    const int n = (tid & 63) * 2, tg = tid >> 6;
    float2 key[16], bq[16];                           // bq: first the decays as they lie in memory, then from the start of the sixteen on
    float2 b = make_float2(1.f, 1.f), B = make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 16; ++i) lc_row_gate(A, p, tg * 16 + i, n, key[i], bq[i]);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      lr_decay(bq[i].x * b.x, 1.0f - bq[i].x, b.x, B.x);
      lr_decay(bq[i].y * b.y, 1.0f - bq[i].y, b.y, B.y);
      bq[i] = b;
    }
    *reinterpret_cast<float2*>(&sh.group[tg][n]) = b;
    *reinterpret_cast<float2*>(&sh.lacks[tg][n]) = B;
    __syncthreads();
    auto through = [&](int g0, int g1) {              // the decay through the sixteens g0 .. g1 - 1
      float2 d = make_float2(1.f, 1.f), l = make_float2(0.f, 0.f);
      for (int g = g0; g < g1; ++g) {
        const float2 dg = *reinterpret_cast<const float2*>(&sh.group[g][n]), lg = *reinterpret_cast<const float2*>(&sh.lacks[g][n]);
        lr_decay(dg.x * d.x, lg.x, d.x, l.x);
        lr_decay(dg.y * d.y, lg.y, d.y, l.y);
      }
      return d;
    };
    auto small = [](float2 d) { return !(d.x >= LC_SMALL) || !(d.y >= LC_SMALL); };
    if (small(through(0, 8))) {
      const int half = tg >> 2 << 2, quarter = tg >> 1 << 1;
      atomicMax(&sh.blocks, small(through(half, half + 4)) ? 4 : 2);
      if (small(through(quarter, quarter + 2))) sh.direct[tg >> 1] = 1;
    }
    __syncthreads();
    const int blocks = sh.blocks, span = 8 / blocks, blk = tg / span;              // sixteens of a block, and this thread's
    const float2 in_blk = through(blk * span, tg);    // the decay from the block's start to this sixteen
    auto put_queries = [&](float2 f) {
#pragma unroll
      for (int g = 0; g < 16; g += 8) {
        float2 q[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int t = tg * 16 + g + i;
          q[i] = t < p.cnt && n < A.N ? *reinterpret_cast<const float2*>(q0 + (size_t)t * A.q_stride + n) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) lc_put2(X, tg * 16 + g + i, n, q[i].x * (bq[g + i].x * f.x), q[i].y * (bq[g + i].y * f.y));
      }
    };
    put_queries(in_blk);
    __syncthreads();
    for (int j = 0; j < blocks; ++j) {
      const int t0 = j * span * 16;
      if (t0 >= p.cnt) break;
      // keys as the queries of block j see them
      if (blk < j) {
        const float2 f = through(tg + 1, j * span);
        float2 d = make_float2(1.f, 1.f), l = make_float2(0.f, 0.f);               // behind a token to the end of its sixteen
#pragma unroll
        for (int i0 = 12; i0 >= 0; i0 -= 4) {         // the decays once more, a few at a time: registers that spill go to L2 here
          float2 decay[4], again;
#pragma unroll
          for (int i = 0; i < 4; ++i) lc_row_gate(A, p, tg * 16 + i0 + i, n, again, decay[i]);
#pragma unroll
          for (int i = 3; i >= 0; --i) {
            lc_put2(Y, tg * 16 + i0 + i, n, key[i0 + i].x * (d.x * f.x), key[i0 + i].y * (d.y * f.y));
            lr_decay(decay[i].x * d.x, 1.0f - decay[i].x, d.x, l.x);
            lr_decay(decay[i].y * d.y, 1.0f - decay[i].y, d.y, l.y);
          }
        }
      } else if (blk == j) {
        const bool direct = blocks == 4 && sh.direct[j] != 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float bx = bq[i].x * in_blk.x, by = bq[i].y * in_blk.y;
          lc_put2(Y, tg * 16 + i, n, direct ? 0.f : key[i].x / bx, direct ? 0.f : key[i].y / by);
        }
      }
      lc_run(sh, [&]() { lc_product<false, false>(acc + t0, y, x + t0 * 128, span * 16); });     // P^T [s][t0 ..]
      lc_done(sh, parity);
    }
    if (blocks > 1) put_queries(through(0, tg));                      // as S_0 sees them
    // Blocks whose decays are too small for a common reference: 16 threads share a token s, eight rows each; they multiply the decays up
    // from s on and meet the queries on the way.  Keys, decays and queries of the 32 tokens lie in shared memory, where the keys' parts
    // were.  Read from memory by every token that comes before, as they were, such blocks made 2,048 tokens of 16 heads (the recurrence, one row in
    // 128 with decays of 0.1) take 280 us; 164 so, 177 in segments, 102 where no block is like that.
    for (int j = 0; j < 4; ++j) {
      if (blocks < 4 || !sh.direct[j]) continue;
      float *ks = reinterpret_cast<float*>(Y), *as = ks + 32 * LC_T, *qs = as + 32 * LC_T;
      const float* k0 = A.k + (size_t)p.t0 * A.k_stride + (size_t)p.hq * A.N;
      const float* a0 = A.a + (size_t)p.t0 * A.a_stride + (size_t)p.hq * A.N;
      for (int i = warp; i < 32; i += 16) {
        *reinterpret_cast<float4*>(ks + i * LC_T + lane * 4) = lc_piece(k0, A.k_stride, j * 32 + i, p.cnt, lane * 4, A.N);
        *reinterpret_cast<float4*>(as + i * LC_T + lane * 4) = lc_piece(a0, A.a_stride, j * 32 + i, p.cnt, lane * 4, A.N);
        *reinterpret_cast<float4*>(qs + i * LC_T + lane * 4) = lc_piece(q0, A.q_stride, j * 32 + i, p.cnt, lane * 4, A.N);
      }
      __syncthreads();
      const int s = tid >> 4, l = tid & 15;
      float4 d1 = *reinterpret_cast<const float4*>(ks + s * LC_T + l * 4), d2 = *reinterpret_cast<const float4*>(ks + s * LC_T + 64 + l * 4);
#pragma unroll 1
      for (int t0 = (warp * 2) & ~7; t0 < 32; t0 += 8) {                             // from the warp's first token on
        float o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float *at = as + (t0 + i) * LC_T + l * 4, *qt = qs + (t0 + i) * LC_T + l * 4;
          const float4 a1 = *reinterpret_cast<const float4*>(at), a2 = *reinterpret_cast<const float4*>(at + 64);
          const float4 q1 = *reinterpret_cast<const float4*>(qt), q2 = *reinterpret_cast<const float4*>(qt + 64);
          if (t0 + i > s) {
            d1.x *= a1.x; d1.y *= a1.y; d1.z *= a1.z; d1.w *= a1.w;
            d2.x *= a2.x; d2.y *= a2.y; d2.z *= a2.z; d2.w *= a2.w;
          }
          o[i] = fmaf(d1.x, q1.x, fmaf(d1.y, q1.y, fmaf(d1.z, q1.z, d1.w * q1.w))) + fmaf(d2.x, q2.x, fmaf(d2.y, q2.y, fmaf(d2.z, q2.z, d2.w * q2.w)));
        }
        lr_meet<8, 8>(o, lane);                       // lanes 2 i and 2 i + 1 of the sixteen: the sum for token t0 + i
        if (!(l & 1)) sh.self[j][s][t0 + (l >> 1)] = o[0];
      }
      __syncthreads();                                // the plane takes the next block's, or the state
    }
  }
  if (MODE == 3) fetch_state();                       // no earlier: the keys' registers
  put_state();
  float pw[32];                                       // P^T of token s (this lane's row), 32 tokens t
  const int s = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
  lc_sum32(mine, pw);
  lc_run(sh, [&]() { lc_product<true, false>(acc, y, x, 128); });                  // O^T [dv][t]: rows of S_0 are K
  {
    const float fs_hi = MODE < 2 ? sh.hi[s] : 0.f, fs_lo = MODE < 2 ? sh.lo[s] : 0.f, take = MODE < 2 ? sh.take[s] : 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int t = c0 + j;
      float w = 0.f;
      if (s <= t && t < p.cnt) {
        w = pw[j];
        if (MODE < 2) {
          w *= MODE == 0 ? expf((sh.hi[t] - fs_hi) + (sh.lo[t] - fs_lo)) * take : expf((fs_hi - sh.m[t]) + (fs_lo - sh.ml[t]));
        }
      }
      pw[j] = w;
    }
  }
  if (MODE == 3 && sh.blocks == 4 && sh.direct[warp >> 2] && (warp & 3) == (warp >> 2)) {
#pragma unroll
    for (int j = 0; j < 32; ++j) if (c0 + j >= s && c0 + j < p.cnt) pw[j] = sh.self[warp >> 2][lane][j];
  }
  // the values, while the products with S_0 run
#pragma unroll
  for (int i = 0; i < 8; ++i) ahead[i] = lc_piece(v0, A.v_stride, warp + i * 16, p.cnt, lane * 4, A.dv);
  lc_done(sh, parity);
#pragma unroll
  for (int i = 0; i < 8; ++i) lc_put_value(Y, sh, warp + i * 16, lane * 4, ahead[i]);
#pragma unroll
  for (int j = 0; j < 32; j += 4) lc_put4(X, s, c0 + j, make_float4(pw[j], pw[j + 1], pw[j + 2], pw[j + 3]));
  float in[32];
  lc_sum32(mine, in);
  lc_run(sh, [&]() { lc_product<true, true>(acc, y, x, 128); });                   // O^T [dv][t]: tokens s are K of both
  if (MODE == 1) {
    lr_meet<16, 32>(pw, lane);                        // lane l: the sum over the warp's 32 tokens s for token c0 + l
    sh.den[warp & 3][c0 + lane] = pw[0];
    __syncthreads();
    if (tid < p.cnt) {
      const float nq = ((sh.den[0][tid] + sh.den[1][tid]) + (sh.den[2][tid] + sh.den[3][tid])) +
                       sh.by[tid] * sh.qn[tid];
      A.den[(size_t)(p.t0 + tid) * A.H + p.h] = fmaxf(fabsf(nq * A.q_scale), sh.take[tid]) + 1e-6f;
    }
  }
  lc_done(sh, parity);
  pdl_launch_dependents();
  {
    float u[32];
    lc_sum32(mine, u);
    const int col = (warp & 3) * 32 + lane;
    if (col < A.dv) {
      const float skip = MODE == 0 ? A.d_skip[p.h] : 0.f;
      const int bad = sh.bad[col], last = min(32, p.cnt - c0);
      float* dst = A.out + (size_t)(p.t0 + c0) * A.out_stride + (size_t)p.h * A.dv + col;
      const float* vv = v0 + (size_t)c0 * A.v_stride + col;
      float o[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        o[j] = (MODE < 2 ? fmaf(sh.by[c0 + j], in[j], u[j]) : in[j] + u[j]) * A.q_scale;
        if (MODE == 0) o[j] = fmaf(skip, j < last ? vv[(size_t)j * A.v_stride] : 0.f, o[j]);
      }
      if (bad < LC_T) {
#pragma unroll
        for (int j = 0; j < 32; ++j) if (c0 + j >= bad) o[j] = NAN;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) if (j < last) dst[(size_t)j * A.out_stride] = o[j];
    }
  }
  lc_tear_down(sh, A.err);
}

// ---------------------------------------------------------------- host side
static void lc_parts(int mode, int T, int chunks, int H, int N, int dv, long (&part)[4]) {
  auto four = [](long n) { return (n + 3) & ~3L; };
  part[0] = four(mode == 0 ? 3L * T * H : mode == 1 ? 6L * T * H : 0);
  part[1] = four((long)chunks * H * N * dv);
  part[2] = four((long)chunks * H * N);
  part[3] = four((long)chunks * H * 4);
}

// Floats of scratch that photon_linrec_chunks needs for requests of `chunks` chunks of 128 tokens in all.
PHOTON_API long photon_linrec_chunks_scratch(int mode, int T, int chunks, int H, int N, int dv) {
  long part[4], sum = 0;
  lc_parts(mode, T, chunks, H, N, dv, part);
  for (long p : part) sum += p;
  return sum;
}

template <int MODE>
static int lc_go(const LcArgs& A, const float* ga, const float* gb, long g_stride, const float* p0, const float* p1, float cap,
                 cudaStream_t stream) {
  const size_t smem = 2 * LC_PLANE + sizeof(LcShared) + 1024;
  cudaError_t e = cudaFuncSetAttribute(lc_ends_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(lc_out_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  if (MODE < 2) {
    lc_gates_kernel<MODE><<<dim3(A.chunks, (A.H + 3) / 4), 128, 0, stream>>>(ga, gb, g_stride, p0, p1, cap, A);
    const int st = launch_status();
    if (st != 0) return st;
  }
  int st = launch_pdl(lc_ends_kernel<MODE>, dim3(A.chunks, A.H), dim3(LC_THREADS), smem, stream, A);
  if (st != 0) return st;
  st = launch_pdl(lc_scan_kernel<MODE>, dim3((A.N * A.dv + 1023) / 1024 + (MODE == 1), A.H, A.S), dim3(256), 0, stream, A);
  if (st != 0) return st;
  return launch_pdl(lc_out_kernel<MODE>, dim3(A.chunks, A.H), dim3(LC_THREADS), smem, stream, A);
}

// As photon_linrec_segments, in chunks of 128 tokens on the tensor cores: `chunks` of them, the sum over the requests of their tokens / 128,
// rounded up.  Modes 0, 1 and 3.  N and dv up to 128, multiples of 4; rows and bases 16-byte aligned.  Mode 1: den has T * H floats for the
// caller and chunks * H behind them.  scratch: photon_linrec_chunks_scratch floats, 16-byte aligned.
PHOTON_API int photon_linrec_chunks(int mode, const float* q, long q_stride, const float* k, long k_stride, const float* v,
                                    long v_stride, const float* a, long a_stride, const float* ga, const float* gb, long g_stride,
                                    const float* p0, const float* p1, const float* p2, float cap, float q_scale,
                                    const int* cu_tokens, const int* state_slots, float* state, long state_stride, int num_slots,
                                    float* out, long out_stride, float* den, float* scratch, int T, int S, int H, int qk_heads,
                                    int N, int dv, int chunks, int* err, cudaStream_t stream) {
  if (S <= 0 || T <= 0) return 0;
  if (mode < 0 || mode > 3 || mode == 2 || H <= 0 || qk_heads <= 0 || H % qk_heads || N <= 0 || dv <= 0 || chunks <= 0) return PHOTON_ERR_ARGUMENT;
  if (scratch == nullptr || ((uintptr_t)scratch & 15) || (mode == 1 && (!(cap > 0.f) || den == nullptr)) || (mode == 3) != (a != nullptr))
    return PHOTON_ERR_ARGUMENT;
  if (N > LC_T || dv > LC_T || (N & 3) || (dv & 3) || H > 65535 || S > 65535 || (q_stride & 3) || (k_stride & 3) || (v_stride & 3) ||
      (a_stride & 3) || (state_stride & 3) || ((uintptr_t)q & 15) || ((uintptr_t)k & 15) || ((uintptr_t)v & 15) || ((uintptr_t)a & 15) ||
      ((uintptr_t)state & 15))
    return PHOTON_ERR_UNSUPPORTED;
  LcArgs A;
  A.q = q; A.q_stride = q_stride; A.k = k; A.k_stride = k_stride; A.v = v; A.v_stride = v_stride; A.a = a; A.a_stride = a_stride;
  A.d_skip = p2; A.q_scale = q_scale; A.cu_tokens = cu_tokens; A.state_slots = state_slots; A.state = state; A.state_stride = state_stride;
  A.num_slots = num_slots; A.out = out; A.out_stride = out_stride; A.den = den;
  A.T = T; A.S = S; A.H = H; A.qk_heads = qk_heads; A.N = N; A.dv = dv; A.chunks = chunks; A.err = err;
  long part[4];
  lc_parts(mode, T, chunks, H, N, dv, part);
  A.gates = scratch;
  A.ends = A.gates + part[0];
  A.vecs = A.ends + part[1];
  A.scale = A.vecs + part[2];
  if (mode == 0) return lc_go<0>(A, ga, gb, g_stride, p0, p1, cap, stream);
  if (mode == 1) return lc_go<1>(A, ga, gb, g_stride, p0, p1, cap, stream);
  return lc_go<3>(A, ga, gb, g_stride, p0, p1, cap, stream);
}
