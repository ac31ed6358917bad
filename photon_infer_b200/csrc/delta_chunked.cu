// The gated delta rule (delta.cu) over long prompt portions, 32 tokens at a time.
//
// Per head, with b_t the product of the decays since the chunk's start (b_t / b_s for s <= t is formed from 64-bit sums of
// their logarithms) and S0 the state there, the token-by-token rule
//   S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q
// is, for all tokens of the chunk together,
//   (I + L) U = diag(beta) V - diag(beta b) K S0,          L_ts = beta_t (b_t / b_s) k_t . k_s   for s < t
//   O = diag(b) Q S0 + A U,                                A_ts = (b_t / b_s) q_t . k_s          for s <= t
//   S1 = b_C S0 + sum_s (b_C / b_s) k_s u_s^T
// so with W = (I + L)^-1 diag(beta b) K and U0 = (I + L)^-1 diag(beta) V, which need no state, U = U0 - W S0.
//   1. dc_prep_kernel, a block per (chunk, head), all chunks side by side: W, U0, A, diag(b) Q and the keys of the
//      update, by 32-bit multiply-adds (the triangular system by forward substitution, a column a thread).
//   2. dc_walk_kernel, a block per (head, 16 columns of the state), chunk after chunk: U, O and S1.
// (Yang, Wang, Shen, Panda, Kim: "Parallelizing linear transformers with the delta rule over sequence length", 2024, has the
// chunked form; the gates ride in b and beta.)
//
// The walk's products run on the tensor cores at 32-bit accuracy: every operand is split into two tf32 numbers (a = a1 + a2 up to
// 2^-22 |a|), a1 b1 is formed by mma.m16n8k8 from a zero accumulator and added up by 32-bit additions of this kernel,
// and a1 b2 and a2 b1 in accumulators of their own (Ootomo and Yokota: "Recovering single precision accuracy from Tensor
// Cores while surpassing the FP32 theoretical peak performance", 2022: it is the accumulation inside the tensor cores that
// rounds coarsely).
//
// A token whose inputs are not finite reaches its own and later outputs only, as token by token; there it is NaN where the plain
// rule may leave an infinity (the second part of an infinity's split is NaN).
//
// The walk keeps S^T [16 columns][128 rows] in accumulator registers, a warp 32 of the rows: an accumulator fragment with
// the rows 2 t, 2 t + 1 of a lane is at once the A fragment of the next product, if the other operand's k index is read
// in the same order.  Its operands lie in memory in that order, 16 bytes a lane, and travel by cp.async into a ring of three
// stages that each thread fills for itself; the four warps' partial sums of W S0 and Q S0 meet in shared memory, one
// barrier a chunk.
//
// Measured, 2,048 tokens, 16 heads of 128 x 128: prep 52 us, walk 176 us, against 616 us for the token-by-token kernel, whose chain
// from one token to the next is 300 ns (the look for outputs that are not finite came later: a mixer's step of these tokens 340 -> 355 us);
// 64 tokens 10 + 8 us against 22 us and more for its walk.  The error against 64 bits is
// 2.4e-7 (outputs) and 1.8e-7 (state) where the token-by-token kernel has 2.6e-7 and 2.1e-7.
// What bounds the prep: its blocks' loads and stores (100 MB, 15 us of them) and the gaps between a block's steps; with the keys and queries
// read 4 bytes at a time in turn, and the values only when the substitution asks for them, it took 103 us.  Three or four blocks an SM
// instead of two take the same time.  The walk takes 2.75 us a chunk, 156 products of 16 x 8 x 8 and
// their operands' splits for each scheduler; eight warps of 16 rows instead of four of 32 take 181 us, the same walk in plain 32-bit
// multiply-adds (tiles of 4 x 4 from shared memory) 218 us.
#include "portions.cuh"
#include <float.h>
#include <math.h>

#define DC 32                                          // tokens of a chunk
#define DC_D 128                                       // rows of the state (a head's keys), zeros behind the head
#define DC_CB 16                                       // columns of a block of the walk
#define DC_MAT (DC * DC_D)                             // floats of W, of Q and of the update's keys
#define DC_STAGES 3
#define DC_STAGE (3 * DC_MAT + DC * DC + DC * DC_CB)   // floats of a stage: W, Q, K, A, U0 of the block's columns
#define DC_RED (4 * 8 * 32 * 4)                        // floats of the warps' partial sums

__device__ __forceinline__ float dc_softplus(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

// Scratch of a (chunk, head): W, Q, K [4 warps][4 token tiles][2][32 lanes][4]; A [4][2][32][4]; U0 [dvp / 16][4][32][4]; b_C.
__host__ __device__ __forceinline__ long dc_floats(int dvp) { return 3L * DC_MAT + DC * DC + (long)DC * dvp + 4; }

// ---------------------------------------------------------------- 1: what needs no state
#define DP_LD (DC_D + 4)

__global__ void __launch_bounds__(256, 2)
dc_prep_kernel(const float* __restrict__ y, const void* ab, long ab_stride, int ab_bf16, const float* __restrict__ a_log,
               const float* __restrict__ dt_bias, const int* __restrict__ cu_tokens, int S, int from, float* __restrict__ scratch, int Gq,
               int H, int dim, int dv, int dvp) {
  extern __shared__ __align__(16) float dp[];
  float* ks = dp;                                      // [DC][DP_LD]
  float* qs = ks + DC * DP_LD;                         // [DC][DP_LD]
  float* Ls = qs + DC * DP_LD;                         // [DC][DC + 4]
  float* us = Ls + DC * (DC + 4);                      // [DC][dvp + 4]
  __shared__ double lg[DC];
  __shared__ float beta_s[DC], b_s[DC], tail_s[DC];
  const int h = blockIdx.y, tid = threadIdx.x;
  const Portion at = find_portion<false>(cu_tokens, S, from, DC, blockIdx.x);
  if (at.seq < 0) return;
  const int t0 = cu_tokens[at.seq] + ((int)blockIdx.x - at.before) * DC, n = min(DC, cu_tokens[at.seq + 1] - t0);
  const int C = 2 * Gq * dim + H * dv, hq = h / (H / Gq);
  float* dst = scratch + ((size_t)blockIdx.x * H + h) * dc_floats(dvp);
  // Keys, queries and values (at first U0's place holds them) all at once, zeros behind the heads' sizes and the chunk's end.
  const bool pieces = dim % 4 == 0 && dv % 4 == 0 && C % 4 == 0 && (uintptr_t)y % 16 == 0;
  auto bring = [&](float* to, int ld, int width, int from, int held) {
    if (pieces) {
      for (int i = tid; i < DC * (width / 4); i += 256) {
        const int t = i / (width / 4), d = i % (width / 4) * 4;
        const bool there = t < n && d < held;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to + t * ld + d)),
                     "l"(there ? y + (size_t)(t0 + t) * C + from + d : y), "r"(there ? 16 : 0) : "memory");
      }
    } else {
      for (int i = tid; i < DC * width; i += 256) {
        const int t = i / width, d = i % width;
        to[t * ld + d] = t < n && d < held ? y[(size_t)(t0 + t) * C + from + d] : 0.f;
      }
    }
  };
  bring(ks, DP_LD, DC_D, (Gq + hq) * dim, dim);
  bring(qs, DP_LD, DC_D, hq * dim, dim);
  bring(us, dvp + 4, dvp, 2 * Gq * dim + h * dv, dv);
  if (tid < 32) {
    // the chunk's gates: tokens behind its end decay nothing and write nothing
    float lgate = 0.f, beta = 0.f;
    if (tid < n) {
      const size_t at = (size_t)(t0 + tid) * ab_stride + h;
      const float ra = ab_bf16 ? __bfloat162float(((const bf16*)ab)[at]) : ((const float*)ab)[at];
      const float rb = ab_bf16 ? __bfloat162float(((const bf16*)ab)[at + H]) : ((const float*)ab)[at + H];
      lgate = -expf(a_log[h]) * dc_softplus(ra + dt_bias[h]);
      if (lgate < -1e4f) lgate = -1e4f;                // a decay of 0 either way; infinities have no differences
      beta = 1.0f / (1.0f + expf(-rb));
    }
    double d = lgate;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, d, o);
      if (tid >= o) d += up;
    }
    const double end = __shfl_sync(0xffffffffu, d, 31);
    lg[tid] = d;
    beta_s[tid] = beta;
    b_s[tid] = expf((float)d);
    tail_s[tid] = expf((float)(end - d));
    if (tid == 31) dst[3 * DC_MAT + DC * DC + (size_t)DC * dvp] = b_s[31];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  {
    // L and A: thread (t, j) has the pairs (t, j), (t, j + 8) ..
    const int t = tid >> 3, j = tid & 7;
    float kk[4] = {0.f, 0.f, 0.f, 0.f}, qk[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int d = 0; d < DC_D; d += 4) {
      const float4 kt = *reinterpret_cast<const float4*>(ks + t * DP_LD + d), qt = *reinterpret_cast<const float4*>(qs + t * DP_LD + d);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 x = *reinterpret_cast<const float4*>(ks + (j + 8 * u) * DP_LD + d);
        kk[u] = fmaf(kt.x, x.x, kk[u]); kk[u] = fmaf(kt.y, x.y, kk[u]); kk[u] = fmaf(kt.z, x.z, kk[u]); kk[u] = fmaf(kt.w, x.w, kk[u]);
        qk[u] = fmaf(qt.x, x.x, qk[u]); qk[u] = fmaf(qt.y, x.y, qk[u]); qk[u] = fmaf(qt.z, x.z, qk[u]); qk[u] = fmaf(qt.w, x.w, qk[u]);
      }
    }
    float* A = dst + 3 * DC_MAT;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int sx = j + 8 * u;
      const float ratio = sx <= t ? expf((float)(lg[t] - lg[sx])) : 0.f;
      Ls[t * (DC + 4) + sx] = sx < t ? beta_s[t] * ratio * kk[u] : 0.f;
      // A [warp t / 8][sx / 16][lane (t % 8) * 4 + (sx % 8) / 2][(sx % 16) / 8 * 2 + sx % 2]
      A[((t >> 3) * 2 + (sx >> 4)) * 128 + ((t & 7) * 4 + ((sx & 7) >> 1)) * 4 + ((sx >> 3) & 1) * 2 + (sx & 1)] = sx <= t ? ratio * qk[u] : 0.f;
    }
  }
  // Q and K of the walk, in its order of lanes (qs and ks are read by rows)
  for (int i = tid; i < DC_MAT / 4; i += 256) {
    const int lane = i & 31, j2 = (i >> 5) & 1, ti = (i >> 6) & 3, w = i >> 8;
    const int g = lane >> 2, t = lane & 3;
    {
      const int r = 8 * ti + g, d = 32 * w + 16 * j2 + 2 * t;
      const float b = b_s[r];
      const float* p = qs + r * DP_LD + d;
      reinterpret_cast<float4*>(dst + DC_MAT)[i] = make_float4(b * p[0], b * p[1], b * p[8], b * p[9]);
    }
    {
      const int r = 8 * ti + 2 * t, d = 32 * w + 16 * j2 + g;
      const float e0 = tail_s[r], e1 = tail_s[r + 1];
      const float* p = ks + r * DP_LD + d;
      reinterpret_cast<float4*>(dst + 2 * DC_MAT)[i] = make_float4(e0 * p[0], e1 * p[DP_LD], e0 * p[8], e1 * p[DP_LD + 8]);
    }
  }
  __syncthreads();                                     // L is there, and qs is free for W
  for (int col = tid; col < DC_D + dvp; col += 256) {
    const bool isw = col < DC_D;
    const int vc = col - DC_D;
    float x[DC];
#pragma unroll
    for (int t = 0; t < DC; ++t) {
      float r;
      if (isw) r = b_s[t] * ks[t * DP_LD + col];
      else r = us[t * (dvp + 4) + vc];
      x[t] = beta_s[t] * r;
    }
#pragma unroll
    for (int t = 1; t < DC; ++t) {
      float a = x[t];
#pragma unroll
      for (int s4 = 0; s4 < t; s4 += 4) {
        const float4 l = *reinterpret_cast<const float4*>(Ls + t * (DC + 4) + s4);     // zeros from the diagonal on
        a = fmaf(-l.x, x[s4], a);
        if (s4 + 1 < t) a = fmaf(-l.y, x[s4 + 1], a);
        if (s4 + 2 < t) a = fmaf(-l.z, x[s4 + 2], a);
        if (s4 + 3 < t) a = fmaf(-l.w, x[s4 + 3], a);
      }
      x[t] = a;
    }
    float* to = isw ? qs + col : us + vc;
    const int ld = isw ? DP_LD : dvp + 4;
#pragma unroll
    for (int t = 0; t < DC; ++t) to[t * ld] = x[t];
  }
  __syncthreads();
  for (int i = tid; i < DC_MAT / 4; i += 256) {
    const int lane = i & 31, j2 = (i >> 5) & 1, ti = (i >> 6) & 3, w = i >> 8;
    const float* p = qs + (8 * ti + (lane >> 2)) * DP_LD + 32 * w + 16 * j2 + 2 * (lane & 3);
    reinterpret_cast<float4*>(dst)[i] = make_float4(p[0], p[1], p[8], p[9]);
  }
  float4* U = reinterpret_cast<float4*>(dst + 3 * DC_MAT + DC * DC);
  for (int i = tid; i < DC * dvp / 4; i += 256) {
    const int lane = i & 31, ti = (i >> 5) & 3, cb = i >> 7;
    const float* p = us + (8 * ti + 2 * (lane & 3)) * (dvp + 4) + 16 * cb + (lane >> 2);
    U[i] = make_float4(p[0], p[dvp + 4], p[8], p[dvp + 4 + 8]);
  }
}

// ---------------------------------------------------------------- 2: the walk over the chunks
__device__ __forceinline__ uint32_t dc_tf32(float x) { uint32_t r; asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x)); return r; }
// x = hi + lo up to 2^-22 |x|, both tf32
__device__ __forceinline__ void dc_split(float x, uint32_t& hi, uint32_t& lo) {
  hi = dc_tf32(x);
  lo = dc_tf32(x - __uint_as_float(hi));
}
__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// An accumulator at 32-bit accuracy: the sum of the large products and, apart, of the two small ones, so that the three products
// of one tile do not wait for each other.
struct DcAcc { float x[4], c1[4], c2[4]; };
__device__ __forceinline__ void dc_clear(DcAcc& a) {
#pragma unroll
  for (int e = 0; e < 4; ++e) a.x[e] = a.c1[e] = a.c2[e] = 0.f;
}
__device__ __forceinline__ float dc_sum(const DcAcc& a, int e) { return a.x[e] + (a.c1[e] + a.c2[e]); }
__device__ __forceinline__ void dc_mma3(DcAcc& acc, const uint32_t (&ah)[4], const uint32_t (&al)[4], float b0, float b1) {
  uint32_t h0, l0, h1, l1;
  dc_split(b0, h0, l0);
  dc_split(b1, h1, l1);
  float d[4] = {0.f, 0.f, 0.f, 0.f};
  dc_mma(d, ah, h0, h1);
  dc_mma(acc.c1, ah, l0, l1);
  dc_mma(acc.c2, al, h0, h1);
#pragma unroll
  for (int e = 0; e < 4; ++e) acc.x[e] += d[e];
}
// the A fragment that an accumulator fragment is: positions t and t + 4 of its k index are columns 2 t and 2 t + 1
__device__ __forceinline__ void dc_operand(const float (&c)[4], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  dc_split(c[0], hi[0], lo[0]);
  dc_split(c[2], hi[1], lo[1]);
  dc_split(c[1], hi[2], lo[2]);
  dc_split(c[3], hi[3], lo[3]);
}

__global__ void __launch_bounds__(128)
dc_walk_kernel(const float* __restrict__ scratch, const int* __restrict__ cu_tokens, int num_seqs, int from, int places,
               const int* __restrict__ state_slots, float* __restrict__ state, long state_stride, int num_slots, float* __restrict__ o_out, int H, int dim, int dv, int dvp, int* err) {
  extern __shared__ __align__(16) float dw[];
  float* red = dw + DC_STAGES * DC_STAGE;              // [2][4 warps][8 tiles][32 lanes][4]
  const int cb = blockIdx.x, h = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  const Portion at = find_portion<true>(cu_tokens, num_seqs, from, DC, blockIdx.z);
  const int s = at.seq;
  if (s < 0) return;
  const int t0 = cu_tokens[s], ntok = cu_tokens[s + 1] - t0, chunks = (ntok + DC - 1) / DC;
  if (at.before + chunks > places) return;             // the caller counted other requests: nothing was formed for this one
  int slot = state_slots[s];
  if (slot >= num_slots) {
    if (tid == 0 && cb == 0) report_error(err, PHOTON_DEV_BAD_SLOT, t0, slot, num_slots);
    return;
  }
  float* S = slot >= 0 ? state + (size_t)slot * state_stride + (size_t)h * dim * dv : nullptr;
  const long per = dc_floats(dvp), step = per * H;
  const float* src0 = scratch + ((size_t)at.before * H + h) * per;

  // a thread's share of a chunk: 8 quads of W, of Q, of K, 2 of A, one of U0 (token tile w of the block's columns)
  auto fetch = [&](int c) {
    if (c < chunks) {
      const float* src = src0 + (size_t)c * step;
      float* d = dw + (c % DC_STAGES) * DC_STAGE;
      auto copy = [&](int at) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d + at)), "l"(src + at) : "memory");
      };
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int i = 0; i < 8; ++i) copy(m * DC_MAT + (w * 8 + i) * 128 + lane * 4);
      copy(3 * DC_MAT + (w * 2) * 128 + lane * 4);
      copy(3 * DC_MAT + (w * 2 + 1) * 128 + lane * 4);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                   ::"r"((uint32_t)__cvta_generic_to_shared(d + 3 * DC_MAT + DC * DC + w * 128 + lane * 4)),
                     "l"(src + 3 * DC_MAT + DC * DC + (cb * 4 + w) * 128 + lane * 4) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < DC_STAGES - 1; ++c) fetch(c);

  // S^T: tile j holds rows 32 w + 8 j + 2 t, + 1 of columns g and g + 8
  float st[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int row = 32 * w + 8 * j + 2 * t + (e & 1), col = cb * DC_CB + g + (e >> 1) * 8;
      st[j][e] = S != nullptr && row < dim && col < dv ? S[(size_t)row * dv + col] : 0.f;
    }
  for (int c = 0; c < chunks; ++c) {
    const float b_end = src0[(size_t)c * step + per - 4];
    asm volatile("cp.async.wait_group %0;" ::"n"(DC_STAGES - 2) : "memory");
    const float4* d4 = reinterpret_cast<const float4*>(dw + (c % DC_STAGES) * DC_STAGE) + lane;
    float4* r4 = reinterpret_cast<float4*>(red + (c & 1) * DC_RED) + lane;
    {
      // this warp's rows' share of W S0 (tiles 0 .. 3: tokens 8 i ..) and of diag(b) Q S0 (tiles 4 .. 7), the tiles side by side
      DcAcc acc[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) dc_clear(acc[i]);
#pragma unroll
      for (int j2 = 0; j2 < 2; ++j2) {
        uint32_t ah[2][4], al[2][4];
        dc_operand(st[2 * j2], ah[0], al[0]);
        dc_operand(st[2 * j2 + 1], ah[1], al[1]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 b = d4[(i >> 2) * (DC_MAT / 4) + (w * 8 + (i & 3) * 2 + j2) * 32];
          dc_mma3(acc[i], ah[0], al[0], b.x, b.y);
          dc_mma3(acc[i], ah[1], al[1], b.z, b.w);
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        r4[(w * 8 + i) * 32] = make_float4(dc_sum(acc[i], 0), dc_sum(acc[i], 1), dc_sum(acc[i], 2), dc_sum(acc[i], 3));
    }
    __syncthreads();                                   // the partial sums and U0 are there for every warp; the sums of the chunk before
    fetch(c + DC_STAGES - 1);                          // last are read no more, and neither is the stage that is filled now
    uint32_t uh[4][4], ul[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 u0 = d4[(3 * DC_MAT + DC * DC) / 4 + i * 32];
      const float4 p0 = r4[i * 32], p1 = r4[(8 + i) * 32], p2 = r4[(16 + i) * 32], p3 = r4[(24 + i) * 32];
      const float u[4] = {u0.x - ((p0.x + p1.x) + (p2.x + p3.x)), u0.y - ((p0.y + p1.y) + (p2.y + p3.y)),
                          u0.z - ((p0.z + p1.z) + (p2.z + p3.z)), u0.w - ((p0.w + p1.w) + (p2.w + p3.w))};
      dc_operand(u, uh[i], ul[i]);
    }
    // the outputs of tokens 8 w .. 8 w + 7 and this warp's rows of the state, side by side
    DcAcc out, nw[4];
    {
      const float4 p0 = r4[(4 + w) * 32], p1 = r4[(12 + w) * 32], p2 = r4[(20 + w) * 32], p3 = r4[(28 + w) * 32];
      dc_clear(out);
      out.x[0] = (p0.x + p1.x) + (p2.x + p3.x); out.x[1] = (p0.y + p1.y) + (p2.y + p3.y);
      out.x[2] = (p0.z + p1.z) + (p2.z + p3.z); out.x[3] = (p0.w + p1.w) + (p2.w + p3.w);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      dc_clear(nw[j]);
#pragma unroll
      for (int e = 0; e < 4; ++e) nw[j].x[e] = b_end * st[j][e];
    }
#pragma unroll
    for (int i2 = 0; i2 < 2; ++i2) {
      const float4 a = d4[3 * DC_MAT / 4 + (w * 2 + i2) * 32];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = 2 * i2 + u;
        const float4 k0 = d4[2 * DC_MAT / 4 + (w * 8 + i * 2) * 32], k1 = d4[2 * DC_MAT / 4 + (w * 8 + i * 2 + 1) * 32];
        dc_mma3(nw[0], uh[i], ul[i], k0.x, k0.y);
        dc_mma3(nw[1], uh[i], ul[i], k0.z, k0.w);
        dc_mma3(nw[2], uh[i], ul[i], k1.x, k1.y);
        dc_mma3(nw[3], uh[i], ul[i], k1.z, k1.w);
        dc_mma3(out, uh[i], ul[i], u ? a.z : a.x, u ? a.w : a.y);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) st[j][e] = dc_sum(nw[j], e);
    bool finite = true;
#pragma unroll
    for (int e = 0; e < 4; ++e) finite &= fabsf(dc_sum(out, e)) <= FLT_MAX;
    if (!__all_sync(0xffffffffu, finite)) {
      // A is zero for later tokens, but zero times their infinities is not.  The warp's outputs again: the tiles of earlier tokens,
      // then its own one, as a plain sum over the tokens that count if U is not finite there.
      {
        const float4 p0 = r4[(4 + w) * 32], p1 = r4[(12 + w) * 32], p2 = r4[(20 + w) * 32], p3 = r4[(28 + w) * 32];
        dc_clear(out);
        out.x[0] = (p0.x + p1.x) + (p2.x + p3.x); out.x[1] = (p0.y + p1.y) + (p2.y + p3.y);
        out.x[2] = (p0.z + p1.z) + (p2.z + p3.z); out.x[3] = (p0.w + p1.w) + (p2.w + p3.w);
      }
      const float4 u0 = d4[(3 * DC_MAT + DC * DC) / 4 + w * 32];
      const float4 p0 = r4[w * 32], p1 = r4[(8 + w) * 32], p2 = r4[(16 + w) * 32], p3 = r4[(24 + w) * 32];
      const float uw[4] = {u0.x - ((p0.x + p1.x) + (p2.x + p3.x)), u0.y - ((p0.y + p1.y) + (p2.y + p3.y)),
                           u0.z - ((p0.z + p1.z) + (p2.z + p3.z)), u0.w - ((p0.w + p1.w) + (p2.w + p3.w))};
      bool wild = false;
#pragma unroll
      for (int e = 0; e < 4; ++e) wild |= !(fabsf(uw[e]) <= FLT_MAX);
      wild = __any_sync(0xffffffffu, wild);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 q = d4[3 * DC_MAT / 4 + (w * 2 + (i >> 1)) * 32];
        if (i < w || (i == w && !wild)) dc_mma3(out, uh[i], ul[i], i & 1 ? q.z : q.x, i & 1 ? q.w : q.y);
      }
      // A [warp][s / 16][lane (t % 8) * 4 + (s % 8) / 2][(s % 16) / 8 * 2 + s % 2], s = 8 w + i
      const float* a = reinterpret_cast<const float*>(d4 - lane) + 3 * DC_MAT + (w * 2 + (w >> 1)) * 128 + (w & 1) * 2;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (!wild) break;
        const int from = (lane & ~3) | (i >> 1);
        const float u0 = __shfl_sync(0xffffffffu, uw[i & 1], from), u1 = __shfl_sync(0xffffffffu, uw[2 + (i & 1)], from);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int tt = 2 * t + (e & 1);
          if (i <= tt) out.x[e] = fmaf(a[(tt * 4 + (i >> 1)) * 4 + (i & 1)], e < 2 ? u0 : u1, out.x[e]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int tok = c * DC + 8 * w + 2 * t + (e & 1), col = cb * DC_CB + g + (e >> 1) * 8;
      if (tok < ntok && col < dv) o_out[(size_t)(t0 + tok) * H * dv + (size_t)h * dv + col] = dc_sum(out, e);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (S != nullptr) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = 32 * w + 8 * j + 2 * t + (e & 1), col = cb * DC_CB + g + (e >> 1) * 8;
        if (row < dim && col < dv) S[(size_t)row * dv + col] = st[j][e];
      }
  }
}

// Tokens of a chunk, and scratch floats of photon_delta_chunked for `chunks` of them.
PHOTON_API int photon_delta_chunk(void) { return DC; }
PHOTON_API long photon_delta_chunked_scratch(long chunks, int H, int dv) { return chunks * H * dc_floats((dv + 15) / 16 * 16); }

// As photon_delta_recurrent, for the requests that bring at least `from` tokens: `longs` of them, with `chunks` chunks of
// photon_delta_chunk tokens (the last one of a request may be short); the others are left alone.  scratch:
// photon_delta_chunked_scratch floats, 16-byte aligned.  dim up to 128, vdim up to 256.
PHOTON_API int photon_delta_chunked(const float* y, const void* ab, long ab_stride, int ab_dtype, const float* a_log, const float* dt_bias,
                                    const int* cu_tokens, const int* state_slots, float* state, long state_stride, int num_slots, float* o,
                                    float* scratch, int S, int from, int longs, int chunks, int Gq, int H, int dim, int vdim, int* err,
                                    cudaStream_t stream) {
  if (S <= 0 || longs <= 0 || chunks <= 0) return 0;
  if (Gq <= 0 || H <= 0 || H % Gq || dim <= 0 || vdim <= 0 || scratch == nullptr || ((uintptr_t)scratch & 15)) return PHOTON_ERR_ARGUMENT;
  if (ab_dtype != PHOTON_F32 && ab_dtype != PHOTON_BF16) return PHOTON_ERR_ARGUMENT;
  const int dvp = (vdim + 15) / 16 * 16;
  if (dim > DC_D || vdim > 256 || longs > 65535 || H > 65535) return PHOTON_ERR_UNSUPPORTED;
  const size_t smem1 = ((size_t)2 * DC * DP_LD + DC * (DC + 4) + DC * (dvp + 4)) * sizeof(float);
  const size_t smem2 = ((size_t)DC_STAGES * DC_STAGE + 2 * DC_RED) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(dc_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(dc_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2);
  if (e != cudaSuccess) return (int)e;
  dc_prep_kernel<<<dim3(chunks, H), 256, smem1, stream>>>(y, ab, ab_stride, ab_dtype == PHOTON_BF16, a_log, dt_bias, cu_tokens, S, from, scratch, Gq,
                                                          H, dim, vdim, dvp);
  const int st = launch_status();
  if (st != 0) return st;
  dc_walk_kernel<<<dim3(dvp / DC_CB, H, longs), 128, smem2, stream>>>(scratch, cu_tokens, S, from, chunks, state_slots, state, state_stride, num_slots, o, H,
                                                                      dim, vdim, dvp, err);
  return launch_status();
}
