// Gated linear attention: a recurrent mixer whose state is one matrix per head, S [dim][vdim] in 32-bit.
// With a decay per key channel a_t = sigmoid(z_t)^(1/tau) (computed as exp(log_sigmoid(z_t) / tau)), whose
// logits are the second half of a low-rank projection, z_t = W_a2 low_t + b (low_t = W_a1 h_t comes in with
// q, k, v and g; the few multiply-adds per channel are done here, in 32-bit),
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T,        o_t = S_t^T (q_t * qscale),
//
// and the head's output is o_t divided by its root mean square over vdim (eps inside the root), times a
// weight shared by the heads, times silu(g_t).  One block owns one (request, head): it reads the state from
// the request's slot, walks the request's tokens of this step in order, and writes the state back, so a
// prompt portion, a single decoded token and a mixed batch are the same case, and a request's result does not
// depend on how it was cut into steps (the per-token arithmetic is the same chain either way).
//
// Thread r * vdim + j holds the state rows r * RPT .. r * RPT + RPT - 1 of value column j in registers; the partial
// sums over rows meet in shared memory in the order of r.  q, k and the decay of the next token are fetched
// while the current one is computed.  Everything is 32-bit; q, k, v and g may be stored as bfloat16.
#include "common.cuh"
#include <math.h>

// Rows of the state per thread and the block's width: as few rows as keep the block within 256 threads (then a
// thread may use 255 registers and nothing spills), else within 512.
static inline void gla_shape(int dim, int vdim, int* rpt, int* maxt) {
  // the narrowest block that holds the state with at most 64 rows a thread: 256 threads may use 255 registers each
  // and nothing spills.  Measured at heads of 128 x 128: blocks of 256, 512 and 1024 threads take the same time.
  for (int limit = 256; limit <= 1024; limit *= 2) {
    for (int r = 8; r <= 64; r *= 2) {
      if ((long)vdim * ((dim + r - 1) / r) <= limit && dim <= limit) { *rpt = r; *maxt = limit; return; }
    }
  }
  *rpt = 64; *maxt = 1024;                               // refused by the launcher when it does not fit
}

// skip_from > 0: requests that bring that many tokens or more are left alone.
template <typename T, int RPT, int MAXT>
__global__ void __launch_bounds__(MAXT) gla_recurrent_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                                     const T* __restrict__ g, const T* __restrict__ low, long in_stride, int rank,
                                     const T* __restrict__ w_a2, const void* __restrict__ b_a2, int b_bf16,
                                     const void* __restrict__ norm_w, int norm_w_bf16, float eps, float inv_tau,
                                     float qscale, const int* __restrict__ cu_tokens,
                                     const int* __restrict__ state_slots, float* __restrict__ state, int num_slots,
                                     T* __restrict__ out, long out_stride, int heads, int dim, int vdim, int* err,
                                     int skip_from) {
  extern __shared__ float sm[];
  const int s = blockIdx.x, h = blockIdx.y;
  const int R = (dim + RPT - 1) / RPT;
  const int tid = threadIdx.x, nthreads = blockDim.x;                       // a whole number of warps
  const bool active = tid < vdim * R;                                        // the others only meet at barriers
  const int j = active ? tid % vdim : 0, r = active ? tid / vdim : R;
  const int dimp = R * RPT;              // rows padded to whole groups: the padding stays zero and adds nothing
  float* qs = sm;                        // 2 x dimp
  float* ks = qs + 2 * dimp;             // 2 x dimp
  float* as = ks + 2 * dimp;             // 2 x dimp
  float* part = as + 2 * dimp;           // R x vdim
  float* red = part + R * vdim;          // 32
  float* wa = red + 32;                  // dim x (rank + 1): this head's rows of W_a2
  float* ba = wa + dim * (rank + 1);     // dim
  const int t0 = cu_tokens[s], t1 = cu_tokens[s + 1];
  if (t1 <= t0 || (skip_from > 0 && t1 - t0 >= skip_from)) return;        // long portions go the chunked way
  const int slot = state_slots[s];
  if (slot >= num_slots) {
    if (tid == 0) report_error(err, PHOTON_DEV_BAD_SLOT, t0, slot, num_slots);
    return;
  }
  float* S = slot >= 0 ? state + ((size_t)slot * heads + h) * dim * vdim : nullptr;
  float st[RPT];
  const int row0 = r * RPT;
#pragma unroll
  for (int i = 0; i < RPT; ++i) st[i] = (S != nullptr && active && row0 + i < dim) ? S[(size_t)(row0 + i) * vdim + j] : 0.f;
  const float wj = load_w(norm_w, norm_w_bf16, j);
  for (int i = tid; i < 6 * dimp; i += nthreads) sm[i] = 0.f;
  for (int i = tid; i < dim * rank; i += nthreads) wa[(i / rank) * (rank + 1) + i % rank] = to_f32(w_a2[(size_t)h * dim * rank + i]);
  for (int i = tid; i < dim; i += nthreads) ba[i] = load_w(b_a2, b_bf16, (size_t)h * dim + i);
  __syncthreads();

  // Two tokens ahead: the raw q, k and low-rank row of token t + 1 wait in registers while token t is computed, and
  // become the decayed inputs in shared memory right before they are needed; v and g of the next token likewise.
  // A block has at least `dim` threads, so thread i < dim owns decay channel i.
  constexpr int LR = MAXT >= 1024 ? 8 : 16;              // low-rank values kept in registers; more are read late
  const bool owner = tid < dim;
  float rq = 0.f, rk = 0.f, rl[LR];
  auto load = [&](int t) {
    if (!owner) return;
    const size_t off = (size_t)t * in_stride + (size_t)h * dim + tid;
    rq = to_f32(q[off]);
    rk = to_f32(k[off]);
    const T* lw = low + (size_t)t * in_stride;
#pragma unroll
    for (int c = 0; c < LR; ++c) rl[c] = c < rank ? to_f32(lw[c]) : 0.f;
  };
  auto commit = [&](int t, int buf) {
    if (!owner) return;
    const int i = tid;
    float zz = 0.f;
#pragma unroll
    for (int c = 0; c < LR; ++c) if (c < rank) zz = fmaf(rl[c], wa[i * (rank + 1) + c], zz);
    const T* lw = low + (size_t)t * in_stride;
    for (int c = LR; c < rank; ++c) zz = fmaf(to_f32(lw[c]), wa[i * (rank + 1) + c], zz);
    zz += ba[i];
    const float ls = fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)));            // log(sigmoid(z))
    const float a = expf(ls * inv_tau);
    qs[buf * dimp + i] = rq * qscale;
    ks[buf * dimp + i] = rk;
    as[buf * dimp + i] = a;
  };
  load(t0);
  commit(t0, 0);
  if (t0 + 1 < t1) load(t0 + 1);
  float vj = to_f32(v[(size_t)t0 * in_stride + (size_t)h * vdim + j]);
  float gj = to_f32(g[(size_t)t0 * in_stride + (size_t)h * vdim + j]);
  __syncthreads();
  for (int t = t0; t < t1; ++t) {
    const int buf = (t - t0) & 1;
    if (t + 1 < t1) commit(t + 1, buf ^ 1);              // its raw values arrived during the last token
    if (t + 2 < t1) load(t + 2);
    const float vcur = vj, gcur = gj;
    if (t + 1 < t1) {
      vj = to_f32(v[(size_t)(t + 1) * in_stride + (size_t)h * vdim + j]);
      gj = to_f32(g[(size_t)(t + 1) * in_stride + (size_t)h * vdim + j]);
    }
    float o = 0.f;
    if (active) {
      // a thread's rows lie side by side: four decays, keys and queries per shared-memory read
      const float4* qb = reinterpret_cast<const float4*>(qs + buf * dimp + row0);
      const float4* kb = reinterpret_cast<const float4*>(ks + buf * dimp + row0);
      const float4* ab = reinterpret_cast<const float4*>(as + buf * dimp + row0);
      float o2 = 0.f;
#pragma unroll
      for (int i = 0; i < RPT / 4; ++i) {
        const float4 a4 = ab[i], k4 = kb[i], q4 = qb[i];
        st[4 * i] = fmaf(a4.x, st[4 * i], k4.x * vcur);
        st[4 * i + 1] = fmaf(a4.y, st[4 * i + 1], k4.y * vcur);
        st[4 * i + 2] = fmaf(a4.z, st[4 * i + 2], k4.z * vcur);
        st[4 * i + 3] = fmaf(a4.w, st[4 * i + 3], k4.w * vcur);
        o = fmaf(st[4 * i], q4.x, o);
        o2 = fmaf(st[4 * i + 1], q4.y, o2);
        o = fmaf(st[4 * i + 2], q4.z, o);
        o2 = fmaf(st[4 * i + 3], q4.w, o2);
      }
      o += o2;
      part[r * vdim + j] = o;
    }
    __syncthreads();
    float tot = 0.f, sq = 0.f;
    if (r == 0) {
      for (int rr = 0; rr < R; ++rr) tot += part[rr * vdim + j];
      sq = tot * tot;
    }
    sq = block_sum(sq, red);                               // two barriers inside: `part` and the next token's
    if (r == 0) {                                          // q, k and decay are settled when it returns
      const float inv = 1.0f / sqrtf(sq / (float)vdim + eps);
      out[(size_t)t * out_stride + (size_t)h * vdim + j] = from_f32<T>(tot * inv * wj * (gcur / (1.0f + expf(-gcur))));
    }
  }
  if (S != nullptr && active) {
#pragma unroll
    for (int i = 0; i < RPT; ++i)
      if (row0 + i < dim) S[(size_t)(row0 + i) * vdim + j] = st[i];
  }
}

// ---------------------------------------------------------------- the inputs of a long portion
// Long portions run in segments (linrec_segments.cu, which walks 32-bit rows): q, k, v and the decays of all tokens as float,
// two channels a thread, GP_TOK tokens a block, whose low-rank rows wait in shared memory.  Bound by memory: it reads 2 bytes and
// writes 4 per number (16 heads of 128 x 128, 2,048 tokens: 92 MB).
#define GP_TOK 16
#define GP_RANK 8                                        // low-rank columns whose weights a thread holds at a time

__device__ __forceinline__ float2 gp_load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 gp_load2(const bf16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }

template <typename T, bool PAIRS>
__global__ void __launch_bounds__(128)
gla_prep_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, const T* __restrict__ low, long in_stride,
                int rank, const T* __restrict__ w_a2, const void* __restrict__ b_a2, int b_bf16, float inv_tau,
                float* __restrict__ q_out, float* __restrict__ k_out, float* __restrict__ v_out, float* __restrict__ a_out,
                long out_stride, int tokens, int nd, int nv, int nd_blocks) {
  extern __shared__ float gp_low[];                      // [GP_TOK][rank]
  const int t0 = blockIdx.y * GP_TOK, n = min(GP_TOK, tokens - t0);
  if ((int)blockIdx.x >= nd_blocks) {
    const int c = ((int)blockIdx.x - nd_blocks) * 256 + threadIdx.x * 2;
    if (PAIRS) {
      if (c < nv) {
#pragma unroll 8
        for (int t = 0; t < n; ++t)
          *reinterpret_cast<float2*>(v_out + (size_t)(t0 + t) * out_stride + c) = gp_load2(v + (size_t)(t0 + t) * in_stride + c);
      }
      return;
    }
    for (int t = 0; t < n; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (c + e < nv) v_out[(size_t)(t0 + t) * out_stride + c + e] = to_f32(v[(size_t)(t0 + t) * in_stride + c + e]);
    return;
  }
  for (int i = threadIdx.x; i < n * rank; i += 128) gp_low[i] = to_f32(low[(size_t)(t0 + i / rank) * in_stride + i % rank]);
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x * 2;
  if (c >= nd) return;
  float z[GP_TOK][2];
#pragma unroll
  for (int t = 0; t < GP_TOK; ++t) z[t][0] = z[t][1] = 0.f;
  for (int r0 = 0; r0 < rank; r0 += GP_RANK) {
    float w[2][GP_RANK];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int r = 0; r < GP_RANK; ++r) w[e][r] = c + e < nd && r0 + r < rank ? to_f32(w_a2[(size_t)(c + e) * rank + r0 + r]) : 0.f;
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) {
      if (t < n) {
#pragma unroll
        for (int r = 0; r < GP_RANK; ++r) {
          if (r0 + r < rank) {
            const float x = gp_low[t * rank + r0 + r];
            z[t][0] = fmaf(x, w[0][r], z[t][0]);
            z[t][1] = fmaf(x, w[1][r], z[t][1]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (c + e >= nd) break;
    const float bias = load_w(b_a2, b_bf16, c + e);
#pragma unroll
    for (int t = 0; t < GP_TOK; ++t) {
      if (t < n) {
        const float zz = z[t][e] + bias;
        const float ls = fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)));            // log(sigmoid(z))
        z[t][e] = expf(ls * inv_tau);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < GP_TOK; ++t) {
    if (t < n) {
      const size_t in = (size_t)(t0 + t) * in_stride + c, at = (size_t)(t0 + t) * out_stride + c;
      if (PAIRS) {
        *reinterpret_cast<float2*>(q_out + at) = gp_load2(q + in);
        *reinterpret_cast<float2*>(k_out + at) = gp_load2(k + in);
        *reinterpret_cast<float2*>(a_out + at) = make_float2(z[t][0], z[t][1]);
        continue;
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (c + e < nd) { q_out[at + e] = to_f32(q[in + e]); k_out[at + e] = to_f32(k[in + e]); a_out[at + e] = z[t][e]; }
      }
    }
  }
}

// q, k [T][heads * dim], v [T][heads * vdim], low [T][rank]: sections of one fused row of `dtype`.  q_out, k_out, a_out float
// [T][heads * dim], v_out float [T][heads * vdim], one row stride: the same numbers in 32-bit, and the decays
// exp(log_sigmoid(w_a2 low + b_a2) / tau).
PHOTON_API int photon_gla_prep(const void* q, const void* k, const void* v, const void* low, long in_stride, int dtype, int rank,
                               const void* w_a2, const void* b_a2, int b_a2_dtype, float tau, float* q_out, float* k_out, float* v_out,
                               float* a_out, long out_stride, int T, int nd, int nv, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (nd <= 0 || nv <= 0 || rank <= 0 || !(tau > 0.f)) return PHOTON_ERR_ARGUMENT;
  const int rows = (T + GP_TOK - 1) / GP_TOK;
  const size_t smem = (size_t)GP_TOK * rank * sizeof(float);
  if (rows > 65535 || smem > 48 * 1024) return PHOTON_ERR_UNSUPPORTED;
  const int nb = (nd + 255) / 256, bb = b_a2_dtype == PHOTON_BF16;
  const dim3 grid(nb + (nv + 255) / 256, rows);
  const float it = 1.0f / tau;
  // pairs of numbers at a time where all of them lie on their boundaries
  const uintptr_t ia = dtype == PHOTON_BF16 ? 3 : 7;
  const bool pairs = nd % 2 == 0 && nv % 2 == 0 && in_stride % 2 == 0 && out_stride % 2 == 0 && ((uintptr_t)q & ia) == 0 && ((uintptr_t)k & ia) == 0 &&
                     ((uintptr_t)v & ia) == 0 && ((uintptr_t)q_out & 7) == 0 && ((uintptr_t)k_out & 7) == 0 && ((uintptr_t)v_out & 7) == 0 &&
                     ((uintptr_t)a_out & 7) == 0;
#define GP_GO(TY, P) gla_prep_kernel<TY, P><<<grid, 128, smem, stream>>>((const TY*)q, (const TY*)k, (const TY*)v, (const TY*)low, in_stride, rank, \
    (const TY*)w_a2, b_a2, bb, it, q_out, k_out, v_out, a_out, out_stride, T, nd, nv, nb)
  if (dtype == PHOTON_BF16) { if (pairs) GP_GO(bf16, true); else GP_GO(bf16, false); }
  else if (dtype == PHOTON_F32) { if (pairs) GP_GO(float, true); else GP_GO(float, false); }
  else return PHOTON_ERR_ARGUMENT;
  return launch_status();
}

template <typename T, int RPT, int MAXT>
static int gla_launch(const void* q, const void* k, const void* v, const void* g, const void* low, long in_stride,
                      int rank, const void* w_a2, const void* b_a2, int b_bf16, const void* norm_w, int norm_w_bf16, float eps, float inv_tau, float qscale,
                      const int* cu_tokens, const int* state_slots, float* state, int num_slots, void* out,
                      long out_stride, int S, int heads, int dim, int vdim, int* err, cudaStream_t stream, int skip_from) {
  const int R = (dim + RPT - 1) / RPT;
  if (vdim * R > MAXT) return PHOTON_ERR_UNSUPPORTED;
  const size_t smem = ((size_t)6 * R * RPT + dim + (size_t)R * vdim + 32 + (size_t)dim * (rank + 1)) * sizeof(float);
  if (smem > 200 * 1024) return PHOTON_ERR_UNSUPPORTED;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(gla_recurrent_kernel<T, RPT, MAXT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  int threads = (vdim * R + 31) / 32 * 32;
  if (threads < dim) threads = (dim + 31) / 32 * 32;                  // thread i < dim owns decay channel i
  if (threads > MAXT) return PHOTON_ERR_UNSUPPORTED;
  gla_recurrent_kernel<T, RPT, MAXT><<<dim3(S, heads), dim3(threads), smem, stream>>>(
      (const T*)q, (const T*)k, (const T*)v, (const T*)g, (const T*)low, in_stride, rank, (const T*)w_a2, b_a2, b_bf16,
      norm_w, norm_w_bf16, eps, inv_tau,
      qscale, cu_tokens, state_slots, state, num_slots, (T*)out, out_stride, heads, dim, vdim, err, skip_from);
  return launch_status();
}

// q, k [T][heads * dim], v, g [T][heads * vdim], low [T][rank]: sections of one fused row (one row stride, in
// elements).  w_a2 [heads * dim][rank] (the type of q), b_a2 [heads * dim]: the decay logits are w_a2 low + b_a2.  state [num_slots][heads][dim][vdim] float; a request whose slot
// is negative starts from zero and stores nothing.  out [T][heads * vdim].
PHOTON_API int photon_gla_recurrent(const void* q, const void* k, const void* v, const void* g, const void* low,
                                    long in_stride, int dtype, int rank, const void* w_a2, const void* b_a2,
                                    int b_a2_dtype, const void* norm_w, int norm_w_dtype,
                                    float eps, float tau, float qscale, const int* cu_tokens, const int* state_slots,
                                    float* state, int num_slots, void* out, long out_stride, int S, int heads, int dim,
                                    int vdim, int skip_from, int* err, cudaStream_t stream) {
  if (S <= 0) return 0;
  if (heads <= 0 || dim <= 0 || vdim <= 0 || rank <= 0 || !(tau > 0.f)) return PHOTON_ERR_ARGUMENT;
  const int bb = b_a2_dtype == PHOTON_BF16;
  if (heads > 65535) return PHOTON_ERR_UNSUPPORTED;
  const int wb = norm_w_dtype == PHOTON_BF16;
  const float it = 1.0f / tau;
  int rpt = 0, maxt = 256;
  gla_shape(dim, vdim, &rpt, &maxt);
#define GLA_ARGS q, k, v, g, low, in_stride, rank, w_a2, b_a2, bb, norm_w, wb, eps, it, qscale, cu_tokens, state_slots, state, \
                 num_slots, out, out_stride, S, heads, dim, vdim, err, stream
#define GLA_DISPATCH_T(MAXT)                                                      \
  if (dtype == PHOTON_BF16) {                                                     \
    if (rpt == 8) return gla_launch<bf16, 8, MAXT>(GLA_ARGS, skip_from);          \
    if (rpt == 16) return gla_launch<bf16, 16, MAXT>(GLA_ARGS, skip_from);        \
    if (rpt == 32) return gla_launch<bf16, 32, MAXT>(GLA_ARGS, skip_from);        \
    return gla_launch<bf16, 64, MAXT>(GLA_ARGS, skip_from);                       \
  }                                                                               \
  if (rpt == 8) return gla_launch<float, 8, MAXT>(GLA_ARGS, skip_from);           \
  if (rpt == 16) return gla_launch<float, 16, MAXT>(GLA_ARGS, skip_from);         \
  if (rpt == 32) return gla_launch<float, 32, MAXT>(GLA_ARGS, skip_from);         \
  return gla_launch<float, 64, MAXT>(GLA_ARGS, skip_from);
  if (maxt == 1024) { GLA_DISPATCH_T(1024) }
  if (maxt == 512) { GLA_DISPATCH_T(512) }
  GLA_DISPATCH_T(256)
}
