// The recurrences of linrec.cu (and gated linear attention's) over long prompt portions, cut into segments of tokens that run
// side by side.
//
//   S_t = keep_t S_(t-1) + take_t k_t v_t^T        modes 0 (state space) and 1 (matrix memory): one number per head and token
//   S_t = S_(t-1) + k_t (v_t^T - S_(t-1))           mode 2 (forget and write): a number per row
//   S_t = diag(a_t) S_(t-1) + k_t v_t^T             mode 3 (gated linear attention): a number per row
//
// The update is linear in the state, so a segment's end is (its decay) x (its start) + (its end from a zero start).
// The requests' segments stand one behind the other in the grid, a request of few tokens is one segment; only requests of several
// have room in scratch.
//   1. ls_gates_kernel (modes 0, 1): the gates of all tokens, and what a segment does to the scale of the state.
//   2. the walk, first pass: every segment but the last, from zero (the first from the request's state), keeps its
//      end state and its decay in scratch.  No queries.
//   3. the walk, second pass: every segment folds the ends before it into its start state, in their order, and walks
//      its tokens again with the queries; the last one leaves the state in the request's slot.
// Mode 1's running maximum only sets the scale in which S and n are held: with F the sum of the forget gates since the
// segment's start and L the running maximum from nothing, m_t = max(F_t + m_start, L_t), so both come from one scan per
// segment, and keep_t = exp(f_t + (m_(t-1) - m_t)) holds whatever the last bits of m are.
//
// Everything is 32-bit as in the token-by-token kernels; what differs is the scale in which a chunk's state is held (below) and
// the fold (one multiply-add per segment and state element, two where the decay is one number per row).  Decays near 1 are
// carried by what they lack to 1 (lr_decay).  Error of the state against 64 bits, 2,048 tokens, token by token in brackets:
// write gates of 1e-5 to 1e-2 that hardly change 2.3e-7 (3.3e-7), of 0.01 to 0.5 6.2e-8 (5.2e-8); row decays of 0.999 to
// 0.9999 2.9e-7 (1.0e-6), of 0.96 1.2e-7 (1.4e-7).  With products of rounded decays the first was 5.8e-6, the third 2.7e-6.
//
// What bounds it: the FP32 pipe.  A packed multiply-add with three operands takes three cycles and a packed product two, so
// the decay is taken out of the walk: over a chunk of 16 tokens the state is held relative to the product b_t of the decays
// since the chunk's start, S_t = b_t Z_t with Z_t = Z_(t-1) + (k_t / b_t) v_t^T and o_t = Z_t^T (b_t q_t), which leaves one
// multiply-add for the update and one for the read-out per token and pair, and one product per pair and chunk.  A chunk
// whose decays multiply to less than LS_SMALL (1 / b_t would leave the comfortable range) walks the plain form.
// A lane owns 8 rows x 8 columns, so that the reads of keys and queries, the copies and the barriers of a chunk are shared by 32
// packed multiply-adds a token (with 4 columns a lane the second pass issued 107 instructions a token and warp, of which
// 32 were multiply-adds, and its FP32 pipe was busy 42 % of the time).  The walk of one request then has 32 blocks of four
// warps at 16 heads of 128 x 128; the portion is cut into as many segments as give the GPU LS_BLOCKS_PER_SM blocks an SM.
// Measured, heads of 128 x 128 (gates, both passes): state space, 16 heads, 2,048 tokens 379 -> 153 us; matrix memory, two requests of
// 2,815 tokens 411 -> 234 us; forget and write 240 -> 155 us (777 tokens 94 -> 77 us); gated linear attention 416 us (chunks of
// 32 tokens joined by a scan) -> 156 us and 37 us for its inputs.  That was before decays near 1 were carried by what they lack to
// 1, which takes 3 to 7 % of a mixer's step (2,048 tokens of 16 heads: gated linear attention 281 -> 300 us, state space 277 -> 284;
// two requests of 2,815, matrix memory 365 -> 380; 777 tokens, forget and write 136 -> 143).  Half of the time is the FP32 pipe; the rest is the barriers of a
// chunk, the folds and the blocks' start, which two or three blocks an SM hide equally (100 us either way for the second pass).
#include "linrec.cuh"
#include "portions.cuh"

#define LS_CHUNK 16
#define LS_THREADS 128
#define LS_BLOCKS_PER_SM 2
#define LS_C 8                  // columns of a lane
#define LS_SMALL 0x1p-40f

struct alignas(16) LsCols { float x[LS_C]; };        // the lane's columns of one row

__device__ __forceinline__ lr_pair ls_mask2(float c0, float c1) { return (lr_pair)lr_mask(c1) << 32 | lr_mask(c0); }

struct LsArgs {
  const float* q; long q_stride;                     // [T][qk_heads * N]
  const float* k; long k_stride;                     // [T][qk_heads * N]: keys; mode 2: write gates
  const float* v; long v_stride;                     // [T][H * dv]
  const float* a; long a_stride;                     // mode 3: [T][qk_heads * N] decays
  const float* gates;                                // modes 0, 1: planes [T][H]: keep, take | f, i, F, L
  const float* d_skip;                               // mode 0: [H]
  float q_scale;
  const int* cu_tokens;
  const int* state_slots;
  float* state; long state_stride; int num_slots;
  float* out; long out_stride;                       // [T][H * dv]; mode 1: before the division
  float* den;                                        // mode 1: [T][H], what the outputs are to be divided by
  float* ends;                                       // [cut_segs][H][N * dv]: the requests of several segments
  float* vecs;                                       // [cut_segs][H][N]: mode 1 n at the end; modes 2, 3 the rows' decay (lr_code)
  float* scale;                                      // [segs][H][2]: mode 0 the decay; mode 1 F and L at the end
  float* first;                                      // [cuts][H][N * dv], then [cuts][H][N]: the state of those requests before the step
  float* first_m;                                    // [S][H]: mode 1, the running maximum before the step
  int T, S, H, qk_heads, N, dv, seg, segs, cuts, cut_segs, vec;
  int* err;
};

// ---------------------------------------------------------------- 1: gates
// A warp per (segment, head), 32 tokens at a time.  The sum over a segment is 64-bit.
template <int MODE>
__global__ void __launch_bounds__(128)
ls_gates_kernel(const float* __restrict__ ga, const float* __restrict__ gb, long g_stride, const float* __restrict__ p0,
                const float* __restrict__ p1, float cap, float* __restrict__ gates, LsArgs A) {
  const int lane = threadIdx.x & 31;
  const int h = blockIdx.y * 4 + (threadIdx.x >> 5);
  const Portion place = find_portion<false>(A.cu_tokens, A.S, 1, A.seg, blockIdx.x);
  const int s = place.seq, sg = (int)blockIdx.x - place.before;
  if (h >= A.H || s < 0) return;
  const int t0 = A.cu_tokens[s], t1 = A.cu_tokens[s + 1];
  const int b0 = t0 + sg * A.seg, b1 = min(t1, b0 + A.seg);
  const size_t TH = (size_t)A.T * A.H;
  if (MODE == 1 && sg == 0 && lane == 0) {
    const int slot = A.state_slots[s];
    A.first_m[(size_t)s * A.H + h] =
        slot >= 0 && slot < A.num_slots ? A.state[(size_t)slot * A.state_stride + (size_t)A.H * A.N * (A.dv + 1) + h] : 0.f;
  }
  const float a_h = MODE == 0 ? expf(p0[h]) : 0.f;
  double sum = 0.0;                                  // of dt or f over the segment's tokens before these 32
  float last = -INFINITY;                            // mode 1: L at the token before these 32
  float x = 0.f, y = 0.f;
  auto fetch = [&](int t) {
    x = 0.f; y = 0.f;
    if (t < b1) {
      x = ga[(size_t)t * g_stride + h];
      if (MODE == 1) y = gb[(size_t)t * g_stride + h];
    }
  };
  fetch(b0 + lane);
  for (int t = b0; t < b1; t += 32) {
    const bool live = t + lane < b1;
    const size_t at = (size_t)(t + lane) * A.H + h;
    const float xi = x, yi = y;
    fetch(t + 32 + lane);                            // the next 32 tokens' gates are on their way
    if (MODE == 0) {
      const float dt = live ? lr_softplus(xi + p1[h]) : 0.f;
      if (live) { gates[at] = expf(-a_h * dt); gates[TH + at] = dt; }
      sum += warp_sum(dt);
    } else {
      const float gi = cap * tanhf((xi + p0[h]) / cap);                             // log input gate
      const float gf = live ? lr_logsigmoid(cap * tanhf((yi + p1[h]) / cap)) : 0.f;  // log forget gate
      float F = gf;                                  // since the first of these 32; tokens behind the segment add nothing
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, F, o);
        if (lane >= o) F += up;
      }
      float d = live ? gi - F : -INFINITY;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, d, o);
        if (lane >= o) d = fmaxf(d, up);
      }
      const float Lt = F + fmaxf(d, last);
      if (live) { gates[at] = gf; gates[TH + at] = gi; gates[2 * TH + at] = (float)(sum + F); gates[3 * TH + at] = Lt; }
      sum += __shfl_sync(0xffffffffu, F, 31);
      last = __shfl_sync(0xffffffffu, Lt, 31);
    }
  }
  if (lane == 0) {
    float* sc = A.scale + ((size_t)blockIdx.x * A.H + h) * 2;
    sc[0] = MODE == 0 ? expf((float)(-(double)a_h * sum)) : (float)sum;
    sc[1] = last;
  }
}

// ---------------------------------------------------------------- 2 and 3: the walk
// A lane owns R rows x LS_C columns of the state as pairs of neighbouring rows, L lanes share the columns (lane i of them holds
// rows (j L + i) 4 .. + 3), a block of four warps 4 * LS_C * 32 / L neighbouring columns of one (segment, head).  Vectors that
// follow the rows are kept by a thread per row: n (mode 1, with n . q per token in the second pass) and, in the first pass of
// modes 2 and 3, the rows' decay; the block of the head's first columns writes them.
template <int MODE, int L, int R, int PASS>
__global__ void __launch_bounds__(LS_THREADS, LS_BLOCKS_PER_SM)
ls_walk_kernel(const LsArgs A) {
  constexpr int NP = L * R;                            // rows, padded
  constexpr int BC = 4 * LS_C * (32 / L);              // columns of a block
  constexpr int RT = (NP + LS_THREADS - 1) / LS_THREADS;     // rows of a thread that follows rows
  constexpr int TG = 2;                                // tokens at a time
  constexpr bool HAS_Q = PASS == 2, HAS_A = MODE == 3, SCALAR = MODE < 2;
  extern __shared__ __align__(16) float ls_smem[];
  float* ks = ls_smem;                                 // [2][CHUNK][NP]
  float* qs = ks + 2 * LS_CHUNK * NP;                  // [2][CHUNK][NP], second pass
  float* as = qs + (HAS_Q ? 2 * LS_CHUNK * NP : 0);    // [2][CHUNK][NP], mode 3
  float* vs = as + (HAS_A ? 2 * LS_CHUNK * NP : 0);    // [2][CHUNK][BC]
  float* os = vs + 2 * LS_CHUNK * BC;                  // [CHUNK][BC], second pass
  __shared__ float keep_s[LS_CHUNK], take_s[LS_CHUNK], floor_s[LS_CHUNK], by_s[LS_CHUNK];
  __shared__ __align__(16) float end_s[MODE < 2 ? 4 : NP];    // the decay through the chunk (lr_code), modes 2 and 3 per row
  __shared__ int plain_s;
  __shared__ float den_s[4][LS_CHUNK];
  const int N = A.N, dv = A.dv, H = A.H;
  const Portion place = find_portion<false>(A.cu_tokens, A.S, 1, A.seg, blockIdx.z);
  const int s = place.seq, sg = (int)blockIdx.z - place.before;
  if (s < 0) return;
  const int t0 = A.cu_tokens[s], t1 = A.cu_tokens[s + 1];
  const int nseg = (t1 - t0 + A.seg - 1) / A.seg;
  if (PASS == 1 && sg == nseg - 1) return;
  // a caller that counted other requests than cu_tokens holds has made no room for them
  if (nseg > 1 && (place.cut_rank >= A.cuts || place.cut_before + nseg > A.cut_segs)) return;
  const int b0 = t0 + sg * A.seg, b1 = min(t1, b0 + A.seg);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sub = lane & (L - 1);
  const int col = (warp * (32 / L) + lane / L) * LS_C;   // the lane's first column within the block
  const int h = blockIdx.y;
  const bool leads = blockIdx.x == 0;                  // this block keeps the vectors
  const int c0 = blockIdx.x * BC;
  const int ncol = min(BC, dv - c0);
  const int hq = h / (H / A.qk_heads);
  int slot = A.state_slots[s];
  if (slot >= A.num_slots) {
    if (PASS == 2 && tid == 0 && blockIdx.x == 0 && h == 0 && sg == 0) report_error(A.err, PHOTON_DEV_BAD_SLOT, s, slot, A.num_slots);
    slot = -1;
  }
  float* row0 = slot >= 0 ? A.state + (size_t)slot * A.state_stride : nullptr;
  float* S_h = row0 ? row0 + (size_t)h * N * dv : nullptr;
  float* n_h = row0 ? row0 + (size_t)H * N * dv + (size_t)h * N : nullptr;           // mode 1
  const size_t SH = (size_t)A.cuts * H, sh = (size_t)place.cut_rank * H + h;
  auto seg_at = [&](int i) { return (size_t)(place.cut_before + i) * H + h; };                         // the request's segment i in scratch
  auto scale_at = [&](int i) { return A.scale + ((size_t)(place.before + i) * H + h) * 2; };
  float* first_S = A.first + sh * N * dv;
  float* first_n = A.first + SH * N * dv + sh * N;
  const bool wide = A.vec && c0 + col + LS_C <= dv;   // all of the lane's columns at a time

  // the lane's share of a matrix [N][dv]: rows row_of(j, e), columns c0 + col ..
  auto row_of = [&](int j, int e) { return ((j >> 1) * L + sub) * 4 + (j & 1) * 2 + e; };
  auto load = [&](const float* m, int j, int e, float (&x)[LS_C]) {
    const int r = row_of(j, e);
#pragma unroll
    for (int c = 0; c < LS_C; ++c) x[c] = 0.f;
    if (m == nullptr || r >= N) return;
    const float* src = m + (size_t)r * dv + c0 + col;
    if (wide) {
      const LsCols f = *reinterpret_cast<const LsCols*>(src);
#pragma unroll
      for (int c = 0; c < LS_C; ++c) x[c] = f.x[c];
    } else {
#pragma unroll
      for (int c = 0; c < LS_C; ++c) if (c0 + col + c < dv) x[c] = src[c];
    }
  };
  auto store = [&](float* m, int j, int e, const float (&x)[LS_C]) {
    const int r = row_of(j, e);
    if (m == nullptr || r >= N) return;
    float* dst = m + (size_t)r * dv + c0 + col;
    if (wide) {
      LsCols f;
#pragma unroll
      for (int c = 0; c < LS_C; ++c) f.x[c] = x[c];
      *reinterpret_cast<LsCols*>(dst) = f;
    } else {
#pragma unroll
      for (int c = 0; c < LS_C; ++c) if (c0 + col + c < dv) dst[c] = x[c];
    }
  };

  lr_pair S[R / 2][LS_C];
  float m0 = 0.f;                                      // mode 1: the running maximum before the segment
  float follow[RT], lacks[RT];                         // the thread's rows of n, or of the decay since the segment's start and 1 minus it
  {
    const bool zero = PASS == 1 && sg > 0;
    const bool kept = PASS == 2 && nseg > 1;           // the first pass put the state before the step aside: the last segment
    const float* m = zero ? nullptr : kept ? first_S : S_h;                          // overwrites the slot
    const float* vec = zero ? nullptr : kept ? first_n : n_h;
    if (PASS == 2 && sg > 0) {
      m = A.ends + seg_at(0) * N * dv;
      vec = A.vecs + seg_at(0) * N;
    }
#pragma unroll
    for (int j = 0; j < R / 2; ++j) {
      float x[2][LS_C];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        load(m, j, e, x[e]);
        if (PASS == 1 && sg == 0) store(first_S, j, e, x[e]);
      }
#pragma unroll
      for (int c = 0; c < LS_C; ++c) S[j][c] = lr_make(x[0][c], x[1][c]);
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = tid + i * LS_THREADS;
      follow[i] = 1.f; lacks[i] = 0.f;
      if (MODE == 1 && leads) {
        follow[i] = vec != nullptr && r < N ? vec[r] : 0.f;
        if (PASS == 1 && sg == 0 && r < N) first_n[r] = follow[i];
      }
    }
    if (MODE == 1) m0 = zero ? -INFINITY : A.first_m[(size_t)s * H + h];
    if (PASS == 2 && sg > 0) {
      // S is the state at the end of segment 0; the segments after it, one behind the other
      if (MODE == 1) m0 = fmaxf(scale_at(0)[0] + m0, scale_at(0)[1]);
      for (int i = 1; i < sg; ++i) {
        const size_t at = seg_at(i);
        const float* sc = scale_at(i);
        const float* em = A.ends + at * N * dv;
        const float* ev = A.vecs + at * N;
        float c1 = 1.f, c2 = 1.f;
        if (MODE == 0) c1 = sc[0];
        if (MODE == 1) {
          const float fm = sc[0] + m0, lm = sc[1];
          const float mn = fmaxf(fm, lm);
          c1 = expf(fm - mn); c2 = expf(lm - mn); m0 = mn;
          if (leads) {
#pragma unroll
            for (int u = 0; u < RT; ++u) if (tid + u * LS_THREADS < N) follow[u] = fmaf(c1, follow[u], c2 * ev[tid + u * LS_THREADS]);
          }
        }
#pragma unroll
        for (int j = 0; j < R / 2; ++j) {
          float x[2][LS_C], d[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            load(em, j, e, x[e]);
            d[e] = SCALAR ? c1 : (row_of(j, e) < N ? ev[row_of(j, e)] : 0.f);
          }
          const lr_pair dd = lr_make(d[0], d[1]), kept = ls_mask2(d[0], d[1]), one = lr_dup(1.0f);
#pragma unroll
          for (int c = 0; c < LS_C; ++c) {
            const lr_pair end = lr_make(MODE == 1 ? c2 * x[0][c] : x[0][c], MODE == 1 ? c2 * x[1][c] : x[1][c]);
            S[j][c] = lr_fma2(dd, S[j][c], SCALAR ? end : lr_fma2(one, S[j][c] & kept, end));
          }
        }
      }
    }
  }
  // what no copy writes: rows beyond N, columns beyond the head
  if (N < NP) for (int i = tid; i < (2 + (HAS_Q ? 2 : 0) + (HAS_A ? 2 : 0)) * LS_CHUNK * NP; i += LS_THREADS) ks[i] = 0.f;
  if (ncol < BC) for (int i = tid; i < 2 * LS_CHUNK * BC; i += LS_THREADS) vs[i] = 0.f;
  __syncthreads();

  // walks the pieces tid, tid + LS_THREADS .. of `rows` rows of `per` pieces each
  auto pieces = [&](int rows, int per, auto fn) {
    const int dt = LS_THREADS / per, dr = LS_THREADS - dt * per;
    int tt = tid / per, r = tid - tt * per;
    for (; tt < rows; tt += dt) {
      fn(tt, r);
      r += dr;
      if (r >= per) { r -= per; ++tt; }
    }
  };
  auto issue = [&](int base, int stage) {
    const int cnt = min(LS_CHUNK, b1 - base);
    float* kd = ks + (size_t)stage * LS_CHUNK * NP;
    float* qd = qs + (size_t)stage * LS_CHUNK * NP;
    float* ad = as + (size_t)stage * LS_CHUNK * NP;
    float* vd = vs + (size_t)stage * LS_CHUNK * BC;
    const float* kg = A.k + (size_t)base * A.k_stride + (size_t)hq * N;
    const float* qg = A.q + (size_t)base * A.q_stride + (size_t)hq * N;
    const float* ag = A.a + (HAS_A ? (size_t)base * A.a_stride + (size_t)hq * N : 0);
    const float* vg = A.v + (size_t)base * A.v_stride + (size_t)h * dv + c0;
    if (A.vec) {
      pieces(cnt, N / 4, [&](int tt, int r) {
        lr_cp16(kd + tt * NP + r * 4, kg + tt * A.k_stride + r * 4);
        if (HAS_Q) lr_cp16(qd + tt * NP + r * 4, qg + tt * A.q_stride + r * 4);
        if (HAS_A) lr_cp16(ad + tt * NP + r * 4, ag + tt * A.a_stride + r * 4);
      });
      pieces(cnt, ncol / 4, [&](int tt, int c) { lr_cp16(vd + tt * BC + c * 4, vg + tt * A.v_stride + c * 4); });
    } else {
      pieces(cnt, N, [&](int tt, int r) {
        lr_cp4(kd + tt * NP + r, kg + tt * A.k_stride + r);
        if (HAS_Q) lr_cp4(qd + tt * NP + r, qg + tt * A.q_stride + r);
        if (HAS_A) lr_cp4(ad + tt * NP + r, ag + tt * A.a_stride + r);
      });
      pieces(cnt, ncol, [&](int tt, int c) { lr_cp4(vd + tt * BC + c, vg + tt * A.v_stride + c); });
    }
    lr_commit();
  };

  const lr_pair minus = lr_dup(-1.0f);
  int oslot;                                           // where the first of the sums that this lane is left with stands in os
  {
    int at = 0, n = LS_C * TG;
#pragma unroll
    for (int d = L / 2; d > 0; d >>= 1) {
      n = n > 1 ? n / 2 : 0;
      if (sub & d) at += n;
    }
    oslot = at / LS_C * BC + col + at % LS_C;
  }
  const size_t TH = (size_t)A.T * H;
  float raw[6];                                        // lanes 0 .. 15 of warp 0: a token's gates as they lie in memory
  auto fetch_gates = [&](int base) {
    const int t = base + lane;
    if (!SCALAR || warp != 0 || lane >= LS_CHUNK || t >= b1) return;
    const size_t at = (size_t)t * H + h;
    raw[0] = A.gates[at]; raw[1] = A.gates[TH + at];
    if (MODE == 1) {
      raw[2] = A.gates[2 * TH + at]; raw[3] = A.gates[3 * TH + at];
      if (t > b0) { raw[4] = A.gates[2 * TH + at - H]; raw[5] = A.gates[3 * TH + at - H]; }
    }
  };
  fetch_gates(b0);
  issue(b0, 0);
  int stage = 0;
  for (int base = b0; base < b1; base += LS_CHUNK, stage ^= 1) {
    const int cnt = min(LS_CHUNK, b1 - base);
    // the chunk's gates (their raw numbers came in under the chunk before).  Tokens behind the chunk keep everything and take
    // nothing.
    float gk = 1.f, gt = 0.f, gfl = 0.f, gb = 1.f, gB = 0.f;
    int gplain = 0;
    if (SCALAR && warp == 0) {
      if (lane < cnt) {
        if (MODE == 0) {
          gk = raw[0]; gt = raw[1];
        } else {
          const float m = fmaxf(raw[2] + m0, raw[3]);
          const float mp = base + lane == b0 ? m0 : fmaxf(raw[4] + m0, raw[5]);
          gk = expf(raw[0] + (mp - m)); gt = expf(raw[1] - m); gfl = expf(-m);
        }
      }
      fetch_gates(base + LS_CHUNK);
      gb = gk; gB = 1.0f - gk;                         // the decay since the chunk's start
#pragma unroll
      for (int o = 1; o < LS_CHUNK; o <<= 1) {
        float up = __shfl_up_sync(0xffffffffu, gb, o), upB = __shfl_up_sync(0xffffffffu, gB, o);
        if (lane >= o) { lr_decay(gb * up, gB, up, upB); gb = up; gB = upB; }
      }
      gplain = !(__shfl_sync(0xffffffffu, gb, LS_CHUNK - 1) >= LS_SMALL);
      if (!gplain) gt = gt / gb;
    }
    __syncthreads();                                   // the chunk before is written out: the other stage is free
    if (base + LS_CHUNK < b1) { issue(base + LS_CHUNK, stage ^ 1); lr_wait<1>(); } else lr_wait<0>();
    if (SCALAR && tid < LS_CHUNK) {
      keep_s[tid] = gk; take_s[tid] = gt; floor_s[tid] = gfl; by_s[tid] = gplain ? 1.f : gb;
      if (tid == 0) plain_s = gplain;
      if (tid == LS_CHUNK - 1) end_s[0] = lr_code(gb, gB);
    }
    __syncthreads();                                   // this chunk has landed for every thread
    float* kd = ks + (size_t)stage * LS_CHUNK * NP;
    float* qd = qs + (size_t)stage * LS_CHUNK * NP;
    float* ad = as + (size_t)stage * LS_CHUNK * NP;
    float* vd = vs + (size_t)stage * LS_CHUNK * BC;
    bool plain;
    if (SCALAR) {
      plain = plain_s != 0;
    } else {
      // a thread per row: the row's decays multiplied up, then its keys and queries brought into the chunk's scale
      auto row_decay = [&](int at, float& b, float& B) {
        const float x = HAS_A ? ad[at] : kd[at];           // the decay, or what it lacks to 1
        lr_decay(HAS_A ? x * b : fmaf(-x, b, b), HAS_A ? 1.0f - x : x, b, B);
      };
      float b_end[RT];
      bool small = false;
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int r = tid + i * LS_THREADS;
        float bt = 1.f, Bt = 0.f;
        if (r < N) for (int tt = 0; tt < cnt; ++tt) row_decay(tt * NP + r, bt, Bt);
        b_end[i] = lr_code(bt, Bt);
        const float f = follow[i];
        lr_decay(lr_apply(b_end[i], f), Bt, follow[i], lacks[i]);
        small |= !(bt >= LS_SMALL);
      }
      plain = __syncthreads_or(small) != 0;
      if (!plain) {
#pragma unroll
        for (int i = 0; i < RT; ++i) {
          const int r = tid + i * LS_THREADS;
          if (r < N) {
            float bt = 1.f, Bt = 0.f;
#pragma unroll 4
            for (int tt = 0; tt < cnt; ++tt) {
              const int at = tt * NP + r;
              const float kk = kd[at];
              row_decay(at, bt, Bt);
              kd[at] = kk / bt;
              if (HAS_Q) qd[at] *= bt;
            }
          }
          if (r < NP) end_s[r] = b_end[i];
        }
      }
    }
    if (cnt % TG != 0) {                               // the last tokens' group is filled up with tokens that change nothing
      const int fill = TG - cnt % TG;
      for (int i = tid; i < fill * NP; i += LS_THREADS) {
        kd[cnt * NP + i] = 0.f;
        if (HAS_Q) qd[cnt * NP + i] = 0.f;
        if (HAS_A) ad[cnt * NP + i] = 1.f;
      }
      for (int i = tid; i < fill * BC; i += LS_THREADS) vd[cnt * BC + i] = 0.f;
    }
    if (!SCALAR || cnt % TG != 0) __syncthreads();
    if (MODE == 1 && leads) {
      // a thread per row: n after every token of the chunk, and its share of n . q
      float nq[LS_CHUNK];
#pragma unroll
      for (int tt = 0; tt < LS_CHUNK; ++tt) nq[tt] = 0.f;
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const int r = tid + i * LS_THREADS;
        if (r < N) {
#pragma unroll
          for (int tt = 0; tt < LS_CHUNK; ++tt) {
            if (tt < cnt) {
              follow[i] = fmaf(take_s[tt], kd[tt * NP + r], plain ? keep_s[tt] * follow[i] : follow[i]);
              if (HAS_Q) nq[tt] = fmaf(follow[i], qd[tt * NP + r], nq[tt]);
            }
          }
          if (!plain) follow[i] = lr_apply(end_s[0], follow[i]);
        }
      }
      if (HAS_Q) {
        // the 16 tokens' sums over the warp's rows: lane l is left with token l / 2's
        lr_meet<16, LS_CHUNK>(nq, lane);
        if ((lane & 1) == 0) den_s[warp][lane >> 1] = nq[0];
      }
    }
    // TG tokens at a time, their read-outs' shares in val
    auto compute = [&](const bool PLAIN, int t, float (&val)[LS_C * TG]) __attribute__((always_inline)) {
#pragma unroll
      for (int u = 0; u < TG; ++u) {
        const LsCols v2 = *reinterpret_cast<const LsCols*>(vd + (t + u) * BC + col);
        lr_pair o[LS_C], vp[LS_C], keep2;
        if (SCALAR) {
          const float w = take_s[t + u];
          if (PLAIN) keep2 = lr_dup(keep_s[t + u]);
#pragma unroll
          for (int c = 0; c < LS_C; ++c) vp[c] = lr_dup(w * v2.x[c]);
        } else {
#pragma unroll
          for (int c = 0; c < LS_C; ++c) vp[c] = lr_dup(v2.x[c]);
        }
#pragma unroll
        for (int j = 0; j < R / 4; ++j) {
          const int at = (t + u) * NP + (j * L + sub) * 4;
          const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(kd + at);
          ulonglong2 q2, a2;
          if (HAS_Q) q2 = *reinterpret_cast<const ulonglong2*>(qd + at);
          if (PLAIN && HAS_A) a2 = *reinterpret_cast<const ulonglong2*>(ad + at);
#pragma unroll
          for (int c = 0; c < LS_C; ++c) {
            if (!PLAIN) {
              S[2 * j][c] = lr_fma2(k2.x, vp[c], S[2 * j][c]);
              S[2 * j + 1][c] = lr_fma2(k2.y, vp[c], S[2 * j + 1][c]);
            } else if (MODE == 2) {
              S[2 * j][c] = lr_fma2(k2.x, lr_fma2(S[2 * j][c], minus, vp[c]), S[2 * j][c]);       // v - S, one rounding
              S[2 * j + 1][c] = lr_fma2(k2.y, lr_fma2(S[2 * j + 1][c], minus, vp[c]), S[2 * j + 1][c]);
            } else {
              S[2 * j][c] = lr_fma2(k2.x, vp[c], lr_mul2(HAS_A ? a2.x : keep2, S[2 * j][c]));
              S[2 * j + 1][c] = lr_fma2(k2.y, vp[c], lr_mul2(HAS_A ? a2.y : keep2, S[2 * j + 1][c]));
            }
            if (HAS_Q) {
              o[c] = j == 0 ? lr_mul2(q2.x, S[0][c]) : lr_fma2(q2.x, S[2 * j][c], o[c]);
              o[c] = lr_fma2(q2.y, S[2 * j + 1][c], o[c]);
            }
          }
        }
        if (HAS_Q) {
#pragma unroll
          for (int c = 0; c < LS_C; ++c) val[LS_C * u + c] = lr_sum2(o[c]);
        }
      }
    };
    auto meet = [&](int t, float (&val)[LS_C * TG]) {
      if (!HAS_Q) return;
      lr_meet<L / 2, LS_C * TG>(val, sub);
      constexpr int LEFT = LS_C * TG > L ? LS_C * TG / L : 1;  // sums a lane is left with
      constexpr int SPARE = LS_C * TG < L ? L / (LS_C * TG) : 1;   // lanes that end up with the same sum
      if ((sub & (SPARE - 1)) == 0) {
#pragma unroll
        for (int i = 0; i < LEFT; ++i) os[t * BC + oslot + i / LS_C * BC + i % LS_C] = val[i];
      }
    };
    {
      if (plain) {
        // rare: a loop of its own, so that the usual form keeps the registers
#pragma unroll 1
        for (int t = 0; t < cnt; t += TG) {
          float val[LS_C * TG];
          compute(true, t, val);
          meet(t, val);
        }
      } else {
        if (cnt == LS_CHUNK) {
          // straight-line code: the shuffles of one group of tokens run beside the arithmetic of the next
          float val[2][LS_C * TG];
          compute(false, 0, val[0]);
#pragma unroll
          for (int g = 1; g < LS_CHUNK / TG; ++g) {
            compute(false, g * TG, val[g & 1]);
            meet((g - 1) * TG, val[(g - 1) & 1]);
          }
          meet(LS_CHUNK - TG, val[(LS_CHUNK / TG - 1) & 1]);
        } else {
          for (int t = 0; t < cnt; t += TG) {
            float val[LS_C * TG];
            compute(false, t, val);
            meet(t, val);
          }
        }
        lr_pair e2[2], kept[2];
        if (SCALAR) { e2[0] = e2[1] = lr_dup(end_s[0]); kept[0] = kept[1] = ls_mask2(end_s[0], end_s[0]); }
#pragma unroll
        for (int j = 0; j < R / 4; ++j) {
          if (!SCALAR) {
            const float4 e = *reinterpret_cast<const float4*>(end_s + (j * L + sub) * 4);
            e2[0] = lr_make(e.x, e.y); e2[1] = lr_make(e.z, e.w);
            kept[0] = ls_mask2(e.x, e.y); kept[1] = ls_mask2(e.z, e.w);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int c = 0; c < LS_C; ++c) S[2 * j + i][c] = lr_fma2(e2[i], S[2 * j + i][c], S[2 * j + i][c] & kept[i]);
        }
      }
    }
    if (PASS == 2) {
      __syncthreads();
      if (MODE == 1 && leads && tid < cnt) {
        const float nq = (den_s[0][tid] + den_s[1][tid]) + (den_s[2][tid] + den_s[3][tid]);
        A.den[(size_t)(base + tid) * H + h] = fmaxf(fabsf(nq * by_s[tid] * A.q_scale), floor_s[tid]) + 1e-6f;
      }
      float* og = A.out + (size_t)base * A.out_stride + (size_t)h * dv + c0;
      const float skip = MODE == 0 ? A.d_skip[h] : 0.f;
      if (A.vec) {
        pieces(cnt, ncol / 4, [&](int tt, int c) {
          const float f = SCALAR ? by_s[tt] * A.q_scale : A.q_scale;
          float4 y = *reinterpret_cast<const float4*>(os + tt * BC + c * 4);
          y.x *= f; y.y *= f; y.z *= f; y.w *= f;
          if (MODE == 0) {
            const float4 x = *reinterpret_cast<const float4*>(vd + tt * BC + c * 4);
            y.x = fmaf(skip, x.x, y.x); y.y = fmaf(skip, x.y, y.y); y.z = fmaf(skip, x.z, y.z); y.w = fmaf(skip, x.w, y.w);
          }
          *reinterpret_cast<float4*>(og + tt * A.out_stride + c * 4) = y;
        });
      } else {
        pieces(cnt, ncol, [&](int tt, int c) {
          const float y = os[tt * BC + c] * (SCALAR ? by_s[tt] * A.q_scale : A.q_scale);
          og[tt * A.out_stride + c] = MODE == 0 ? fmaf(skip, vd[tt * BC + c], y) : y;
        });
      }
    }
  }
  float* m = nullptr;
  float* vec = nullptr;
  if (PASS == 1) {
    m = A.ends + seg_at(sg) * N * dv;
    vec = A.vecs + seg_at(sg) * N;
  } else if (sg == nseg - 1) {
    m = S_h; vec = n_h;
    if (MODE == 1 && leads && tid == 0 && row0) {
      const float* sc = scale_at(sg);
      row0[(size_t)H * N * (dv + 1) + h] = fmaxf(sc[0] + m0, sc[1]);
    }
  }
#pragma unroll
  for (int j = 0; j < R / 2; ++j) {
    float x[2][LS_C];
#pragma unroll
    for (int c = 0; c < LS_C; ++c) lr_split(S[j][c], x[0][c], x[1][c]);
#pragma unroll
    for (int e = 0; e < 2; ++e) store(m, j, e, x[e]);
  }
  if (leads && vec != nullptr && (MODE == 1 || (PASS == 1 && !SCALAR))) {
#pragma unroll
    for (int i = 0; i < RT; ++i) if (tid + i * LS_THREADS < N) vec[tid + i * LS_THREADS] = MODE == 1 ? follow[i] : lr_code(follow[i], lacks[i]);
  }
}

template <int MODE, int L, int R, int PASS>
static int ls_walk(LsArgs A, cudaStream_t stream) {
  constexpr int BC = 4 * LS_C * (32 / L), NP = L * R;
  const size_t smem = ((size_t)2 * LS_CHUNK * NP * (1 + (PASS == 2) + (MODE == 3)) + (2 + (PASS == 2)) * LS_CHUNK * BC) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(ls_walk_kernel<MODE, L, R, PASS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  ls_walk_kernel<MODE, L, R, PASS><<<dim3((A.dv + BC - 1) / BC, A.H, A.segs), LS_THREADS, smem, stream>>>(A);
  return launch_status();
}

template <int MODE, int L, int R>
static int ls_go(const LsArgs& A, cudaStream_t stream) {
  if (A.cuts > 0) {
    const int st = ls_walk<MODE, L, R, 1>(A, stream);
    if (st != 0) return st;
  }
  return ls_walk<MODE, L, R, 2>(A, stream);
}

template <int MODE>
static int ls_rows(const LsArgs& A, cudaStream_t stream) {
  if (A.N <= 32) return ls_go<MODE, 8, 4>(A, stream);
  if (A.N <= 64) return ls_go<MODE, 8, 8>(A, stream);
  if (A.N <= 128) return ls_go<MODE, 16, 8>(A, stream);
  if (A.N <= 256) return ls_go<MODE, 32, 8>(A, stream);
  return ls_go<MODE, 32, 16>(A, stream);
}

// Blocks of one (segment, head), for the caller that cuts a step into segments.
PHOTON_API int photon_linrec_segment_blocks(int N, int dv) {
  const int bc = 4 * LS_C * (N <= 64 ? 4 : N <= 128 ? 2 : 1);
  return (dv + bc - 1) / bc;
}

// The parts of photon_linrec_segments' scratch in floats: gates, ends, vectors, scales, the states and the running maxima before
// the step.
static void ls_parts(int mode, int T, int S, int segs, int cuts, int cut_segs, int H, int N, int dv, long (&part)[6]) {
  auto four = [](long n) { return (n + 3) & ~3L; };
  part[0] = four(mode == 0 ? 2L * T * H : mode == 1 ? 4L * T * H : 0);
  part[1] = four((long)cut_segs * H * N * dv);
  part[2] = four((long)cut_segs * H * N);
  part[3] = four((long)segs * H * 2);
  part[4] = four((long)cuts * H * ((long)N * dv + N));
  part[5] = four((long)S * H);
}

PHOTON_API long photon_linrec_segments_scratch(int mode, int T, int S, int segs, int cuts, int cut_segs, int H, int N, int dv) {
  long part[6], sum = 0;
  ls_parts(mode, T, S, segs, cuts, cut_segs, H, N, dv, part);
  for (long p : part) sum += p;
  return sum;
}

// As photon_linrec, for requests cut into segments of `seg` tokens (a multiple of 16): `segs` of them in all, `cut_segs` of which
// belong to the `cuts` requests that have more than one; mode 3: a float [T][qk_heads * N] the rows' decays, ga .. p2 unused.  Mode 2: q and k as photon_linrec_gates leaves them.  Mode 1: den
// float [T][H] gets what the outputs are to be divided by, and out is not divided.  scratch: photon_linrec_segments_scratch
// floats, 16-byte aligned.  N up to 512.
PHOTON_API int photon_linrec_segments(int mode, const float* q, long q_stride, const float* k, long k_stride, const float* v,
                                      long v_stride, const float* a, long a_stride, const float* ga, const float* gb, long g_stride,
                                      const float* p0, const float* p1, const float* p2, float cap, float q_scale,
                                      const int* cu_tokens, const int* state_slots, float* state, long state_stride, int num_slots,
                                      float* out, long out_stride, float* den, float* scratch, int T, int S, int H, int qk_heads,
                                      int N, int dv, int seg, int segs, int cuts, int cut_segs, int* err, cudaStream_t stream) {
  if (S <= 0 || T <= 0) return 0;
  if (mode < 0 || mode > 3 || H <= 0 || qk_heads <= 0 || H % qk_heads || N <= 0 || dv <= 0 || seg <= 0 || seg % LS_CHUNK || segs <= 0 ||
      cuts < 0 || cut_segs < 0)
    return PHOTON_ERR_ARGUMENT;
  if (scratch == nullptr || ((uintptr_t)scratch & 15) || (mode == 1 && (!(cap > 0.f) || den == nullptr)) || (mode == 3) != (a != nullptr))
    return PHOTON_ERR_ARGUMENT;
  if (N > 512 || H > 65535 || segs > 65535) return PHOTON_ERR_UNSUPPORTED;
  LsArgs A;
  A.q = q; A.q_stride = q_stride; A.k = k; A.k_stride = k_stride; A.v = v; A.v_stride = v_stride; A.a = a; A.a_stride = a_stride;
  A.d_skip = p2; A.q_scale = q_scale; A.cu_tokens = cu_tokens; A.state_slots = state_slots; A.state = state; A.state_stride = state_stride;
  A.num_slots = num_slots; A.out = out; A.out_stride = out_stride; A.den = den;
  A.T = T; A.S = S; A.H = H; A.qk_heads = qk_heads; A.N = N; A.dv = dv; A.seg = seg; A.segs = segs; A.cuts = cuts;
  A.cut_segs = cut_segs; A.err = err;
  long part[6];
  ls_parts(mode, T, S, segs, cuts, cut_segs, H, N, dv, part);
  float* gates = scratch;
  A.gates = gates;
  A.ends = gates + part[0];
  A.vecs = A.ends + part[1];
  A.scale = A.vecs + part[2];
  A.first = A.scale + part[3];
  A.first_m = A.first + part[4];
  A.vec = N % 4 == 0 && dv % 4 == 0 && q_stride % 4 == 0 && k_stride % 4 == 0 && v_stride % 4 == 0 && state_stride % 4 == 0 && out_stride % 4 == 0 &&
          ((uintptr_t)out & 15) == 0 && ((uintptr_t)q & 15) == 0 && ((uintptr_t)k & 15) == 0 && ((uintptr_t)v & 15) == 0 && ((uintptr_t)state & 15) == 0 &&
          (a == nullptr || (a_stride % 4 == 0 && ((uintptr_t)a & 15) == 0));
  if (mode < 2) {
    const dim3 grid(segs, (H + 3) / 4);
    if (mode == 0) ls_gates_kernel<0><<<grid, 128, 0, stream>>>(ga, gb, g_stride, p0, p1, cap, gates, A);
    else ls_gates_kernel<1><<<grid, 128, 0, stream>>>(ga, gb, g_stride, p0, p1, cap, gates, A);
    const int st = launch_status();
    if (st != 0) return st;
  }
  if (mode == 0) return ls_rows<0>(A, stream);
  if (mode == 1) return ls_rows<1>(A, stream);
  if (mode == 2) return ls_rows<2>(A, stream);
  return ls_rows<3>(A, stream);
}
