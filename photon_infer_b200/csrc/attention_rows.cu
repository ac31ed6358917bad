// Paged causal attention of several tokens of a request in true 32-bit: attention.cu's sums, bit for bit, for prompt portions with
// heads of 64 or 128.
//
// attention.cu gives every (token, key/value head) a block of its own, which reads the keys and values that the token before it
// has read and takes two numbers from shared memory for every product.  Here a block takes up to 32 rows, the query heads of a key/value head for
// 32 / heads tokens of one request, and walks the same tiles of 32 keys from key 0.  A thread holds the scores of four rows with
// four keys, then the outputs of those rows for D / 8 numbers, and reads 16 bytes at a time: eight 16-byte reads for 64 products
// of the scores, twelve for 128 of the outputs (D = 64), none of which conflict, since a thread's rows are 8 apart and rows are padded by 16
// bytes.  Keys and values come by cp.async, a tile's values while its scores form, the next tile's keys behind those.  Two warps
// a block: small blocks so that a short portion fills the chip.
//
// The order of every sum is attention.cu's: a score adds its D products up one behind the other, the sum over a tile's 32
// probabilities is a butterfly from 16 apart to 1 apart (the first two steps lie within a thread), an output is scaled and takes the
// tile's keys in order.  Keys behind a row's token are never multiplied.
//
// Bound by the products' issue and the reads beside them, and at few units by a tile's latency (4 us).  512 tokens, 32/8 heads of
// 64: 88 us, attention.cu 264; heads of 128: 167 and 545.
#include "common.cuh"
#include <math.h>

#define AR_TILE 32
#define AR_ROWS 32
#define AR_THREADS 64

__device__ __forceinline__ void ar_copy16(float* dst, const float* src, bool there) {     // not there: the bytes become zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0));
}
__device__ __forceinline__ void ar_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ar_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int D>
__global__ void __launch_bounds__(AR_THREADS, D == 64 ? 7 : 4)
attention_rows_kernel(const float* __restrict__ q, long q_stride, float* __restrict__ out, long out_stride, const float* __restrict__ k_cache,
                      const float* __restrict__ v_cache, const int* __restrict__ block_table, int max_pages, const int* __restrict__ cu_tokens,
                      const int* __restrict__ positions, int num_seqs, int n_q, int n_kv, int page_size, int num_pages, float scale, int* err) {
  constexpr int S = D + 4, PS = AR_TILE + 4, C4 = D / 32;     // strides in shared memory; a thread's groups of four output numbers
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                                           // [AR_ROWS][S]
  float* ks = qs + AR_ROWS * S;                               // [AR_TILE][S]
  float* vs = ks + AR_TILE * S;                               // [AR_TILE][D]
  float* ps = vs + AR_TILE * D;                               // [AR_ROWS][PS]
  __shared__ long long krow[2][AR_TILE];
  const int tid = threadIdx.x, lane = tid & 31;
  const int tr = tid >> 3, tc = tid & 7;                      // rows tr, tr + 8, tr + 16, tr + 24; keys tc, tc + 8, ..; columns 4 tc, 4 tc + 32, ..
  const int g = blockIdx.y, G = n_q / n_kv, tok = AR_ROWS / G;
  // Units of `tok` tokens, one request behind the other; the last units (of a lone request: the most keys) start first.  Every warp
  // walks the requests, 32 at a time, to the one that holds its unit.
  const int unit = gridDim.x - 1 - blockIdx.x;
  int seq = -1, before = 0, total = 0;
  for (int s0 = 0; s0 < num_seqs; s0 += 32) {
    const int s = s0 + lane;
    const int n = s < num_seqs ? (cu_tokens[s + 1] - cu_tokens[s] + tok - 1) / tok : 0;
    int upto = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, total + upto > unit);
    if (hit != 0) {
      const int l = __ffs(hit) - 1;
      seq = s0 + l;
      before = total + __shfl_sync(0xffffffffu, upto - n, l);
      break;
    }
    total += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (seq < 0) return;                                        // the grid is an upper bound
  const int t0 = cu_tokens[seq] + (unit - before) * tok;
  const int rows = min(tok, cu_tokens[seq + 1] - t0) * G;
  const int* table = block_table + (size_t)seq * max_pages;

  int pos[4];                                                 // the positions of this thread's rows; -1: no such row
  int pmax = 0, pmin = 0x7fffffff;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = tr + 8 * i;
    pos[i] = r < rows ? positions[t0 + r / G] : -1;
  }
  for (int t = 0; t * G < rows; ++t) {
    const int p = positions[t0 + t];
    pmax = max(pmax, p);
    pmin = min(pmin, p);
  }
  const int tiles = pmax / AR_TILE + 1;

  auto find_rows = [&](int tile) {                            // threads 0 .. 31: the cache rows of a tile's keys
    const int kk = tile * AR_TILE + tid;
    long long row = -1;
    if (kk <= pmax) {
      const int page = table[kk / page_size];
      if (page < 0 || page >= num_pages) {
        int t = 0;                                            // the first token that sees the key
        while ((t + 1) * G < rows && positions[t0 + t] < kk) ++t;
        report_error(err, PHOTON_DEV_BAD_PAGE, t0 + t, kk, page);
      } else {
        row = ((long long)page * n_kv + g) * page_size + (kk % page_size);
      }
    }
    krow[tile & 1][tid] = row;
  };
  auto fetch = [&](const float* cache, float* dst, int stride, int tile) {
#pragma unroll
    for (int i = 0; i < AR_TILE * (D / 4) / AR_THREADS; ++i) {
      const int e = tid + i * AR_THREADS, key = e / (D / 4), j = e % (D / 4) * 4;
      const long long row = krow[tile & 1][key];
      ar_copy16(dst + key * stride + j, cache + (row >= 0 ? row * D + j : 0), row >= 0);
    }
    ar_commit();
  };

  if (tid < AR_TILE) find_rows(0);
  for (int e = tid; e < AR_ROWS * (D / 4); e += AR_THREADS) {
    const int r = e / (D / 4), j = e % (D / 4) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) v = *reinterpret_cast<const float4*>(q + (size_t)(t0 + r / G) * q_stride + (size_t)(g * G + r % G) * D + j);
    *reinterpret_cast<float4*>(qs + r * S + j) = v;
  }
  __syncthreads();
  fetch(k_cache, ks, S, 0);

  float acc[4][C4 * 4], m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < C4 * 4; ++c) acc[i][c] = 0.f;
  }
  for (int tile = 0; tile < tiles; ++tile) {
    const int tile0 = tile * AR_TILE;
    ar_wait<0>();                                             // this tile's keys
    __syncthreads();                                          // .. of every thread; the values of the tile before are read
    fetch(v_cache, vs, D, tile);
    if (tid < AR_TILE && tile + 1 < tiles) find_rows(tile + 1);
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) s[i][c] = 0.f;
#pragma unroll 4
    for (int j = 0; j < D; j += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (tr + 8 * i) * S + j);
#pragma unroll
      for (int c = 0; c < 4; ++c) b[c] = *reinterpret_cast<const float4*>(ks + (tc + 8 * c) * S + j);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          s[i][c] = fmaf(a[i].x, b[c].x, s[i][c]); s[i][c] = fmaf(a[i].y, b[c].y, s[i][c]);
          s[i][c] = fmaf(a[i].z, b[c].z, s[i][c]); s[i][c] = fmaf(a[i].w, b[c].w, s[i][c]);
        }
    }
    bool seen[4];                                             // keys whose page is there
#pragma unroll
    for (int c = 0; c < 4; ++c) seen[c] = krow[tile & 1][tc + 8 * c] >= 0;
    __syncthreads();                                          // the keys are read, the next tile's rows are known
    if (tile + 1 < tiles) fetch(k_cache, ks, S, tile + 1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float mt = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[i][c] = seen[c] && tile0 + tc + 8 * c <= pos[i] ? s[i][c] * scale : -INFINITY;
        mt = fmaxf(mt, s[i][c]);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) mt = fmaxf(mt, __shfl_xor_sync(0xffffffffu, mt, o));
      const float m_new = fmaxf(m[i], mt);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[i][c] = s[i][c] == -INFINITY ? 0.f : expf(s[i][c] - m_new);
        ps[(tr + 8 * i) * PS + tc + 8 * c] = s[i][c];
      }
      float sum = (s[i][0] + s[i][2]) + (s[i][1] + s[i][3]);
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
      l[i] = fmaf(l[i], corr, sum);
      m[i] = m_new;
#pragma unroll
      for (int c = 0; c < C4 * 4; ++c) acc[i][c] *= corr;
    }
    if (tile + 1 < tiles) ar_wait<1>(); else ar_wait<0>();    // this tile's values
    __syncthreads();
    const bool whole = tile0 + AR_TILE - 1 <= pmin;      // rows that are not there take any numbers
#pragma unroll 2
    for (int k = 0; k < AR_TILE; k += 4) {
      float4 w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(ps + (tr + 8 * i) * PS + k);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 v[C4];
#pragma unroll
        for (int c = 0; c < C4; ++c) v[c] = *reinterpret_cast<const float4*>(vs + (k + u) * D + 4 * tc + 32 * c);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float p = u == 0 ? w[i].x : u == 1 ? w[i].y : u == 2 ? w[i].z : w[i].w;
          if (whole || tile0 + k + u <= pos[i]) {
#pragma unroll
            for (int c = 0; c < C4; ++c) {
              acc[i][4 * c] = fmaf(p, v[c].x, acc[i][4 * c]); acc[i][4 * c + 1] = fmaf(p, v[c].y, acc[i][4 * c + 1]);
              acc[i][4 * c + 2] = fmaf(p, v[c].z, acc[i][4 * c + 2]); acc[i][4 * c + 3] = fmaf(p, v[c].w, acc[i][4 * c + 3]);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = tr + 8 * i;
    if (r >= rows) continue;
    float* dst = out + (size_t)(t0 + r / G) * out_stride + (size_t)(g * G + r % G) * D + 4 * tc;
#pragma unroll
    for (int c = 0; c < C4; ++c) {
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
      if (l[i] > 0.f) y = make_float4(acc[i][4 * c] / l[i], acc[i][4 * c + 1] / l[i], acc[i][4 * c + 2] / l[i], acc[i][4 * c + 3] / l[i]);
      *reinterpret_cast<float4*>(dst + 32 * c) = y;
    }
  }
}

template <int D>
static int attention_rows_launch(const float* q, long q_stride, float* out, long out_stride, const float* k_cache, const float* v_cache,
                                 const int* block_table, int max_pages, const int* cu_tokens, const int* positions, int T_, int num_seqs,
                                 int n_q, int n_kv, int page_size, int num_pages, float scale, int* err, cudaStream_t stream) {
  const size_t smem = ((size_t)2 * AR_ROWS * (D + 4) + AR_TILE * D + AR_ROWS * (AR_TILE + 4)) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  const int tok = AR_ROWS / (n_q / n_kv);
  attention_rows_kernel<D><<<dim3(T_ / tok + num_seqs, n_kv), AR_THREADS, smem, stream>>>(
      q, q_stride, out, out_stride, k_cache, v_cache, block_table, max_pages, cu_tokens, positions, num_seqs, n_q, n_kv, page_size, num_pages,
      scale, err);
  return launch_status();
}

// q, out [T][n_q * d] float (row strides in elements); k_cache, v_cache [num_pages][n_kv][page_size][d] float; cu_tokens [num_seqs + 1]: the
// tokens of the requests, T in all; a token at positions[t] sees the keys 0 .. positions[t].  d 64 or 128, up to 32 query heads per
// key/value head, 16-byte aligned rows (others: PHOTON_ERR_UNSUPPORTED).
PHOTON_API int photon_attention_rows(const float* q, long q_stride, float* out, long out_stride, const float* k_cache, const float* v_cache,
                                     const int* block_table, int max_pages, const int* cu_tokens, const int* positions, int T_, int num_seqs,
                                     int n_q, int n_kv, int d, int page_size, int num_pages, float scale, int* err, cudaStream_t stream) {
  if (T_ <= 0 || num_seqs <= 0) return 0;
  if (n_kv <= 0 || n_q % n_kv || page_size <= 0) return PHOTON_ERR_ARGUMENT;
  if ((d != 64 && d != 128) || n_q / n_kv > AR_ROWS || n_kv > 65535 || q_stride % 4 || out_stride % 4 ||
      ((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) % 16)
    return PHOTON_ERR_UNSUPPORTED;
  return (d == 64 ? attention_rows_launch<64> : attention_rows_launch<128>)(q, q_stride, out, out_stride, k_cache, v_cache, block_table,
      max_pages, cu_tokens, positions, T_, num_seqs, n_q, n_kv, page_size, num_pages, scale, err, stream);
}
